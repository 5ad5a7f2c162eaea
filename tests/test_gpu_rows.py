"""Packed rows of a row evaluation: uploaded, unpacked on the device and
evaluated (GPU), at row counts around a block of the unpacking kernel (8 rows)
and past the limits up to which the engine keeps a call's memory; and the
host arrays of the call, field by field (CPU)."""
import dataclasses

import numpy as np
import pytest

from gagp_b200 import abi, task as T, workloads as W
from oracle import oracle


def _task(tmp_path, **kw):
    files = W.poly4(generations=2, **kw)
    return T.load(files.write(str(tmp_path)), str(tmp_path / "search.json"))


def _take(rows, index):
    out = abi.RowsBuffer(len(index), rows.stride)
    out.node_counts[:], out.constant_counts[:] = rows.node_counts[index], rows.constant_counts[index]
    out.origins[:], out.constants[:] = rows.origins[index], rows.constants[index]
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("count", [1, 7, 8, 9, 301])
def test_packed_rows_match_the_oracle(tmp_path, count):
    from gagp_b200.engine import Engine, evaluate_rows_static
    lt = _task(tmp_path, population=512, seed=31, cases=65)
    blob = abi.GrammarBlob(lt.tables)
    # the longest rows last, so that a short row follows no longer one
    rows = oracle.initial_population(blob, lt.settings)
    rows = _take(rows, np.argsort(rows.node_counts, kind="stable")[-count:])
    want_f, want_w, _ = oracle.evaluate(blob, lt.cases, lt.settings, rows)
    with Engine(0) as engine:
        f, w = engine.evaluate_rows(lt, rows)
    assert np.array_equal(f, want_f) and np.array_equal(w, want_w)
    f, w = evaluate_rows_static(lt, rows)
    assert np.array_equal(f, want_f) and np.array_equal(w, want_w)


@pytest.mark.gpu
def test_rows_past_the_kept_memory(tmp_path):
    """70,000 rows (more device memory than the engine keeps), then 3,000,000
    cases (more staging than it keeps), then a small call again."""
    from gagp_b200.engine import Engine
    lt = _task(tmp_path, population=512, seed=32, cases=20)
    rows = oracle.initial_population(abi.GrammarBlob(lt.tables), lt.settings)
    want_f, want_w, _ = oracle.evaluate(abi.GrammarBlob(lt.tables), lt.cases, lt.settings, rows)
    index = np.arange(70000) % 512
    c = lt.cases
    many = dataclasses.replace(lt, cases=abi.CasesBlob(np.tile(c.inputs, (150000, 1)), c.input_tags,
                                                       np.tile(c.expected, 150000)))
    few = _take(rows, np.arange(5))
    with Engine(0) as engine:
        f, w = engine.evaluate_rows(lt, _take(rows, index))
        assert np.array_equal(f, want_f[index]) and np.array_equal(w, want_w[index])
        f, w = engine.evaluate_rows(many, few)
        assert np.array_equal(f, 150000 * want_f[:5]) and np.array_equal(w, 150000 * want_w[:5])
        f, w = engine.evaluate_rows(lt, rows)
        assert np.array_equal(f, want_f) and np.array_equal(w, want_w)


def test_grammar_arrays_hold_every_field(tmp_path):
    lt = _task(tmp_path, population=8, seed=1, cases=4)
    blob = abi.GrammarBlob(lt.tables)
    for e, x in zip(lt.tables.expressions, blob.expressions):
        for name in ("kind", "node_kind", "opcode", "operand", "arity", "fuel", "merge_fuel", "type", "target",
                     "scope_count"):
            assert getattr(x, name) == getattr(e, name), name
        assert list(x.children) == list(e.children) and list(x.child_scope) == list(e.child_scope)


def test_verdict_summaries_match_one_by_one():
    out = (abi.Verdict * 3)()
    for v, (cases, correct, errors, loss) in zip(out, [(7, 7, 0, 0.0), (7, 3, 1, 40.0), (7, 0, 7, 7e9)]):
        v.cases, v.correct, v.runtime_errors, v.loss = cases, correct, errors, loss
    got = abi.verdict_summaries(out, 2)
    assert got == [out[0].summary(), out[1].summary()]
    assert [type(x) for x in got[0].values()] == [type(x) for x in out[0].summary().values()]


@pytest.mark.gpu
def test_rows_from_several_threads(tmp_path):
    """Host threads that evaluate and judge rows on one engine at the same
    time, calls of unequal sizes (the engine's staging grows meanwhile), while
    another reads a search's result: every call gets its own rows' scores."""
    from concurrent.futures import ThreadPoolExecutor
    from gagp_b200.engine import Engine
    lt = _task(tmp_path, population=512, seed=33, cases=40)
    blob = abi.GrammarBlob(lt.tables)
    rows = oracle.initial_population(blob, lt.settings)
    want_f, want_w, _ = oracle.evaluate(blob, lt.cases, lt.settings, rows)
    rng = np.random.default_rng(5)
    picks = [rng.integers(0, 512, size=size) for size in (3, 4000, 17, 900, 12000, 64, 2500, 5)]

    def evaluate(pick):
        out = []
        for _ in range(8):
            f, w = engine.evaluate_rows(lt, _take(rows, pick))
            out.append(np.array_equal(f, want_f[pick]) and np.array_equal(w, want_w[pick]))
        return all(out)

    def judge(pick):
        taken = _take(rows, pick)
        return all([v["wrong"] for v in engine.judge_rows(lt, taken, lt.cases)] == list(want_w[pick])
                   for _ in range(8))

    with Engine(0) as engine:
        s = engine.admit(lt)
        s.run()
        want = s.result()

        def read(_):
            return all(s.result() == want for _ in range(8))

        with ThreadPoolExecutor(len(picks) + 1) as pool:
            jobs = [pool.submit(judge if i % 3 == 2 else evaluate, pick) for i, pick in enumerate(picks)]
            jobs.append(pool.submit(read, None))
            assert all(job.result() for job in jobs)
        s.close()


@pytest.mark.gpu
def test_rows_past_the_arena_limit(tmp_path):
    """An engine that may hold 8 MiB evaluates 20,000 rows (some 120 MiB on the
    device) and keeps none of it afterwards."""
    import torch
    from gagp_b200.engine import Engine
    lt = _task(tmp_path, population=512, seed=34, cases=20)
    rows = oracle.initial_population(abi.GrammarBlob(lt.tables), lt.settings)
    want_f, want_w, _ = oracle.evaluate(abi.GrammarBlob(lt.tables), lt.cases, lt.settings, rows)
    index = np.arange(20000) % 512
    with Engine(0, arena_bytes=8 << 20) as engine:
        engine.evaluate_rows(lt, _take(rows, np.arange(9)))  # the kernels are loaded
        before = torch.cuda.mem_get_info(0)[0]
        f, w = engine.evaluate_rows(lt, _take(rows, index))
        held = before - torch.cuda.mem_get_info(0)[0]
    assert np.array_equal(f, want_f[index]) and np.array_equal(w, want_w[index])
    assert held <= 16 << 20, held


@pytest.mark.gpu
@pytest.mark.parametrize("name,cases,count", [("poly4", 256, 5631), ("polynomial", 21, 16316),
                                              ("list_threshold", 200, 2836), ("list_statements", 200, 1380),
                                              ("grid_paths", 40, 1936)])
def test_static_rows_at_the_limit(name, cases, count):
    """Row counts that just fit the static 32 MiB with rows, bytecode and lists
    of their least size."""
    from gagp_b200.engine import Engine, evaluate_rows_static
    kw = {} if name == "polynomial" else {"cases": cases}
    lt = T.from_files(W.make(name, population=128, generations=2, seed=8, **kw))
    assert len(lt.cases.expected) == cases
    with Engine(0) as engine:
        s = engine.admit(lt)
        s.run()
        rows = s.result_buffer().final_rows
        s.close()
        want_f, want_w = engine.evaluate_rows(lt, rows)
    index = np.arange(count) % rows.count
    f, w = evaluate_rows_static(lt, _take(rows, index))
    assert np.array_equal(f, want_f[index]) and np.array_equal(w, want_w[index])
