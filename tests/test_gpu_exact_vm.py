"""Register code on the exact VM against the interpreter of the reference
bytecode (GPU).

The device lowers list, let, statement and charged programs straight to
register code and sums their fuel per straight-line stretch; the host
harness lowers the same rows to the reference's bytecode and runs it
instruction by instruction (both pinned to the reference by
test_lower_host.py).  Every program must score the same at case counts around
the VM's tiles and at fuels that run out before, inside and after its loops,
and programs with more constants than the VM keeps in slots must too.  All
scores are integers, so the comparison is exact."""
import copy
import glob
import gzip
import json
import os

import numpy as np
import pytest

from gagp_b200 import abi, grammar as G, task as T, workloads as W
from oracle import oracle

import golden_util as GU
import host_harness as H

pytestmark = pytest.mark.gpu
LOWER_DIR = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "lower")
NAMES = sorted(os.path.basename(p)[:-len(".json.gz")] for p in glob.glob(os.path.join(LOWER_DIR, "*.json.gz"))
               if "grid" not in p)


@pytest.fixture(scope="module")
def engine():
    from gagp_b200 import build
    from gagp_b200.engine import Engine
    build.build()
    with Engine(0) as e:
        yield e


def _cycled(cases, n):
    at = np.arange(n) % len(cases.expected)
    return abi.CasesBlob(cases.inputs[at], cases.input_tags, cases.expected[at], cases.expected_tag, cases.list_values)


def _expected(lt, rows, programs, fuel):
    """Fitness and wrong count of each lowered program by the interpreter."""
    cases, penalty = lt.cases, int(abs(lt.settings.penalty))
    fitness, wrong = [], []
    for code, consts, n_locals, _ in programs:
        loss = bad = 0
        for c in range(len(cases.expected)):
            ok, value, tag, _ = H.run(cases, lt.tables.local_types, fuel, code, consts, n_locals, c)
            want = int(cases.expected[c])
            same = ok and tag == cases.expected_tag and value == want
            bad += not same
            if lt.settings.metric == "exact":
                loss += not same
            elif not ok or tag != G.TAG_INT or cases.expected_tag != G.TAG_INT:
                loss += penalty
            else:
                loss += min(abs(value - want), penalty)
        fitness.append(float(-loss))
        wrong.append(bad)
    return fitness, wrong


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("count,fuel", [(1, None), (31, 40), (33, 173), (65, 9)])
def test_register_code_matches_interpreter(engine, name, count, fuel):
    with gzip.open(os.path.join(LOWER_DIR, name + ".json.gz"), "rt") as f:
        fx = json.load(f)
    lt = GU.load_task(fx)
    blob = abi.GrammarBlob(lt.tables)
    picked = [r for r in fx["lower"]["rows"] if r["status"] == 0][:48]
    rows = abi.RowsBuffer.from_rows([(r["origins"], r["constants"]) for r in picked],
                                    lt.tables.max_nodes - lt.tables.fixed_nodes)
    lt.cases = _cycled(lt.cases, count)
    lt.settings.fuel = fuel or lt.settings.fuel
    programs = [H.lower(blob, r["origins"], r["constants"]) for r in picked]
    got_f, got_w = engine.evaluate_rows(lt, rows)
    want_f, want_w = _expected(lt, rows, programs, lt.settings.fuel)
    assert list(got_f) == want_f
    assert list(got_w) == want_w


def test_programs_of_many_constants(engine):
    files = W.list_threshold(population=96, generations=2, seed=11, cases=40)
    grammar = copy.deepcopy(files.grammar)
    for alt in grammar["nonterminals"][2]["alternatives"]:
        if alt["id"] == "one":
            alt["weight"] = 6
            alt["expression"] = {"constant": {"type": "Int", "range": ["-40000000000", "40000000000"]}}
        if alt["id"] in ("add", "sub"):
            alt["weight"] = 8
    files.grammar = grammar
    lt = T.from_files(files)
    blob = abi.GrammarBlob(lt.tables)
    rows = oracle.initial_population(blob, lt.settings)
    assert max(len(set(rows.row(i)[1])) for i in range(rows.count)) > 8
    programs = [H.lower(blob, *rows.row(i)) for i in range(rows.count)]
    got_f, got_w = engine.evaluate_rows(lt, rows)
    want_f, want_w = _expected(lt, rows, programs, lt.settings.fuel)
    assert list(got_f) == want_f
    assert list(got_w) == want_w


@pytest.mark.parametrize("cases", [33, 96])
def test_long_programs(engine, cases):
    """Programs of up to 200 nodes over a modulo that can fail: register code
    past what a warp stages in shared memory, ifs too large for a select."""
    files = W.poly4(population=256, generations=2, seed=3, cases=cases, max_nodes=200)
    grammar = copy.deepcopy(files.grammar)
    for alt in grammar["nonterminals"][0]["alternatives"]:
        alt["weight"] = {"x": 2, "c": 1, "iflt": 3}.get(alt["id"], 2)
        if alt["id"] == "imod0":
            alt["expression"]["signature"] = "mod(Int,Int)->Int"
    files.grammar = grammar
    lt = T.from_files(files)
    blob = abi.GrammarBlob(lt.tables)
    rows = oracle.initial_population(blob, lt.settings)
    assert max(rows.node_counts) > 150
    got_f, got_w = engine.evaluate_rows(lt, rows)
    want_f, want_w, _ = oracle.evaluate(blob, lt.cases, lt.settings, rows)
    assert np.array_equal(got_f, want_f)
    assert np.array_equal(got_w, want_w)


def _statement(lt, name, kind, operand=None):
    """The first expression of a printed name and tree kind (and target)."""
    return next(i for i, e in enumerate(lt.tables.expressions)
                if lt.tables.names[i] == name and e.node_kind == kind and operand in (None, e.operand))


def test_loop_bounds_that_are_no_int(engine):
    """A for_range over a Bool fails the case that reaches it, as the
    bytecode's is_int test does; rows to be scored need not derive from the
    grammar, so they can hold one."""
    lt = T.from_files(W.list_statements(population=64, generations=2, seed=4, cases=70))
    blob = abi.GrammarBlob(lt.tables)
    at = lambda name, kind, operand=None: _statement(lt, name, kind, operand)  # noqa: E731
    main, cons, nil = at("program", G.TK_PROGRAM), at("block_cons", G.TK_BLOCK), at("block_nil", G.TK_NIL)
    acc_is, ret, var = at("assign", G.TK_ASSIGN, 0), at("return", G.TK_RETURN), at("var", G.TK_VAR, 0)
    loop, when, gt = at("for_range", G.TK_FOR_RANGE), at("if_stmt", G.TK_IF), at("gt", G.TK_OPERATION)
    t = next(i for i, e in enumerate(lt.tables.expressions) if e.kind == G.EK_INPUT and lt.tables.names[i] == "t")
    one = next(i for i, e in enumerate(lt.tables.expressions) if e.kind == G.EK_CONSTANT)
    add = at("add", G.TK_OPERATION)
    positive = [gt, t, one]
    body = [cons, acc_is, add, var, one, nil]
    begin, end = [main, cons, acc_is, one], [cons, ret, var, nil]
    rows = [(begin + [cons, loop] + positive + body + end, [5, 0, 1]),        # every case reaches the Bool bound
            (begin + [cons, loop, t] + body + end, [5, 1]),                    # an Int bound, negative ones fail
            (begin + [cons, when] + positive + [cons, loop] + positive + body + [nil, nil] + end, [5, 0, 0, 1])]
    programs = [H.lower(blob, *r) for r in rows]
    buffer = abi.RowsBuffer.from_rows(rows, lt.tables.max_nodes - lt.tables.fixed_nodes)
    got_f, got_w = engine.evaluate_rows(lt, buffer)
    want_f, want_w = _expected(lt, buffer, programs, lt.settings.fuel)
    assert want_w[0] == 70 and want_f[0] < min(want_f[1:])
    assert list(got_f) == want_f
    assert list(got_w) == want_w
    assert [v["runtime_errors"] for v in engine.judge_rows(lt, buffer, lt.cases)][0] == 70


@pytest.mark.parametrize("nested", ["value", "body"])
@pytest.mark.parametrize("lets", [8, 9, 16, 17])
def test_open_lets(engine, nested, lets):
    """Rows of nested lets score up to the reference compiler's 16 open lets
    and are refused past them, also where their slots would fit."""
    with gzip.open(os.path.join(LOWER_DIR, "lower_scalar_let.json.gz"), "rt") as f:
        fx = json.load(f)
    lt = GU.load_task(fx)
    blob = abi.GrammarBlob(lt.tables)
    ex = lt.tables.expressions
    let = next(i for i, e in enumerate(ex) if e.kind == G.EK_OPERATION and e.node_kind == G.TK_LET)
    read = next(i for i, e in enumerate(ex) if e.kind == G.EK_BOUND)
    add = next(i for i, e in enumerate(ex) if e.kind == G.EK_OPERATION and lt.tables.names[i] == "add")
    x = next(i for i, e in enumerate(ex) if e.kind == G.EK_INPUT)
    row = ([let] * lets + [x] + [read] * lets if nested == "value" else [let, x] * lets + [read], [])
    program = H.lower(blob, *row)
    assert (program is None) == (lets > 16)
    buffer = abi.RowsBuffer.from_rows([row], lt.tables.max_nodes - lt.tables.fixed_nodes)
    if program is None:
        with pytest.raises(Exception, match="row evaluation failed"):
            engine.evaluate_rows(lt, buffer)
        return
    got_f, got_w = engine.evaluate_rows(lt, buffer)
    want_f, want_w = _expected(lt, buffer, [program], lt.settings.fuel)
    assert list(got_f) == want_f
    assert list(got_w) == want_w


@pytest.mark.parametrize("lets", [9, 15, 16])
def test_live_locals(engine, lets):
    """Lets nested in one another's values inside five traversals over four
    inputs: the row is refused past the compiler's 64 live locals (nine a
    traversal, one a let), also where its slots would fit."""
    with gzip.open(os.path.join(LOWER_DIR, "lower_list_let.json.gz"), "rt") as f:
        fx = json.load(f)
    fx["grammar"]["search_limits"]["max_nodes"] = 70
    for name in ("u", "v"):
        fx["grammar"]["inputs"].append({"name": name, "type": "Int"})
        for case in fx["train"] + fx["test"]:
            case["inputs"][name] = {"type": "int", "value": 1}
    lt = GU.load_task(fx)
    blob = abi.GrammarBlob(lt.tables)
    ex, names = lt.tables.expressions, lt.tables.names
    let, walk = (next(i for i, e in enumerate(ex) if e.kind == G.EK_OPERATION and e.node_kind == kind)
                 for kind in (G.TK_LET, G.TK_TRAVERSE))
    xs, t = (next(i for i, e in enumerate(ex) if e.kind == G.EK_INPUT and names[i] == name) for name in ("xs", "t"))
    read = next(i for i, e in enumerate(ex) if e.kind == G.EK_BOUND and e.operand == ex[let].operand)
    row = ([walk, xs, t, t] * 5 + [let] * lets + [t] + [read] * lets, [])
    program = H.lower(blob, *row)
    assert (program is None) == (4 + 45 + lets > 64)
    buffer = abi.RowsBuffer.from_rows([row], lt.tables.max_nodes - lt.tables.fixed_nodes)
    if program is None:
        with pytest.raises(Exception, match="row evaluation failed"):
            engine.evaluate_rows(lt, buffer)
        return
    lt.settings.fuel = 600  # some cases finish their nested loops
    got_f, got_w = engine.evaluate_rows(lt, buffer)
    want_f, want_w = _expected(lt, buffer, [program], lt.settings.fuel)
    assert list(got_f) == want_f
    assert list(got_w) == want_w


@pytest.mark.parametrize("lists", [7, 8, 9, 12, 15, 16, 30])
def test_programs_of_many_list_inputs(engine, lists):
    """A fold whose step adds the lengths of every other list input: with and
    without slots for the lengths, and past the slots altogether."""
    files = W.list_threshold(population=64, generations=2, seed=6, cases=40, max_nodes=100)
    grammar = copy.deepcopy(files.grammar)
    others = [f"y{j}" for j in range(lists - 1)]
    grammar["inputs"] += [{"name": y, "type": "IntList"} for y in others]
    step = next(nt for nt in grammar["nonterminals"] if nt["id"] == "Step")
    step["alternatives"] += [{"id": "len_" + y, "weight": 1,
                              "expression": {"signature": "len(IntList)->Int", "args": [{"input": y}]}} for y in others]
    for k, case in enumerate(files.train):
        for j, y in enumerate(others):
            case["inputs"][y] = {"type": "int_list", "value": list(range((k * (j + 2)) % 7))}
    files.grammar = grammar
    lt = T.from_files(files)
    blob = abi.GrammarBlob(lt.tables)
    ex, names = lt.tables.expressions, lt.tables.names
    at = lambda name, kind: next(i for i, e in enumerate(ex) if names[i] == name and e.kind == kind)  # noqa: E731
    length, add = at("len", G.EK_OPERATION), at("add", G.EK_OPERATION)
    body = [at("acc", G.EK_BOUND), at("element", G.EK_BOUND)]
    for y in others:
        body = [add] + body + [length, at(y, G.EK_INPUT)]
    row = ([at("traverse", G.EK_OPERATION), at("xs", G.EK_INPUT), at("const", G.EK_CONSTANT), at("t", G.EK_INPUT),
            add] + body, [0])
    program = H.lower(blob, *row)
    buffer = abi.RowsBuffer.from_rows([row], lt.tables.max_nodes - lt.tables.fixed_nodes)
    for fuel in (200, lt.settings.fuel):
        lt.settings.fuel = fuel
        got_f, got_w = engine.evaluate_rows(lt, buffer)
        want_f, want_w = _expected(lt, buffer, [program], fuel)
        assert list(got_f) == want_f
        assert list(got_w) == want_w
