"""Steady-state placement against the oracle (GPU) at the sizes where its form
changes: the placement levels in one block (rounds and populations of at most
2048) or a cluster, the placement in one block (1 or 4 children a thread) or,
from 4096 children, a cluster; and several of them in one batch."""
import pytest

from gagp_b200 import abi, task as T, workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu

# (population, children per round)
SHAPES = [(2, 2), (3, 3), (31, 31), (1023, 1023), (1024, 1024), (1025, 1025), (2047, 2047), (2048, 2048), (2049, 2049),
          (4095, 4095), (4096, 4096), (4097, 4097), (4096, 1024), (4096, 2048), (8192, 4096), (6000, 3000)]


@pytest.fixture(scope="module")
def engine():
    from gagp_b200 import build
    from gagp_b200.engine import Engine
    build.build()
    e = Engine(0)
    yield e
    e.close()


def _task(tmp_path, population, children):
    files = W.poly4(population=population, generations=4, seed=population + children, cases=9, max_nodes=24)
    if children != population:
        files.search["schedule"] = {"mode": "steady_state", "batch": children}
    return T.load(files.write(str(tmp_path)), str(tmp_path / "search.json"))


def _check(lt, got):
    want = oracle.search(abi.GrammarBlob(lt.tables), lt.cases, lt.settings, member_reuse=True)
    assert got["history"] == want["history"]
    assert got["final"] == want["final"]
    assert got["reused_programs"] == want["reused_programs"]


@pytest.mark.parametrize("population,children", SHAPES)
def test_placement_matches_oracle(engine, tmp_path, population, children):
    lt = _task(tmp_path, population, children)
    s = engine.admit(lt)
    try:
        s.run()
        _check(lt, s.result())
    finally:
        s.close()


def test_placements_of_several_sizes_in_one_batch(engine, tmp_path):
    tasks = [_task(tmp_path / str(p), p, p) for p in (31, 1025, 2048, 2049, 4097)]
    searches = [engine.admit(lt) for lt in tasks]
    try:
        engine.run_batch(searches)
        for lt, s in zip(tasks, searches):
            _check(lt, s.result())
    finally:
        for s in searches:
            s.close()
