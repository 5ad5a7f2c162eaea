"""The accumulator VM against the oracle (GPU): every operation and operand
class, with one, two and three inputs, at case counts around its lane tiling
(1, 2 and 4 cases per lane), and its division at the edges of the range that
takes the estimated quotient."""
import random

import numpy as np
import pytest

from gagp_b200 import abi, task as T, workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu

DIVISIONS = ("idiv0", "imod0", "trunc_div0", "trunc_mod0")
NARROW = 1 << 30


def _grammar(inputs):
    ref, test = {"ref": "Expr"}, {"ref": "Test"}
    two = lambda op, a, t, r: {"signature": f"{op}({t},{t})->{r}", "args": [a, a]}  # noqa: E731
    alt = [{"id": f"in_{n}", "weight": 2, "expression": {"input": n}} for n in inputs]
    alt.append({"id": "c", "weight": 2, "expression": {"constant": {"type": "Int", "range": ["-3", "5"]}}})
    alt += [{"id": op, "weight": 1, "expression": two(op, ref, "Int", "Int")}
            for op in ("add", "sub", "mul", "min", "max") + DIVISIONS]
    alt += [{"id": op, "weight": 1, "expression": {"signature": f"{op}(Int)->Int", "args": [ref]}}
            for op in ("neg", "abs")]
    alt.append({"id": "if", "weight": 2, "expression": {"signature": "if(Bool,Int,Int)->Int", "args": [test, ref, ref]}})
    tests = [{"id": op, "weight": 2, "expression": two(op, ref, "Int", "Bool")}
             for op in ("lt", "le", "gt", "ge", "eq", "ne")]
    tests.append({"id": "not", "weight": 1, "expression": {"signature": "not(Bool)->Bool", "args": [test]}})
    return {"format_version": "grammar-definition-v2", "entry": {"nonterminal": "Expr", "type": "Int"},
            "inputs": [{"name": n, "type": "Int"} for n in inputs],
            "search_limits": {"max_nodes": 48, "max_depth": 10}, "execution_limits": {"fuel": 1000},
            "nonterminals": [{"id": "Expr", "type": "Int", "scope": [], "alternatives": alt},
                             {"id": "Test", "type": "Bool", "scope": [], "alternatives": tests}]}


def _task(tmp_path, inputs, values, expected):
    train = [{"inputs": {n: {"type": "int", "value": int(v)} for n, v in zip(inputs, row)},
              "expected": {"type": "int", "value": int(e)}} for row, e in zip(values, expected)]
    files = W.TaskFiles(name="accumulator", grammar=_grammar(inputs), train=train,
                        fitness={"metric": "absolute", "case_cap": 2147483647}, search=W.search_config(400, 2, 7))
    return T.load(files.write(str(tmp_path)), str(tmp_path / "search.json"))


def _compare(lt, rows):
    from gagp_b200.engine import Engine
    want_f, want_w, _ = oracle.evaluate(abi.GrammarBlob(lt.tables), lt.cases, lt.settings, rows)
    with Engine(0) as engine:
        f, w = engine.evaluate_rows(lt, rows)
    assert np.array_equal(f, want_f) and np.array_equal(w, want_w)


@pytest.mark.parametrize("cases", [1, 32, 33, 64, 65, 128, 129, 515])
@pytest.mark.parametrize("inputs", ["x", "xy", "xyz"])
def test_every_operation(tmp_path, inputs, cases):
    rng = random.Random(cases)
    value = lambda: rng.choice([rng.randint(-9, 9), rng.randint(-NARROW, NARROW), rng.randint(-(1 << 62), 1 << 62)])  # noqa: E731
    lt = _task(tmp_path, inputs, [[value() for _ in inputs] for _ in range(cases)], [value() for _ in range(cases)])
    _compare(lt, oracle.initial_population(abi.GrammarBlob(lt.tables), lt.settings))


@pytest.mark.parametrize("cases", [32, 64, 4096])
def test_division_at_the_edges_of_the_estimated_range(tmp_path, cases):
    rng = random.Random(3)
    edges = [0, 1, 2, 3, 7, 10, 1 << 15, (1 << 20) - 1, 1 << 20, (1 << 24) + 1, NARROW - 2, NARROW - 1]
    edges = [s * v for v in edges for s in (1, -1)] + [-NARROW]
    inside = [(a, b) for a in edges for b in edges]  # 625 pairs
    inside += [(rng.randint(-NARROW, NARROW - 1), rng.randint(-(1 << rng.randint(1, 30)), (1 << rng.randint(1, 30)) - 1))
               for _ in range(2047 - len(inside))]
    outside = edges + [NARROW, -NARROW - 1, (1 << 31) - 1, 1 << 31, -(1 << 31), -(1 << 31) - 1, (1 << 63) - 1, -(1 << 63)]
    outside = [(a, b) for a in outside for b in outside]
    pairs = inside + [(0, 0)] + outside  # tiles of 128 inside the range first
    pairs = (pairs if cases > 64 else rng.sample(inside, cases))[:cases]
    expected = [rng.randint(-NARROW, NARROW) // (1 << rng.randint(0, 30)) for _ in pairs]
    lt = _task(tmp_path, "xy", pairs, expected)
    op = lt.tables.names.index
    x, y, constant = op("x"), op("y"), op("const")
    rows = []
    for d in DIVISIONS:
        rows.append(([op(d), x, y], []))                             # input operand
        rows.append(([op(d), x, op("add"), y, constant], [0]))       # reversed: the accumulator divides an input
        rows.append(([op(d), op("add"), x, y, op("sub"), x, y], []))  # temporary operand
        rows.append(([op(d), x, constant], [-7]))
        rows.append(([op(d), constant, y], [NARROW - 1]))
        rows.append(([op(d), x, x], []))
    _compare(lt, abi.RowsBuffer.from_rows(rows, lt.tables.max_nodes - lt.tables.fixed_nodes))

