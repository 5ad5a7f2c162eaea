"""Which VMs a grammar's programs can need (vm_choice.cuh).

Where the rule says that no program can need the exact VM, a row that the
accumulator lowering rejects is an error, so the rule must be right at each
of its edges: node kinds without an accumulator operation (lets and bounded
regions that nothing reads from), the node budget at which a program can need
a seventh temporary, and the fuel that bounds every bytecode.  On the GPU the
rows at those edges score as the interpreter of the reference bytecode does
(pinned to the reference by test_lower_host.py); all scores are integers, so
the comparison is exact."""
import copy
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from gagp_b200 import abi, grammar as G, task as T, workloads as W

import host_harness as H

SOURCE = os.path.join(H.HERE, "native", "vm_choice_host.cu")
LIB = os.path.join(H.HERE, "_build", "libvm_choice_host.so")
CSRC = os.path.join(H.ROOT, "gagp_b200", "csrc")
DEPS = [SOURCE, os.path.join(H.ROOT, "include", "gagp_b200.h")] + \
    [os.path.join(CSRC, f) for f in ("vm_choice.cuh", "lower.cuh", "device_ops.cuh", "search_state.h")]


@pytest.fixture(scope="module")
def rule():
    if not os.path.exists(LIB) or any(os.path.getmtime(d) > os.path.getmtime(LIB) for d in DEPS):
        from gagp_b200.build import nvcc
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        subprocess.run([nvcc(), "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a",
                        "-Xcompiler", "-fPIC", "-shared", SOURCE, "-o", LIB], check=True)
    return C.CDLL(LIB)


@pytest.fixture(scope="module")
def engine():
    from gagp_b200 import build
    from gagp_b200.engine import Engine
    build.build()
    with Engine(0) as e:
        yield e


def _unread_let(**kwargs):
    """The large scalar grammar with a let whose name nothing reads."""
    files = W.poly4(**kwargs)
    files.grammar = copy.deepcopy(files.grammar)
    ref = {"ref": "Expr"}
    files.grammar["nonterminals"][0]["alternatives"].append(
        {"id": "let", "weight": 2, "expression": {"signature": "let(Int,Int)->Int", "args": [ref, ref],
                                                  "bind": {"1": ["y"]}}})
    return T.from_files(files)


def _unread_region(**kwargs):
    """The lattice paths with phases that read none of their bindings."""
    files = W.grid_paths(**kwargs)
    files.grammar = copy.deepcopy(files.grammar)
    ref = lambda n: {"ref": n}  # noqa: E731
    small = {"constant": {"type": "Int", "values": ["0", "1", "2"]}}
    binary = lambda op, t, a: {"signature": f"{op}(Int,Int)->{t}", "args": [a, a]}  # noqa: E731
    alternatives = {
        "Test": [{"id": "lt", "weight": 1, "expression": binary("lt", "Bool", small)}],
        "Base": [{"id": "k", "weight": 2, "expression": small},
                 {"id": "sub", "weight": 1, "expression": binary("sub", "Int", ref("Base"))}],
        "Join": [{"id": "k", "weight": 2, "expression": small},
                 {"id": "max", "weight": 1, "expression": binary("max", "Int", ref("Join"))}]}
    for nt in files.grammar["nonterminals"]:
        nt["alternatives"] = alternatives.get(nt["id"], nt["alternatives"])
    return T.from_files(files)


def _deep(max_nodes, cases=40):
    """Ints and Bools, unary operations and ifs over both: the grammar with the
    smallest trees of a given need of temporaries."""
    files = W.poly4(population=64, generations=2, seed=5, cases=cases)
    e, b = {"ref": "Expr"}, {"ref": "Cond"}
    files.grammar = {
        "format_version": "grammar-definition-v2", "entry": {"nonterminal": "Expr", "type": "Int"},
        "inputs": [{"name": "x", "type": "Int"}, {"name": "flag", "type": "Bool"}],
        "search_limits": {"max_nodes": max_nodes, "max_depth": 16}, "execution_limits": {"fuel": 1000},
        "nonterminals": [
            {"id": "Expr", "type": "Int", "scope": [], "alternatives": [
                {"id": "x", "weight": 2, "expression": {"input": "x"}},
                {"id": "neg", "weight": 1, "expression": {"signature": "neg(Int)->Int", "args": [e]}},
                {"id": "sub", "weight": 1, "expression": {"signature": "sub(Int,Int)->Int", "args": [e, e]}},
                {"id": "if", "weight": 1, "expression": {"signature": "if(Bool,Int,Int)->Int", "args": [b, e, e]}}]},
            {"id": "Cond", "type": "Bool", "scope": [], "alternatives": [
                {"id": "flag", "weight": 2, "expression": {"input": "flag"}},
                {"id": "not", "weight": 1, "expression": {"signature": "not(Bool)->Bool", "args": [b]}},
                {"id": "if", "weight": 1, "expression": {"signature": "if(Bool,Bool,Bool)->Bool",
                                                         "args": [b, b, b]}}]}]}
    for k, case in enumerate(files.train):
        case["inputs"]["flag"] = {"type": "bool", "value": k % 3 == 0}
        case["expected"] = {"type": "int", "value": 3 * k - 50}
    return T.from_files(files)


def _variable_nodes(lt):
    return lt.tables.max_nodes - lt.tables.fixed_nodes


def _deep_with(variable_nodes):
    lt = _deep(64)
    return _deep(variable_nodes + lt.tables.fixed_nodes)


def _needy_row(lt, need):
    """A smallest row that needs `need` temporaries (even, or odd by a
    subtraction of two of one less)."""
    def find(name, tag):
        return next(i for i, e in enumerate(lt.tables.expressions)
                    if lt.tables.names[i] == name and e.kind != G.EK_REFERENCE and e.type == tag)

    ex = lt.tables.expressions
    leaf = {tag: next(i for i, e in enumerate(ex) if e.kind == G.EK_INPUT and lt.tables.names[i] == name)
            for tag, name in ((G.TAG_INT, "x"), (G.TAG_BOOL, "flag"))}
    unary = {G.TAG_INT: find("neg", G.TAG_INT), G.TAG_BOOL: find("not", G.TAG_BOOL)}
    chooses = {tag: next(i for i, e in enumerate(ex) if e.kind == G.EK_OPERATION and e.node_kind == G.TK_IF
                         and _target_leaf(lt, e.children[1]) == leaf[tag])
               for tag in (G.TAG_INT, G.TAG_BOOL)}

    def tree(k, tag):
        if k == 0:
            return [unary[tag], leaf[tag]]
        return [chooses[tag]] + tree(k - 2, G.TAG_BOOL) + tree(k - 2, tag) + tree(k - 2, tag)

    if need % 2 == 0:
        return tree(need, G.TAG_INT)
    return [find("sub", G.TAG_INT)] + 2 * tree(need - 1, G.TAG_INT)


def _target_leaf(lt, reference):
    """The input expression among a reference's productions."""
    off, count = lt.tables.nonterminals[lt.tables.expressions[reference].target][:2]
    return next(x for x, _ in lt.tables.productions[off:off + count]
                if lt.tables.expressions[x].kind == G.EK_INPUT)


def _expected(lt, rows, fuel):
    """Fitness and wrong count of each row by the interpreter of its bytecode."""
    blob, cases, penalty = abi.GrammarBlob(lt.tables), lt.cases, int(abs(lt.settings.penalty))
    fitness, wrong = [], []
    for origins, constants in rows:
        code, consts, n_locals, _, n_main, main_consts = H.lower(blob, origins, constants, shape=True)
        loss = bad = 0
        for c in range(len(cases.expected)):
            if n_main < len(code):
                ok, value, tag, _ = H.run_regions(blob, cases, fuel, code, n_main, consts, main_consts, n_locals, c)
            else:
                ok, value, tag, _ = H.run(cases, lt.tables.local_types, fuel, code, consts, n_locals, c)
            want = int(cases.expected[c])
            bad += not (ok and tag == cases.expected_tag and value == want)
            loss += min(abs(value - want), penalty) if ok and tag == G.TAG_INT else penalty
        fitness.append(float(-loss))
        wrong.append(bad)
    return fitness, wrong


def _check_rows(engine, lt, rows):
    got_f, got_w = engine.evaluate_rows(lt, abi.RowsBuffer.from_rows(rows, _variable_nodes(lt)))
    want_f, want_w = _expected(lt, rows, lt.settings.fuel)
    assert list(got_f) == want_f
    assert list(got_w) == want_w


def test_rule_over_grammars(rule):
    def possible(lt, fuel=None):
        return bool(rule.host_exact_possible(abi.GrammarBlob(lt.tables).ref(), fuel or lt.tables.fuel))

    small = dict(population=64, generations=2, cases=20)
    assert not possible(T.from_files(W.polynomial(population=64, generations=2)))
    assert not possible(T.from_files(W.poly4(**small)))
    for make in (W.list_threshold, W.list_statements, W.grid_paths):
        assert possible(T.from_files(make(**small)))
    assert possible(_unread_let(**small))
    assert possible(_unread_region(**small))
    assert not possible(_deep_with(134))
    assert possible(_deep_with(135))
    lt = _deep_with(60)
    bound = rule.host_bytecode_bound(abi.GrammarBlob(lt.tables).ref())
    assert not possible(lt, bound)
    assert possible(lt, bound - 1)


def test_smallest_tree_of_each_need():
    """The fewest nodes of a tree of each need, by growing trees of every need
    from smaller ones with lower_accumulator_emit's formula: the children that
    are no leaves in decreasing need, the largest of need + position."""
    best = {0: 2}  # a unary operation over a leaf
    while True:
        grown = dict(best)
        items = [(None, 1)] + list(best.items())
        for arity in (1, 2, 3):
            def grow(chosen, nodes):
                if len(chosen) == arity:
                    needs = sorted((n for n in chosen if n is not None), reverse=True)
                    need = max([n + k for k, n in enumerate(needs)], default=0)
                    if need <= 8 and nodes + 1 < grown.get(need, 1 << 30):
                        grown[need] = nodes + 1
                    return
                for n, size in items:
                    grow(chosen + [n], nodes + size)
            grow([], 0)
        if grown == best:
            break
        best = grown
    assert min(size for need, size in best.items() if need > 6) == 135
    assert [best[k] for k in range(8)] == [2, 5, 7, 15, 22, 45, 67, 135]


@pytest.mark.gpu
def test_rows_with_an_unread_let(engine):
    lt = _unread_let(population=64, generations=2, seed=9, cases=33)
    names = lt.tables.names
    ex = lt.tables.expressions
    let = next(i for i, e in enumerate(ex) if e.node_kind == G.TK_LET and e.kind == G.EK_OPERATION)
    add = next(i for i, e in enumerate(ex) if names[i] == "add" and e.kind == G.EK_OPERATION)
    x = next(i for i, e in enumerate(ex) if e.kind == G.EK_INPUT)
    k = next(i for i, e in enumerate(ex) if e.kind == G.EK_CONSTANT)
    rows = [([let, x, k], [2]), ([add, let, k, x, let, x, x], [-1]), ([let, let, x, x, add, x, k], [3]), ([x], [])]
    _check_rows(engine, lt, rows)


@pytest.mark.gpu
@pytest.mark.parametrize("make", [_unread_let, _unread_region], ids=["let", "region"])
def test_search_with_unread_bindings(engine, make):
    lt = make(population=96, generations=4, seed=3, cases=24)
    s = engine.admit(lt)
    try:
        s.run()
        result = s.result_buffer()
    finally:
        s.close()
    rows = [result.final_rows.row(i) for i in range(result.final_rows.count)]
    structured = {G.TK_LET, G.TK_REGION}
    assert any(lt.tables.expressions[o].node_kind in structured for r in rows for o in r[0])
    want_f, _ = _expected(lt, rows, lt.settings.fuel)
    assert list(result.final_fitness) == want_f


@pytest.mark.gpu
@pytest.mark.parametrize("nodes", [134, 135])
def test_rows_at_the_temporaries_limit(engine, nodes):
    lt = _deep_with(nodes)
    rows = [(_needy_row(lt, need), []) for need in (0, 2, 5, 6, 7)]
    assert [len(r[0]) for r in rows] == [2, 7, 45, 67, 135]
    _check_rows(engine, lt, [r for r in rows if len(r[0]) <= nodes])


@pytest.mark.gpu
@pytest.mark.parametrize("below", [0, 1])
def test_rows_at_the_fuel_bound(engine, rule, below):
    lt = _deep_with(60)
    blob = abi.GrammarBlob(lt.tables)
    row = (_needy_row(lt, 5), [])
    lt.settings.fuel = rule.host_bytecode_bound(blob.ref()) - below
    _check_rows(engine, lt, [row])
    # the row's own longest path, and one unit less
    lt.settings.fuel = len(H.lower(blob, *row)[0]) - below
    _check_rows(engine, lt, [row])
