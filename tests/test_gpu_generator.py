"""Subtree generation's draw tables at their edges against the oracle (GPU).

A nonterminal of more productions than a warp has lanes (one of next to no
weight, the last one a leaf), constant domains of one value, of a width past
32 bits and of every Int, and a node budget that takes the narrower draw
levels; each a whole small search, so that the initial population (a thread per
member) and the mutations (a warp per child) both draw from the tables.
Everything is an integer: the comparison is exact.  (The productions' root
nodes differ: the engine re-derives the initial rows of an ambiguous grammar,
which the oracle does not.)"""
import pytest

from gagp_b200 import abi, task as T, workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu
RANGES = {"one": ("7", "7"), "every": ("-9223372036854775808", "9223372036854775807"), "wide": ("0", "1099511627777"),
          "small": ("-3", "61")}


def _files(inputs, domain, max_nodes):
    files = W.poly4(population=96, generations=4, seed=inputs, cases=9)
    g = W.poly4_grammar(max_nodes=max_nodes)
    names = ["x%02d" % i for i in range(inputs)]
    g["inputs"] = [{"name": n, "type": "Int"} for n in names]
    operations = g["nonterminals"][0]["alternatives"][2:]
    leaves = [{"id": n, "weight": 1 + i % 3, "expression": {"input": n}} for i, n in enumerate(names)]
    constant = {"id": "c", "weight": 5, "expression": {"constant": {"type": "Int", "range": list(RANGES[domain])}}}
    operations[1] = dict(operations[1], weight=1e-6)
    g["nonterminals"][0]["alternatives"] = [constant] + [dict(o, weight=o["weight"] * inputs / 3) for o in operations] + leaves
    files.grammar = g
    files.train = [{"inputs": {n: {"type": "int", "value": (7 * c + i) % 23 - 11} for i, n in enumerate(names)},
                    "expected": {"type": "int", "value": c * c}} for c in range(9)]
    files.search["mutation"] = {"probability": 0.9}
    return files


@pytest.mark.parametrize("inputs,domain,max_nodes", [(1, "every", 24), (24, "one", 40), (26, "wide", 64), (50, "small", 12)])
def test_draw_tables_match_oracle(inputs, domain, max_nodes):
    from gagp_b200 import build
    from gagp_b200.engine import Engine
    build.build()
    lt = T.from_files(_files(inputs, domain, max_nodes))
    with Engine(0) as eng:
        s = eng.admit(lt)
        s.run()
        got = s.result()
        s.close()
    want = oracle.search(abi.GrammarBlob(lt.tables), lt.cases, lt.settings)
    assert got["history"] == want["history"]
    assert got["final"] == want["final"]
