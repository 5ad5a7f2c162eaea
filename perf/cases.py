"""The calls that programs make of this engine, as cases that can be timed.

A case is one call sequence through the public Python front end
(``gagp_b200.engine``), on tasks of ``gagp_b200.workloads``:

* ``score_static``  rows scored without device allocation (``evaluate_rows_static``): the smallest call,
  a program that scores a handful of candidates in a loop of its own.
* ``score``         rows scored on a case set (``Engine.evaluate_rows``): a saved population on new cases.
* ``judge``         verdicts of the best rows on a test split (``Engine.judge_rows``), what follows a run.
* ``search``        one whole search: admitted, run, its result read, released.  Steady state or
  generational with elites, absolute or exact metric, generated or imported population; scalar, list,
  statement and bounded-region grammars.
* ``batch``         many searches of one mix advanced together, half scalar and half list programs.
* ``serve``         a request stream through the continuous-batching server, a few requests per step.

A program keeps its engine (and a service its server's engine) for its whole
life, so those are made once per process; tasks are loaded before the call.
"""
import math
import os
import random

# the engine's rounds run on many CUDA streams: give each a hardware work queue
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

import numpy as np  # noqa: E402

from gagp_b200 import abi, task as T, workloads as W  # noqa: E402
from gagp_b200.engine import Engine, Server, evaluate_rows_static  # noqa: E402

_engine = None
_tables = {}  # compiled phase tables by grammar, as a program that loads many tasks of one grammar shares them


def _one_engine():
    global _engine
    if _engine is None:
        _engine = Engine(0)
    return _engine


def _task(case, seed, population=None, generations=None):
    """A loaded task of the case's workload, its cases and its search seeded by `seed`."""
    args = dict(population=population or case["population"], generations=generations or case["generations"], seed=seed)
    if case["workload"] != "polynomial":
        args["cases"] = case["cases"]
    if case["workload"].startswith("list"):
        args["target"] = W.LIST_TARGETS[case.get("target", 0)]
    files = W.make(case["workload"], **args)
    if case.get("generational"):
        files.search["schedule"] = {"mode": "generational"}
        files.search["elitism"] = case["elites"]
        files.search["selection"] = {"method": "tournament", "size": case["tournament"]}
    if case.get("exact_metric"):
        files.fitness = {"metric": "exact", "case_cap": 1000}
    if case["workload"] == "polynomial":
        # the 21 points are the benchmark task's, the cubic's coefficients the seed's
        a, b, c = 1 + seed % 5, seed // 5 % 7 - 3, seed // 35 % 9 - 4
        files.train = [W._int_case(x, a * x ** 3 + b * x + c) for x in range(-10, 11)]
    return T.from_files(files, table_cache=_tables)


def _saved_rows(case, task_seed, count):
    """Rows of a population a few generations old, in rank order: what a program loads to score, judge or resume."""
    eng = _one_engine()
    early = _task(dict(case, generational=False, exact_metric=False), task_seed, population=max(count, 64), generations=6)
    s = eng.admit(early)
    try:
        s.run()
        res = s.result_buffer()
    finally:
        s.close()
    rows = abi.RowsBuffer(count, res.final_rows.stride)
    for name in ("node_counts", "origins", "constant_counts", "constants"):
        getattr(rows, name)[:] = getattr(res.final_rows, name)[:count]
    return rows


def _mix(case, seed):
    """The requests of a batch or a service: alternately scalar regressions and list programs, sizes spread over the range."""
    rng = random.Random(1000003 * case["count"] + case["largest_population"] + case["most_cases"])
    tasks = []
    for i in range(case["count"]):
        p = int(256 * (case["largest_population"] / 256) ** rng.random())
        one = {"workload": "poly4" if i % 2 == 0 else "list_threshold", "target": i // 2 % 3, "population": p,
               "cases": rng.randint(16, case["most_cases"]),
               "generations": rng.randint(case["generations"] // 2, case["generations"]) if case["kind"] == "serve"
               else case["generations"]}
        tasks.append(_task(one, 1000 * seed + i))
    return tasks


def listed():
    return [
        # a handful of candidates scored in a program's own loop: launches and copies
        {"name": "score_static_small", "kind": "score_static", "workload": "polynomial", "rows": 32, "cases": 21},
        # a saved population scored on a large case set: the accumulator VM
        {"name": "score_poly4_large", "kind": "score", "workload": "poly4", "rows": 16384, "cases": 2000},
        # the best rows of a list run judged on its test split: the exact VM on few programs
        {"name": "judge_list", "kind": "judge", "workload": "list_threshold", "target": 1, "rows": 200, "cases": 1000},
        # a short continuation of a small saved population, odd sizes: host work and launches
        {"name": "search_resume_small", "kind": "search", "workload": "poly4", "population": 777, "generations": 24,
         "cases": 101, "imported": True},
        # the default search of the smallest benchmark task
        {"name": "search_polynomial", "kind": "search", "workload": "polynomial", "population": 1024,
         "generations": 64, "cases": 21},
        # the benchmark's headline search
        {"name": "search_poly4", "kind": "search", "workload": "poly4", "population": 16384, "generations": 128,
         "cases": 256},
        # generational schedule with elites, larger tournaments, the exact metric, odd sizes
        {"name": "search_generational", "kind": "search", "workload": "poly4", "population": 5001, "generations": 50,
         "cases": 1000, "generational": True, "elites": 3, "tournament": 3, "exact_metric": True},
        # the benchmark's list-program search
        {"name": "search_list", "kind": "search", "workload": "list_threshold", "target": 0, "population": 8192,
         "generations": 96, "cases": 200},
        # statement programs: loops and branches over the list cases
        {"name": "search_statements", "kind": "search", "workload": "list_statements", "target": 2, "population": 2048,
         "generations": 48, "cases": 200},
        # bounded regions: evolved recurrences on the frame-stack executor
        {"name": "search_grid_paths", "kind": "search", "workload": "grid_paths", "population": 1024,
         "generations": 32, "cases": 40},
        # a batch of mixed searches, as a hyper-parameter or seed sweep runs them
        {"name": "batch_mix", "kind": "batch", "count": 32, "largest_population": 4096, "most_cases": 1000,
         "generations": 32},
        # a service: requests of mixed sizes arriving while others run
        {"name": "serve_mix", "kind": "serve", "count": 24, "largest_population": 2048, "most_cases": 500,
         "generations": 48, "arrivals": 3, "rounds_per_step": 8},
    ]


def _spread(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["score_static", "score", "judge", "search", "search", "search", "search", "batch", "serve"])
    if kind == "score_static":
        return {"kind": kind, "workload": "poly4", "rows": _spread(rng, 16, 600), "cases": _spread(rng, 16, 300)}
    if kind == "score":
        return {"kind": kind, "workload": rng.choice(["poly4", "poly4", "list_threshold"]),
                "rows": _spread(rng, 64, 4096), "cases": _spread(rng, 16, 1000)}
    if kind == "judge":
        return {"kind": kind, "workload": rng.choice(["poly4", "list_threshold", "list_statements"]),
                "rows": _spread(rng, 8, 256), "cases": _spread(rng, 100, 1000)}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(4, 32), "largest_population": _spread(rng, 400, 4096),
                "most_cases": _spread(rng, 50, 900), "generations": rng.randint(8, 32)}
    if kind == "serve":
        return {"kind": kind, "count": rng.randint(6, 24), "largest_population": _spread(rng, 400, 2048),
                "most_cases": _spread(rng, 50, 500), "generations": rng.randint(16, 48),
                "arrivals": rng.randint(1, 4), "rounds_per_step": rng.choice([1, 4, 8])}
    workload = rng.choice(["poly4", "poly4", "list_threshold", "list_threshold", "list_statements", "grid_paths"])
    top = {"poly4": (16384, 2000, 128), "list_threshold": (8192, 200, 96), "list_statements": (4096, 200, 48),
           "grid_paths": (2048, 60, 32)}[workload]
    case = {"kind": "search", "workload": workload, "population": _spread(rng, 256, top[0]),
            "cases": _spread(rng, 16, top[1]), "generations": _spread(rng, 12, top[2])}
    if workload.startswith("list"):
        case["target"] = rng.randrange(3)
    if rng.random() < 0.25:
        case.update(generational=True, elites=rng.randint(0, 4), tournament=rng.randint(2, 4))
    if rng.random() < 0.25:
        case["exact_metric"] = True
    if rng.random() < 0.2 and workload != "grid_paths":
        case["imported"] = True
    return case


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": case, "engine": _one_engine()}
    if kind in ("score", "score_static", "judge"):
        # the rows come from a short search of one task, the cases scored from another seed's
        state["task"] = _task(case, seed + 7, population=max(case["rows"], 64), generations=6)
        state["rows"] = _saved_rows(case, seed, case["rows"])
    elif kind == "search":
        state["task"] = _task(case, seed)
        state["initial"] = _saved_rows(case, seed + 7, case["population"]) if case.get("imported") else None
    else:
        state["tasks"] = _mix(case, seed)
    return state


def _outputs(results):
    """The whole results of one or more searches."""
    out = {}
    for name in ("history_best_fitness", "history_mean_fitness", "history_best_wrong", "history_best_nodes",
                 "final_fitness", "final_wrong", "final_nodes"):
        out[name] = [getattr(r, name) for r in results]
    for name in ("node_counts", "origins", "constant_counts", "constants"):
        out["best_" + name] = [getattr(r.history_best, name) for r in results]
        out["final_" + name] = [getattr(r.final_rows, name) for r in results]
    out["counts"] = [np.array([r.struct.evaluated_programs, r.struct.reused_programs, r.struct.program_cases],
                              dtype=np.uint64).astype(np.int64) for r in results]
    if len(results) == 1:
        return {k: v[0] for k, v in out.items()}
    return {k: np.concatenate([x.reshape(-1) for x in v]) for k, v in out.items()}


def _serve(state):
    case, tasks = state["case"], state["tasks"]
    tickets = []
    with Server(state["engine"], rounds_per_step=case["rounds_per_step"]) as server:
        waiting = True
        while waiting or len(tickets) < len(tasks):
            for task in tasks[len(tickets):len(tickets) + case["arrivals"]]:
                tickets.append(server.submit(task))
            running, queued, _ = server.step()
            waiting = running + queued > 0
        return _outputs([server.result_buffer(t) for t in tickets])


def run(state):
    kind, eng = state["kind"], state["engine"]
    if kind == "score_static":
        return evaluate_rows_static(state["task"], state["rows"])
    if kind == "score":
        return eng.evaluate_rows(state["task"], state["rows"])
    if kind == "judge":
        verdicts = eng.judge_rows(state["task"], state["rows"], state["task"].cases)
        return np.array([[v["correct"], v["wrong"], v["runtime_errors"], v["mean_loss"]] for v in verdicts])
    if kind == "search":
        s = eng.admit(state["task"], state["initial"])
        try:
            s.run()
            return _outputs([s.result_buffer()])
        finally:
            s.close()
    if kind == "serve":
        return _serve(state)
    searches = [eng.admit(t) for t in state["tasks"]]
    try:
        eng.run_batch(searches)
        return _outputs([s.result_buffer() for s in searches])
    finally:
        for s in searches:
            s.close()


# Integer operations one program costs on one case: its instructions, and for
# the list grammars those times the list's mean length.
_OPERATIONS = {"polynomial": 8, "poly4": 12, "list_threshold": 250, "list_statements": 80, "grid_paths": 200}
_INPUT_BYTES = {"polynomial": 16, "poly4": 16, "list_threshold": 8 * 29, "list_statements": 8 * 29, "grid_paths": 40}
_ROW_SLOTS = {"polynomial": 27, "poly4": 60, "list_threshold": 44, "list_statements": 64, "grid_paths": 44}


def _search_work(workload, population, generations, cases):
    rows = population + generations  # ranked members and champions: counts, origins, constants, statistics
    return {"bytes": cases * _INPUT_BYTES[workload] + rows * (24 + 12 * _ROW_SLOTS[workload]),
            "flops": population * generations * cases * _OPERATIONS[workload]}


def work(case):
    """Cases in and results out, once each, and the integer operations of the programs on the cases."""
    kind = case["kind"]
    if kind in ("score", "score_static", "judge"):
        w = case["workload"]
        return {"bytes": case["cases"] * _INPUT_BYTES[w] + case["rows"] * (20 + 12 * _ROW_SLOTS[w]),
                "flops": case["rows"] * case["cases"] * _OPERATIONS[w]}
    if kind == "search":
        return _search_work(case["workload"], case["population"], case["generations"], case["cases"])
    # log-uniform populations from 256, uniform case counts
    top = case["largest_population"]
    population = (top - 256) / math.log(top / 256) if top > 256 else 256
    generations = case["generations"] * (0.75 if kind == "serve" else 1)
    each = [_search_work(w, population, generations, (16 + case["most_cases"]) / 2) for w in ("poly4", "list_threshold")]
    return {k: case["count"] / 2 * (each[0][k] + each[1][k]) for k in ("bytes", "flops")}


def _apply(name, args):
    """One operation of the scalar grammars on int64 columns: wrapping arithmetic, a zero divisor giving 0,
    division truncating, modulo with the divisor's sign."""
    a = args[0]
    if name == "if_expr":
        return np.where(a != 0, args[1], args[2])
    b = args[1]
    if name in ("idiv0", "imod0"):
        safe = np.where(b == 0, 1, b)
        rest = np.fmod(a, safe)
        got = (a - rest) // safe if name == "idiv0" else np.where((rest != 0) & ((rest < 0) != (safe < 0)), rest + safe, rest)
        return np.where(b == 0, 0, got)
    return {"add": np.add, "sub": np.subtract, "mul": np.multiply,
            "lt": lambda p, q: (p < q).astype(np.int64)}[name](a, b)


def exact(case, seed):
    """Scores of scalar rows, program by program in 64-bit integers; a search's results have no such value."""
    if case["kind"] not in ("score", "score_static") or case["workload"] not in ("polynomial", "poly4") \
            or case["rows"] * case["cases"] > 40_000_000:
        return None
    state = prepare(case, seed)
    task, rows = state["task"], state["rows"]
    names = [(e.name, e.kind, e.arity) for e in task.tables.expressions]
    x, want = task.cases.inputs[:, 0], task.cases.expected
    constant, leaf = 1, 4  # expression kinds: a constant, an input
    fitness, wrong = np.zeros(rows.count), np.zeros(rows.count, dtype=np.uint32)
    with np.errstate(all="ignore"):
        for i in range(rows.count):
            stack, k = [], int(rows.constant_counts[i])
            for at in range(int(rows.node_counts[i]) - 1, -1, -1):
                name, kind, arity = names[rows.origins[i, at]]
                if kind == leaf:
                    stack.append(x)
                elif kind == constant:
                    k -= 1
                    stack.append(np.full_like(x, rows.constants[i, k]))
                else:
                    args = [stack.pop() for _ in range(arity)]
                    stack.append(_apply(name, args))
            value = stack.pop()
            gap = np.where(value >= want, value.view(np.uint64) - want.view(np.uint64),
                           want.view(np.uint64) - value.view(np.uint64))
            fitness[i] = -float(np.minimum(gap, np.uint64(1000)).astype(np.int64).sum())
            wrong[i] = int((value != want).sum())
    return fitness, wrong
