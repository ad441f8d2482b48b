"""Performance cases of the solver: what its users have it compute, through its Python API.

A case is one use of the library on one size:

* ``solve``     ``solver.solve``: graph in, verdict, pass counts and the states table out in host
                memory.  The device buffers are created and released inside the call.
* ``resident``  a ``Solver`` kept for a graph: ``init``, ``run`` to the fixed point, ``verdict``;
                the table stays in device memory (``device_states``).
* ``phases``    the six phases of the reference's driver on a new ``Solver``: buildAuxGraph with its
                transition table, ``init``, ``step`` until a pass finds nothing, ``verdict``, table.
* ``batch``     ``batch_solve``: cop numbers of many small graphs in one call.
* ``serve``     requests given to a ``Server`` at once, answered in order of submission, released.

Graphs are the repository's seeded generators (4-regular, connected G(n, p), thinned Delaunay
triangulations) and, for ``phases``, the reference's own matrices with their vertices relabelled
at random (its 199-vertex board and the small graphs its test sweep runs over).
All outputs are whole numbers: table bytes, counts, positions, digests.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

from copsandrobbers_gb300 import graphs as G
from copsandrobbers_gb300 import native as N
from copsandrobbers_gb300.serving import Server, request_stream
from copsandrobbers_gb300.solver import Context, Solver, batch_solve, solve

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MATRICES = os.path.join(ROOT, "tests", "golden", "matrices")
# the reference's matrices by their vertex counts
BOARDS = {"scotlandyard-all": 199, "dismantleable48": 48, "grid36": 36, "planar32": 32, "outerplanar32": 32,
          "dodecahedron": 20, "robertson": 19, "rooks": 9, "cycle10": 10}
PASSES = 256  # room for the pass counts of any solve


def _one(name, use, graph, n, k, p=1, rules="v1", stay=False, degree=4.5):
    """One solve: `graph` is regular4, er or delaunay (mean degree `degree`), or one of BOARDS."""
    case = {"use": use, "graph": graph, "n": n, "k": k, "p": p, "rules": rules, "stay": stay, "degree": degree}
    return {"name": name} | case if name else case


def listed():
    return [
        # one question about a toy graph: nothing but latency, allocations and launches
        _one("solve er n12 k2", "solve", "er", 12, 2),
        # the size of the reference's own sweep over its small planar graphs (k <= 3, p <= 3)
        _one("solve delaunay n48 k3 p2", "solve", "delaunay", 48, 3, p=2),
        # the reference's board game, driven phase by phase as its drop-in driver does
        _one("phases board n199 k2", "phases", "scotlandyard-all", 199, 2),
        # the large solve of the benchmark: one dense first pass, then sparse ones
        _one("resident regular4 n256 k3", "resident", "regular4", 256, 3),
        # a sparse random graph at the largest size of the batch: a dozen dense passes
        _one("resident er n128 k3", "resident", "er", 128, 3),
        # planar, at the board's size, an odd vertex count: rows that are not whole words
        _one("resident delaunay n199 k3", "resident", "delaunay", 199, 3),
        # the top of the serving range
        _one("resident delaunay n389 k3", "resident", "delaunay", 389, 3),
        # limited visibility under the 2p-column rules, odd size
        _one("resident delaunay n127 k3 p3", "resident", "delaunay", 127, 3, p=3),
        # the classical game (both sides may stay put) with the most cops
        _one("resident er n61 k4 stay", "resident", "er", 61, 4, stay=True),
        # limited visibility under the macro-turn rules: the benchmark's size
        _one("resident v2 n199 k2 p3", "resident", "delaunay", 199, 2, p=3, rules="v2"),
        # cop numbers of a collection of small graphs
        {"name": "batch 256 n16-128", "use": "batch", "count": 256, "n_lo": 16, "n_hi": 128, "kmax": 3},
        # a burst of mixed requests
        {"name": "serve 24 n20-160", "use": "serve", "count": 24, "n_lo": 20, "n_hi": 160, "workers": 8},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    use = rng.choice(["solve", "solve", "resident", "resident", "resident", "resident", "phases", "batch", "serve"])
    if use == "batch":
        n_lo = _log_int(rng, 8, 32)
        return {"use": "batch", "count": _log_int(rng, 16, 256), "n_lo": n_lo,
                "n_hi": _log_int(rng, n_lo + 8, 128), "kmax": rng.choice([2, 3, 3])}
    if use == "serve":
        return {"use": "serve", "count": _log_int(rng, 4, 24), "n_lo": 20, "n_hi": _log_int(rng, 40, 160),
                "workers": rng.choice([4, 8, 16])}
    if use == "phases":
        graph = rng.choice(sorted(BOARDS))
        n = BOARDS[graph]
        return _one("", use, graph, n, rng.choice([1, 2, 3] if n < 100 else [1, 2]), rng.choice([1, 2, 3]))
    rules = rng.choice(["v1", "v1", "v1", "v2"])
    graph = rng.choice(["er", "delaunay", "regular4"])
    if rules == "v2":
        k, p = rng.choice([1, 2]), rng.choice([2, 3])
        top = (100, 199)[graph != "er"] if p == 3 else 199
        n = _log_int(rng, 8, top if use == "resident" else 64)
        degree = 4.5
    else:
        k = rng.choice([1, 2, 2, 3, 3, 3, 4])
        p = rng.choice([1, 1, 1, 2, 3, 4])
        top = {1: 512, 2: 512 if p == 1 else 300, 3: 380 if p == 1 else 160, 4: 61 if p == 1 else 40}[k]
        n = _log_int(rng, 8, top if use == "resident" else (200, 128, 56, 24)[k - 1])
        # (a sparser G(n, p) is hardly ever connected)
        degree = round(max(rng.uniform(4, 6), math.log(n) - 0.5), 1)
    stay = rules == "v1" and rng.random() < 0.2
    return _one("", use, graph, n, k, p, rules, stay, degree)


def _graph(case, seed):
    n = case["n"]
    if case["graph"] in BOARDS:
        a = G.load_matrix(os.path.join(MATRICES, case["graph"] + ".txt")).adj
        at = np.random.default_rng(seed).permutation(a.shape[0])
        return G.Graph(np.ascontiguousarray(a[np.ix_(at, at)]))
    if case["graph"] == "regular4":
        return G.regular4(n, seed)
    if case["graph"] == "er":
        return G.erdos_renyi(n, case["degree"], seed)
    return G.delaunay_thinned(n, seed, case["degree"])


def _rules(case):
    if case["rules"] == "v2":
        return N.CR_RULES_V2
    return N.CR_RULES_V1 | (N.CR_COP_STAY | N.CR_ROBBER_STAY if case["stay"] else 0)


def _sizes(case):
    """The batch's vertex counts: evenly over the range, so that the work is the case's own."""
    lo, hi, count = case["n_lo"], case["n_hi"], case["count"]
    return [lo + (hi - lo) * i // max(count - 1, 1) for i in range(count)]


class _Table:
    """A solver's device table as an array that torch can take up without a copy."""

    def __init__(self, solver):
        ptr, nbytes = solver.device_states()
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (ptr, False), "version": 3}


def _device_table(solver):
    """The table as a tensor.  The memory is the solver's until it is closed, so the tensor keeps it."""
    table = torch.as_tensor(_Table(solver), device="cuda")
    table.solver = solver
    return table


def prepare(case, seed):
    use = case["use"]
    rng = np.random.default_rng(seed)
    if use == "batch":
        graphs = [G.erdos_renyi(n, float(rng.uniform(3, 6)), int(rng.integers(1 << 31))) for n in _sizes(case)]
        return {"case": case, "ctx": Context(0), "graphs": graphs}
    if use == "serve":
        reqs = request_stream(case["count"], 1e6, seed=seed % (1 << 31), n_lo=case["n_lo"], n_hi=case["n_hi"])
        return {"case": case, "requests": reqs, "server": Server(0, 48 << 30, workers=case["workers"])}
    state = {"case": case, "ctx": Context(0), "graph": _graph(case, int(rng.integers(1 << 31)))}
    if use == "resident":
        s = Solver(state["ctx"], state["graph"], case["k"], case["p"], _rules(case))
        state |= {"solver": s, "table": _device_table(s)}
    return state


def _answer(base_captures, counts, verdict):
    """Counts and positions in arrays of one size, zeros behind them."""
    passes = np.zeros(PASSES, dtype=np.int64)
    passes[: len(counts)] = counts
    found = np.zeros(3 + N.CR_MAX_K, dtype=np.int64)
    found[:3] = verdict.win, verdict.capture_plies, verdict.best_config
    found[3 : 3 + len(verdict.positions)] = verdict.positions
    return {"captures": base_captures, "pass_counts": passes, "verdict": found}


def run(state):
    case = state["case"]
    use = case["use"]
    if use == "resident":
        s = state["solver"]
        caps = s.init()
        counts = s.run()
        return _answer(caps, counts, s.verdict()) | {"states": state["table"]}
    if use == "solve":
        r = solve(state["ctx"], state["graph"], case["k"], case["p"], _rules(case))
        return _answer(r.base_captures, r.pass_counts, r.verdict) | {"states": r.states}
    if use == "phases":
        with Solver(state["ctx"], state["graph"], case["k"], case["p"], _rules(case)) as s:
            heads, data = s.transitions()
            caps = s.init()
            while s.step():
                pass
            return _answer(caps, s.pass_counts, s.verdict()) | {
                "states": s.states(), "heads": heads.view(np.int64), "transitions": data.view(np.int64)}
    if use == "batch":
        out = batch_solve(state["ctx"], state["graphs"], case["kmax"])
        fields = ("solved", "win", "capture_plies", "passes", "best_config", "base_captures", "states", "digest",
                  "pass_hash")
        flat = np.array([[r[f] & (1 << 64) - 1 for f in fields] for per in out.results for r in per], dtype=np.uint64)
        return {"cop_numbers": np.array(out.cop_numbers, dtype=np.int64), "solves": flat.view(np.int64)}
    server = state["server"]
    ids = [server.submit(r.graph, r.k, r.p, r.rules) for r in state["requests"]]
    fields = ("status", "win", "capture_plies", "passes", "best_config", "base_captures", "states", "digest",
              "pass_hash")
    rows = []
    for i in ids:
        res = server.poll(i, wait_ms=-1)
        rows.append([res[f] & (1 << 64) - 1 for f in fields])
        server.release(i)
    return {"answers": np.array(rows, dtype=np.uint64).view(np.int64)}


def _solve_bytes(n, k, columns, degree):
    """The table once, and the graph's neighbour lists."""
    return math.comb(n + k - 1, k) * n * columns + n * (4 + 2 * degree)


def work(case):
    """The tables written once.  The work is on whole numbers and bits: there are no flops."""
    use = case["use"]
    if use == "batch":
        # a graph's search ends at its cop number: two or three for almost all of these
        return {"bytes": sum(_solve_bytes(n, k, 2, 4.5) for n in _sizes(case) for k in range(1, case["kmax"] + 1)),
                "flops": 0}
    if use == "serve":
        # k is 1, 2 or 3 and the vertex count log-uniform
        lo, hi = math.log(case["n_lo"]), math.log(case["n_hi"])
        mid = [math.exp(lo + (hi - lo) * (i + 0.5) / 16) for i in range(16)]
        mean = sum(_solve_bytes(int(n), k, 2, 4.5) for n in mid for k in (1, 2, 3)) / 48
        return {"bytes": case["count"] * mean, "flops": 0}
    columns = 1 if case["rules"] == "v2" else 2 * case["p"]
    b = _solve_bytes(case["n"], case["k"], columns, case["degree"])
    if use == "phases":
        b += 8 * math.comb(case["n"] + case["k"] - 1, case["k"]) * (1 + case["degree"] ** case["k"])
    return {"bytes": b, "flops": 0}


def exact(case, seed):
    """Every output is a whole number, compared bit for bit: there is no rounding to measure."""
    return None
