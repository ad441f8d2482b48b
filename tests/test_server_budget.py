"""A server's memory budget bounds what its solves hold.  A request that the budget cannot hold whole is
solved lean -- without the head rows of k = 2 and 4, or the plain values of the v2 rules -- and booked
as such; its results are those of the same solve alone."""
import ctypes
import math

import numpy as np
import pytest

from copsandrobbers_gb300 import graphs as G
from copsandrobbers_gb300 import native as N
from copsandrobbers_gb300.serving import Server
from copsandrobbers_gb300.solver import Solver, footprint, solver_digest
from oracle import oracle as O

V1, V2 = N.CR_RULES_V1, N.CR_RULES_V2


def lean_footprint(n, k, p, rules):
    f = N.lib()["_ZN5crgpu14lean_footprintEiiii"]
    f.restype = ctypes.c_uint64
    return int(f(n, k, p, rules))


def rows(n):
    rw = (n + 31) // 32
    return rw if rw <= 2 else (rw + 3) // 4 * 4


def needed_before(n, k, p, rules):
    """The bytes a server asked for before solvers had head rows for k = 2 and 4, or plain values: what
    its budget admitted then it has to admit for good."""
    c, r = math.comb(n + k - 1, k), rows(n)
    if rules == V2:
        slots = 0
        if p >= 3:
            slots = 1024
            while slots < 2 * c * n and slots < 1 << 24:
                slots *= 2
        return 3 * c * n + 4 * c * r + 3 * c + 4 * n * r + 2 * c * k + slots * (8 + 4 * r) + (1 << 16)
    cols = 2 * p
    b = c * n * cols + cols * c * r * 4 * 3 + c * 2 * r * 4 + (c + 31) // 32 * 4 + c * 4 + cols * c * 4 + 8
    b += n * (n + 1) // 2 * n * 2 * r * 4 if k == 3 and r <= 16 else 0
    b += cols * c + 2 * c * k + n * r * 12 + 4 * k * (n + 1) + (1 << 16) + (1 << 19) + 256
    return b + (8 * n * ((n + 7) // 8 * 8) if cols == 2 else 0)


def test_lean_solves_need_no_more_than_before():
    for rules, ps, top in ((V1, (1, 2, 3, 8, 63), 512), (V2, range(1, 9), 512)):
        for k in range(1, 5):
            for p in ps:
                for n in [*range(1, 70), 96, 97, 127, 128, 129, 200, 255, 256, 257, 300, 384, 389, 416, 500, top]:
                    lean = lean_footprint(n, k, p, rules)
                    if lean > 128 << 30:   # (a table of half the device and more)
                        continue
                    assert lean <= needed_before(n, k, p, rules), (n, k, p, rules)
                    assert lean <= footprint(n, k, p, rules)


def server_with(budget):
    """A server of one worker whose requests may hold `budget` bytes."""
    total = budget
    while total - total // 8 < budget:   # (an eighth is set aside for the worker's block cache)
        total += max(1, (budget - (total - total // 8)) // 2)
    return Server(0, total, workers=1)


def alone(ctx, g, k, p, rules):
    with Solver(ctx, g, k, p, rules) as s:
        s.init()
        counts = s.run()
        return solver_digest(s), N.pass_hash(counts), s.verdict().best_config


CASES = [("er", 9, 2, 1, V1), ("er", 33, 2, 2, V1), ("er", 12, 4, 1, V1), ("delaunay", 17, 4, 2, V1),
         ("delaunay", 66, 2, 1, V1), ("regular4", 260, 2, 1, V1),
         ("path", 2, 1, 2, V2), ("path", 3, 2, 3, V2), ("er", 8, 1, 1, V2), ("er", 13, 2, 2, V2), ("delaunay", 14, 2, 3, V2),
         ("er", 11, 2, 4, V2), ("regular4", 34, 1, 5, V2), ("delaunay", 66, 1, 3, V2), ("er", 10, 3, 2, V2),
         ("delaunay", 40, 2, 3, V2)]


def graph(kind, n):
    if kind == "path":
        adj = np.zeros((n, n), dtype=np.uint8)
        adj[np.arange(n - 1), np.arange(1, n)] = adj[np.arange(1, n), np.arange(n - 1)] = 1
        return G.Graph(adj)
    return {"er": lambda: G.erdos_renyi(n, 3.5, n), "delaunay": lambda: G.delaunay_thinned(n, n),
            "regular4": lambda: G.regular4(n, n)}[kind]()


@pytest.mark.gpu
@pytest.mark.parametrize("kind, n, k, p, rules", CASES)
def test_lean_solve_is_booked_and_right(gpu_ctx, kind, n, k, p, rules):
    g = graph(kind, n)
    lean = lean_footprint(n, k, p, rules)
    between = (lean + footprint(n, k, p, rules)) // 2
    assert lean < between
    with server_with(between) as srv:
        i = srv.submit(g, k, p, rules)
        res = srv.poll(i, wait_ms=-1)
        assert srv.stats()["memory_in_use"] == lean
        srv.release(i)
    assert (res["digest"], res["pass_hash"], res["best_config"]) == alone(gpu_ctx, g, k, p, rules)
    if rules == V2:
        ref = O.solve_v2(g, k, p)
        assert (res["digest"], res["pass_hash"]) == (N.table_digest(ref.states), N.pass_hash(ref.pass_counts))


@pytest.mark.gpu
def test_too_large_even_lean_is_refused():
    with server_with(lean_footprint(64, 4, 1, V1) - 4096) as srv:
        with pytest.raises(N.CrGpuError) as e:
            srv.submit(G.regular4(64, 1), 4, 1, V1)
        assert e.value.code == 2


@pytest.mark.gpu
@pytest.mark.parametrize("n, k, p, rules", [(500, 2, 2, V2), (60, 4, 1, V1)])
def test_a_named_budget_bounds_the_memory_taken(n, k, p, rules):
    import torch

    g = G.delaunay_thinned(n, 1) if rules == V2 else G.regular4(n, 1)
    budget = needed_before(n, k, p, rules)
    with Server(0, 4 * budget, workers=1) as srv:   # (kernels and their local memory are loaded)
        srv.poll(srv.submit(g, k, p, rules), wait_ms=-1)
    with server_with(budget) as srv:
        free = torch.cuda.mem_get_info()[0]
        assert srv.poll(srv.submit(g, k, p, rules), wait_ms=-1)["status"] == 0
        taken = free - torch.cuda.mem_get_info()[0]
    # CUDA hands out 2 MiB pages: up to one more for each of some dozen blocks
    assert taken <= budget + 16 * (2 << 20), (taken, budget)
