"""Verdicts of the smallest graphs, whose table rows are shorter than the pieces findFinalResult reads
them in: every undirected graph of up to four vertices and random ones of up to eight, under all stay
rules, alone and in a batch, against the oracle."""
import itertools

import numpy as np
import pytest

from copsandrobbers_gb300 import graphs as G
from copsandrobbers_gb300 import native as N
from copsandrobbers_gb300.solver import batch_solve, solve
from oracle import oracle as O

pytestmark = pytest.mark.gpu
STAY = [(False, False), (True, False), (False, True), (True, True)]


def graphs_of(n):
    pairs = list(itertools.combinations(range(n), 2))
    rng = np.random.default_rng(n)
    every = itertools.product((0, 1), repeat=len(pairs))
    chosen = every if n <= 4 else ((rng.random(len(pairs)) < rng.uniform(0.2, 0.9)).astype(int) for _ in range(10))
    out = []
    for edges in chosen:
        adj = np.zeros((n, n), dtype=np.uint8)
        for (a, b), e in zip(pairs, edges):
            adj[a, b] = adj[b, a] = e
        out.append(G.Graph(adj))
    return out


def verdict_of(ref):
    if ref.best_config < 0:
        return False, -1, ()
    return True, ref.best_config, tuple(int(v) for v in ref.configs[ref.best_config])


@pytest.mark.parametrize("n", range(1, 9))
def test_verdicts_of_small_graphs(gpu_ctx, n):
    for g in graphs_of(n):
        for k in range(1, 5):
            for cop, robber in STAY:
                ref = O.solve_v1(g, k, 1, threads=1, cop_stay=cop, robber_stay=robber)
                v = solve(gpu_ctx, g, k, 1, N.CR_RULES_V1 | cop * N.CR_COP_STAY | robber * N.CR_ROBBER_STAY).verdict
                assert (v.win, v.best_config, v.positions) == verdict_of(ref), (g.adj.tolist(), k, cop, robber)
                if v.win:
                    assert v.capture_plies == ref.capture_plies, (g.adj.tolist(), k, cop, robber)


@pytest.mark.parametrize("n", range(1, 9))
def test_batch_verdicts_of_small_graphs(gpu_ctx, n):
    graphs = graphs_of(n)
    out = batch_solve(gpu_ctx, graphs, kmax=3, threads=256)
    for g, per in zip(graphs, out.results):
        for k, r in enumerate(per, 1):
            if not r["solved"]:
                continue
            ref = O.solve_v1(g, k, 1, threads=1)
            assert (bool(r["win"]), r["best_config"]) == verdict_of(ref)[:2], (g.adj.tolist(), k)
            if r["win"]:
                assert r["capture_plies"] == ref.capture_plies, (g.adj.tolist(), k)
