"""Robbers whose every walk ends before the visibility period does: on a directed graph with dead ends a
vertex with moves may have no walk of p moves.  Tables, counts and verdicts of such graphs against the
oracle, in every kernel form, and of the entry that allocates nothing."""
import numpy as np
import pytest

from copsandrobbers_gb300 import graphs as G
from copsandrobbers_gb300 import native as N
from copsandrobbers_gb300.solver import Solver, solve
from oracle import oracle as O
from test_forms_gpu import MASKS
from test_zz_no_alloc import _noalloc

pytestmark = pytest.mark.gpu


def dead_ends(n, degree, seed):
    """A digraph of layers: arcs lead forward in a random order, a few back."""
    rng = np.random.default_rng(seed)
    adj = np.triu(rng.random((n, n)) < degree / n, 1) | (rng.random((n, n)) < 0.3 / n)
    np.fill_diagonal(adj, False)
    at = rng.permutation(n)
    return G.Graph(np.ascontiguousarray(adj[np.ix_(at, at)].astype(np.uint8)))


@pytest.mark.parametrize("name", sorted(MASKS))
@pytest.mark.parametrize("n, k, p", [(2, 1, 2), (3, 2, 4), (9, 2, 2), (14, 3, 3), (26, 2, 3), (33, 2, 2), (64, 1, 2), (70, 2, 4),
                                     (115, 1, 3)])
def test_dead_ends_match_the_oracle(gpu_ctx, n, k, p, name):
    for seed in range(3):
        g = dead_ends(n, 3.0, 10 * n + seed)
        ref = O.solve_v1(g, k, p)
        with Solver(gpu_ctx, g, k, p) as s:
            s.set_forms(MASKS[name])
            s.init()
            assert s.run() == ref.pass_counts, seed
            assert np.array_equal(s.states(), ref.states), seed
            assert s.verdict().best_config == ref.best_config


@pytest.mark.parametrize("n, k, p", [(2, 1, 2), (14, 3, 3), (33, 2, 2), (70, 2, 4)])
def test_dead_ends_without_allocation(n, k, p):
    torch = pytest.importorskip("torch")
    g = dead_ends(n, 3.0, n)
    ref = O.solve_v1(g, k, p)
    out = torch.empty(ref.states.size, dtype=torch.uint8, device="cuda")
    rc, counts, caps, err = _noalloc(g, k, p, out.data_ptr(), out.numel())
    assert rc == 0, err
    assert (counts, caps) == (ref.pass_counts, ref.base_captures)
    assert np.array_equal(out.cpu().numpy(), ref.states)
