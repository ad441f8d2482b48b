"""The forms that take dense frontiers -- the last column's tiles of 32 rows and the separable cop
turn through head rows -- against the general forms (every open row tested against the table, cop
turns gathered tuple by tuple), which the other tests pin to the oracle.  Sizes: rows of part and
of whole words, one to sixteen words, lists long enough for tiles (16 rows per warp of the launch)."""
import numpy as np
import pytest

from copsandrobbers_gb300 import graphs as G
from copsandrobbers_gb300 import native as N

pytestmark = pytest.mark.gpu

STAY = N.CR_COP_STAY | N.CR_ROBBER_STAY
GENERAL = N.CR_FORM_PULL  # the tuple-gathering pull and the last column's general form only


def directed(n, seed):
    """A random digraph without a vertex that has no move."""
    rng = np.random.default_rng(seed)
    adj = (rng.random((n, n)) < 4.0 / n).astype(np.uint8)
    adj[np.arange(n), (np.arange(n) + 1) % n] = 1
    np.fill_diagonal(adj, 0)
    return G.Graph(adj)


@pytest.mark.parametrize("graph, n, k, p, rules", [
    ("er", 31, 4, 1, 0), ("er", 32, 4, 1, 0), ("delaunay", 33, 4, 1, STAY), ("er", 45, 4, 1, N.CR_COP_STAY),
    ("delaunay", 64, 3, 1, 0), ("er", 77, 3, 1, 0), ("delaunay", 96, 3, 1, STAY), ("delaunay", 97, 3, 1, 0),
    ("directed", 96, 3, 1, 0), ("er", 128, 3, 1, N.CR_ROBBER_STAY), ("delaunay", 129, 3, 1, 0),
    ("regular4", 192, 3, 1, 0), ("delaunay", 257, 3, 1, 0), ("delaunay", 80, 3, 2, 0), ("er", 81, 3, 3, 0),
    ("delaunay", 395, 2, 1, 0), ("regular4", 512, 2, 1, 0), ("delaunay", 416, 2, 1, 0), ("er", 7, 2, 1, 0),
])
def test_dense_forms_give_the_general_forms_tables(graph, n, k, p, rules):
    from copsandrobbers_gb300.solver import Context, Solver, solver_digest

    g = {"er": lambda: G.erdos_renyi(n, 5.0, n + k), "delaunay": lambda: G.delaunay_thinned(n, n + k),
         "regular4": lambda: G.regular4(n, n + k), "directed": lambda: directed(n, n)}[graph]()
    got = []
    with Context(0) as ctx:
        for forms in (N.CR_FORMS_ALL, GENERAL):
            with Solver(ctx, g, k, p, N.CR_RULES_V1 | rules) as s:
                s.set_forms(forms)
                s.init()
                got.append((s.run(), solver_digest(s), s.verdict()))
    assert got[0] == got[1]
