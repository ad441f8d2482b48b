"""The passes of a small solve run in one launch, by a block or a cluster; with profiling on, the same
passes are launched kernel by kernel.  Both give the same tables, counts and verdicts, on either side of
the lines between block, cluster and launches, run whole and pass by pass."""
import numpy as np
import pytest

from copsandrobbers_gb300 import graphs as G
from copsandrobbers_gb300 import native as N
from copsandrobbers_gb300.solver import Context, Solver

pytestmark = pytest.mark.gpu
STAY = N.CR_COP_STAY | N.CR_ROBBER_STAY


def solved(g, k, p, rules, profiling, stepwise):
    with Context(0) as ctx:
        ctx.set_profiling(profiling)
        with Solver(ctx, g, k, p, N.CR_RULES_V1 | rules) as s:
            s.init()
            if stepwise:
                while s.step():
                    pass
            else:
                s.run()
            return s.pass_counts, s.verdict(), s.states(), s.stats()


# (vertices, cops, period): one block up to some 16 K row words a pass, a cluster up to 48 K, then launches
@pytest.mark.parametrize("n, k, p", [(1, 1, 1), (2, 2, 1), (6, 1, 3), (31, 1, 1), (32, 2, 1), (33, 2, 2), (24, 2, 3), (64, 1, 2),
                                     (65, 1, 1), (129, 1, 2), (199, 1, 1), (256, 1, 1), (256, 1, 3), (257, 1, 1), (40, 2, 2),
                                     (60, 2, 1), (65, 2, 1), (14, 3, 1), (20, 3, 2), (24, 3, 1), (9, 4, 1), (13, 4, 2), (17, 4, 1)])
@pytest.mark.parametrize("rules", [0, STAY])
def test_one_launch_and_launches_agree(n, k, p, rules):
    g = G.Graph(np.ones((n, n), dtype=np.uint8) - np.eye(n, dtype=np.uint8)) if n < 6 else G.delaunay_thinned(n, 5 * n + k)
    ref = solved(g, k, p, rules, True, False)
    for stepwise in (False, True):
        got = solved(g, k, p, rules, False, stepwise)
        assert got[:2] == ref[:2]
        assert np.array_equal(got[2], ref[2])


@pytest.mark.parametrize("n, k, p, one_launch", [(24, 2, 1, True), (199, 1, 1, True), (48, 2, 1, True), (257, 1, 1, False),
                                                 (64, 3, 1, False)])
def test_small_solves_take_the_single_launch(n, k, p, one_launch):
    g = G.delaunay_thinned(n, n)
    counts, _, _, stats = solved(g, k, p, 0, False, False)
    assert len(counts) > 2
    # the folded first pass and the launch for the others
    assert (stats.kernel_launches == 2) == one_launch, stats.kernel_launches
