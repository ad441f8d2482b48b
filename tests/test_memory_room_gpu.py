"""A device with little room: solvers do without head rows (k = 2 and 4) or the plain values of the v2
rules, at their creation and when something is allocated later, and give the same results.  The room is
that of the context's blocks (cr_context_limit_blocks); the GPU itself is never filled."""
import ctypes
from math import comb

import pytest

from copsandrobbers_gb300 import graphs as G
from copsandrobbers_gb300 import native as N
from copsandrobbers_gb300.solver import Context, Solver, batch_solve, solver_digest

pytestmark = pytest.mark.gpu
V1, V2 = N.CR_RULES_V1, N.CR_RULES_V2


def limit(ctx, nbytes):
    """Sets the room; the most that was taken so far."""
    f = N.lib().cr_context_limit_blocks
    f.argtypes = [ctypes.c_void_p, ctypes.c_uint64, ctypes.POINTER(ctypes.c_uint64)]
    peak = ctypes.c_uint64()
    assert f(ctx.ptr, nbytes, ctypes.byref(peak)) == 0
    return int(peak.value)


def solved(ctx, g, k, p, rules, transitions=False):
    """Digest, counts, verdict; the transition table is built between the first pass and the others."""
    with Solver(ctx, g, k, p, rules) as s:
        s.init()
        counts = [s.step()]
        heads, data = s.transitions() if transitions else ((), ())
        while counts[-1]:
            counts.append(s.step())
        return solver_digest(s), counts, s.verdict(), list(heads[-3:]), list(data[-3:])


def optional_bytes(n, k, rules):
    """Head rows, or the plain values."""
    rw = (n + 31) // 32
    row = 4 * (rw if rw <= 2 else (rw + 3) // 4 * 4)
    return comb(n + k - 1, k) * n if rules == V2 else comb(n + k - 2, k - 1) * n * 2 * row


@pytest.mark.parametrize("transitions", [False, True])
@pytest.mark.parametrize("n, k, p, rules", [(400, 2, 1, V1), (40, 4, 1, V1), (200, 2, 2, V1), (300, 2, 2, V2),
                                            (100, 2, 3, V2), (300, 2, 1, V2)])
def test_solves_without_room_for_the_optional_arrays(n, k, p, rules, transitions):
    g = G.regular4(n, n) if rules == V1 else G.delaunay_thinned(n, n)
    with Context(0) as ctx:
        ref = solved(ctx, g, k, p, rules, transitions)
        peak = limit(ctx, 1 << 40)
    # more than a mebibyte, so that the block is exactly as large
    optional = optional_bytes(n, k, rules) if optional_bytes(n, k, rules) >= 1 << 20 else 1
    for less in (0, 1, optional // 2, optional):
        with Context(0) as ctx:
            limit(ctx, peak - less)
            assert solved(ctx, g, k, p, rules, transitions) == ref, less


@pytest.mark.parametrize("n, k, p, rules", [(64, 3, 1, V1), (40, 2, 1, V1), (60, 2, 3, V2)])
def test_a_refusal_leaves_the_context_usable(n, k, p, rules):
    g = G.regular4(n, n)
    with Context(0) as ctx:
        ref = solved(ctx, g, k, p, rules)
        peak = limit(ctx, 1 << 16)
        ctx.set_cache_limit(0)
        for room in (1 << 16, peak // 4, peak // 3):
            limit(ctx, room)
            with pytest.raises(N.CrGpuError) as e:
                solved(ctx, g, k, p, rules)
            assert e.value.code in (2, 3) and "memory" in str(e.value)
        limit(ctx, 1 << 16)   # (a batch of one small graph takes less than the solve)
        with pytest.raises(N.CrGpuError):
            batch_solve(ctx, [g], kmax=2)
        limit(ctx, 1 << 40)
        assert solved(ctx, g, k, p, rules) == ref
        assert batch_solve(ctx, [g], kmax=2).results[0][0]["status"] == 0
