"""The device table is complete when a phase returns: its address, taken once, may be read on another
stream right after the next initializeCaptures and after each pass."""
import numpy as np
import pytest

from copsandrobbers_gb300 import graphs as G
from copsandrobbers_gb300 import native as N
from copsandrobbers_gb300.solver import Context, Solver

pytestmark = pytest.mark.gpu


class Table:
    def __init__(self, solver):
        ptr, nbytes = solver.device_states()
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (ptr, False), "version": 3}


@pytest.mark.parametrize("n, k, p, rules", [(160, 3, 2, N.CR_RULES_V1), (300, 2, 2, N.CR_RULES_V2)])
def test_table_is_complete_when_a_phase_returns(n, k, p, rules):
    import torch

    side = torch.cuda.Stream()
    with Context(0) as ctx, Solver(ctx, G.regular4(n, 3), k, p, rules) as s:
        s.init()
        s.step()
        table = torch.as_tensor(Table(s), device="cuda")
        for phase in (s.init, s.step):
            phase()
            with torch.cuda.stream(side):
                got = table.clone()
            side.synchronize()
            assert np.array_equal(got.cpu().numpy(), s.states())
