"""The finest FP64 level stored with its couplings scaled by the inverse
diagonal (two-colour relaxation that smooths on the way down) takes no more
memory than the plain one (no sweep on the way down)."""
import pytest

pytestmark = pytest.mark.gpu


def test_scaled_level_takes_no_more_memory(ibm):
    import torch
    shape = (160, 64, 64)
    case = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    b = case.array("fluid_p").astype(float)
    used = []
    for nu1 in (0, 0, 1):  # the first for what a process loads once
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        s = ibm.Solver(case, ibm.solver_params(p_pc=1, p_pc_rap_type=0, p_pc_relax_type=2, mg_nu1=nu1, mg_nu2=1,
                                               mg_group_ratio=1.5, mg_omega=1.0, mg_coarse_max=64, p_maxit=1))
        s.solve(ibm.FIELD_P, b)
        used.append(before - torch.cuda.mem_get_info()[0])
        s.close()
    # one more vector of the level would be 5.2 MB; memory comes in pieces of 2 MB
    assert used[2] - used[1] <= 2 << 20
