"""FP64 multigrid: a GMRES cycle updates x from its preconditioned directions
where they could be kept, in the momentum systems' idle basis (vel_kdim + 1
vectors) and then in the pressure basis' unreached vectors, else it applies the
preconditioner to the basis combination. Both forms are the same update to FP64
rounding, and the directions take no memory of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MG = dict(p_pc=1, p_pc_rap_type=0, p_pc_relax_type=2, mg_nu1=1, mg_nu2=1, mg_nu_coarse=1, mg_omega=1.0,
          mg_group_ratio=1.5, mg_coarse_max=64)
SHAPES = [(48, 16, 16), (37, 15, 13)]


def rhs(case, seed):
    fluid = case.array("fluid_p").astype(bool)
    b = np.random.default_rng(seed).standard_normal(fluid.size) * fluid
    return b - fluid * (b.sum() / fluid.sum())


def solution(ibm, case, b, m, kdim, vel_kdim):
    s = ibm.Solver(case, ibm.solver_params(p_kdim=kdim, vel_kdim=vel_kdim, p_maxit=m, p_tol=1e-30, **MG))
    x, st = s.solve(ibm.FIELD_P, b)
    s.close()
    assert st.iters == m
    return x


# the two differ by a V-cycle's rounding of the same sum
def same(x, y):
    return np.abs(x - y).max() <= 1e-12 * np.abs(x).max()


@pytest.mark.parametrize("m", [4, 5, 12])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_kept_and_applied_updates_agree(ibm, shape, m):
    """One direction in the momentum basis: cycles of (p_kdim + 2) / 2 are the
    longest whose directions are kept."""
    case = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    b = rhs(case, 2)
    assert same(*[solution(ibm, case, b, m, kdim, 1) for kdim in (2 * m - 2, 2 * m - 3)])


@pytest.mark.parametrize("m", [4, 12, 30])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_lent_and_own_memory_agree(ibm, shape, m):
    """A whole cycle of p_kdim iterations with none (applied), some and all of
    its directions in the momentum basis."""
    case = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    b = rhs(case, 3)
    x = [solution(ibm, case, b, m, m, vel_kdim) for vel_kdim in (1, m // 2, m - 1, m, 63)]
    for y in x[1:]:
        assert same(x[0], y)


@pytest.mark.parametrize("vel_kdim", [1, 5, 50])
@pytest.mark.parametrize("kdim", [1, 2, 3, 4, 5, 7, 11, 25, 63])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_captured_restarts_equal_host_driven(ibm, shape, kdim, vel_kdim):
    """Cycles below and above the kept length, many of them in a solve."""
    case = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    host = ibm.Solver(case, ibm.solver_params(p_kdim=kdim, vel_kdim=vel_kdim, p_tol=1e-10, use_graph=0, **MG))
    graph = ibm.Solver(case, ibm.solver_params(p_kdim=kdim, vel_kdim=vel_kdim, p_tol=1e-10, use_graph=1, **MG))
    try:
        for _ in range(2):
            a, b = host.step(1.0), graph.step(1.0)
            assert (a.p.iters, a.p.status, a.p.rel_res) == (b.p.iters, b.p.status, b.p.rel_res)
            assert a.p.status == ibm.IBM_OK and a.p.rel_res <= 1e-10
        for x, y in zip(host.fields(), graph.fields()):
            assert np.all(np.isfinite(x))
            assert np.array_equal(x.view(np.uint64), y.view(np.uint64))
    finally:
        host.close()
        graph.close()


def test_directions_take_no_memory(ibm):
    import torch
    case = ibm.Case(ibm.channel_params(96, 48, 48, Um=1.0, dt=1e-3))
    n = 96 * 48 * 48
    used = []
    for kdim in (10, 60):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        s = ibm.Solver(case, ibm.solver_params(p_kdim=kdim, **MG))
        s.step(1.0)
        used.append(before - torch.cuda.mem_get_info()[0])
        s.close()
    # 50 more basis vectors of the pressure box, and allocation granularity
    assert used[1] - used[0] <= 50 * 8 * n + (8 << 20)
