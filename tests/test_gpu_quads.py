"""FP32 multigrid levels with nx % 4 == 0 relax and form residuals four points
a thread and take runs of one record from the kernel's parameters; one point at
a time (mg_quads 0) is the same arithmetic, so V-cycles must agree bit for
bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one, two and three quads a line (no inner quads, one); runs cut by line ends;
# 32 and 33 inner quads; lines in y and z that leave partial runs; above two
# million points with 81 and 30 quads a line
SHAPES = [(4, 8, 8), (8, 8, 8), (12, 9, 8), (136, 12, 12), (140, 13, 11), (324, 81, 83), (120, 129, 137)]


@pytest.mark.parametrize("rap", [0, 1])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_quads_equal_single_points(ibm, shape, rap):
    case = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    prm = dict(p_pc_rap_type=rap, p_pc_relax_type=2, mg_nu1=3, mg_nu2=3, mg_nu_coarse=2, mg_omega=1.0,
               mg_group_ratio=1.5, mg_coarse_max=64, precision=1)
    a = ibm.Solver(case, ibm.solver_params(mg_quads=1, **prm))
    b = ibm.Solver(case, ibm.solver_params(mg_quads=0, **prm))
    try:
        r = np.random.default_rng(3).standard_normal(np.prod(shape))
        za, zb = a.apply_preconditioner(ibm.FIELD_P, r), b.apply_preconditioner(ibm.FIELD_P, r)
        assert np.all(np.isfinite(za))
        assert np.array_equal(za.view(np.uint64), zb.view(np.uint64))
    finally:
        a.close()
        b.close()


def test_solve_equals_single_points(ibm):
    """The whole FP32 solve: the V-cycle's input and output fused into the
    finest level's first and last sweeps."""
    shape = (324, 81, 83)
    case = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    fluid = case.array("fluid_p").astype(bool)
    rhs = np.random.default_rng(4).standard_normal(fluid.size) * fluid
    out = []
    for quads in (1, 0):
        s = ibm.Solver(case, ibm.solver_params(mg_quads=quads, p_pc_rap_type=0, p_pc_relax_type=2, mg_nu1=3, mg_nu2=3,
                                               mg_nu_coarse=2, mg_omega=1.0, mg_group_ratio=1.5, mg_coarse_max=640,
                                               precision=2, p_tol=1e-6))
        x, st = s.solve(ibm.FIELD_P, rhs)
        assert st.status == ibm.IBM_OK
        out.append(x)
        s.close()
    assert np.array_equal(out[0].view(np.uint64), out[1].view(np.uint64))
