"""The V-cycle of a host-driven solve runs its small levels on one
thread-block cluster, a captured one in launches of their own, and both take a
coarsening group's transfers in one launch on small levels. The arithmetic per
point is the same, so host-driven and captured steps must agree bit for bit:
FP64 and FP32 hierarchies, 7- and 27-point levels, Jacobi and two-colour
relaxation, paired and unpaired (odd) lines, hierarchies that fit the cluster
whole, from a coarse level on, and with the dense level in a launch of its
own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GROUPED = dict(p_pc_rap_type=0, p_pc_relax_type=2, mg_nu1=3, mg_nu2=3, mg_nu_coarse=2, mg_omega=1.0,
               mg_group_ratio=1.5, vel_inner_sweeps=2)
FORMS = {
    "default": {},
    "jacobi27": dict(p_pc_rap_type=0),
    "collapsed-two-colour": dict(p_pc_relax_type=2),
    "fp64-grouped": dict(GROUPED, mg_coarse_max=640),
    "fp64-grouped-small-dense": dict(GROUPED, mg_coarse_max=64),
    "fp32-cycles-grouped": dict(GROUPED, mg_coarse_max=640, precision=2),
    "fp32-multigrid-collapsed": dict(precision=1, p_pc_relax_type=2, mg_nu1=2, mg_nu2=1),
    "fp32-multigrid-jacobi": dict(precision=1),
}


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("shape", [(32, 12, 12), (37, 15, 13), (72, 24, 20), (100, 33, 28)])
def test_host_driven_and_captured_steps_agree(ibm, shape, form):
    case = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    a = ibm.Solver(case, ibm.solver_params(use_graph=0, **FORMS[form]))
    b = ibm.Solver(case, ibm.solver_params(use_graph=1, **FORMS[form]))
    try:
        for _ in range(2):
            sa, sb = a.step(1.0), b.step(1.0)
            assert (sa.p.iters, sa.status) == (sb.p.iters, sb.status)
        for x, y in zip(a.fields(), b.fields()):
            assert np.all(np.isfinite(x))
            assert np.array_equal(x.view(np.uint64), y.view(np.uint64))
        names = ibm.kernel_names()
        assert a.profile().launches[names.index("mg_cluster")] > 0
        assert b.profile().launches[names.index("mg_cluster")] == 0
    finally:
        a.close()
        b.close()
