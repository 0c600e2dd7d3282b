"""All sweeps of a small 27-point level run in one launch on one cluster within
a solve; ibm_apply_preconditioner runs a launch per phase. One GMRES iteration
from zero gives x = c M b, so x and M b must have one direction: to FP64
rounding (1e-12) and FP32 rounding of a V-cycle (1e-5). Levels of exactly as
many points as the cluster's registers hold and just above, of one block, with
odd and even lines, an odd number of points, and rows that reach several
blocks. Where levels run on one launch per phase in a host-driven solve, a
captured step must still give its bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GROUPED = dict(p_pc_rap_type=0, p_pc_relax_type=2, mg_nu1=3, mg_nu2=3, mg_nu_coarse=2, mg_omega=1.0,
               mg_group_ratio=1.5, p_pc=1)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dense", [64, 640])
@pytest.mark.parametrize("shape", [(160, 32, 32), (168, 32, 32), (97, 33, 21), (98, 33, 20), (128, 24, 24), (144, 24, 24),
                                   (24, 12, 12)], ids=lambda s: "x".join(map(str, s)))
def test_one_iteration_is_the_preconditioner(ibm, shape, dense, precision):
    case = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    s = ibm.Solver(case, ibm.solver_params(precision=precision, p_maxit=1, mg_coarse_max=dense, **GROUPED))
    try:
        fluid = case.array("fluid_p").astype(bool)
        b = np.random.default_rng(8).standard_normal(fluid.size) * fluid
        b -= fluid * (b.sum() / fluid.sum())
        x, _ = s.solve(ibm.FIELD_P, b)
        z = s.apply_preconditioner(ibm.FIELD_P, b)
        x, z = x / np.linalg.norm(x), z / np.linalg.norm(z)
        assert np.linalg.norm(x - z * np.sign(x @ z)) <= (1e-12 if precision == 0 else 1e-5)
    finally:
        s.close()


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", [(160, 32, 32), (168, 32, 32), (98, 33, 20)], ids=lambda s: "x".join(map(str, s)))
def test_captured_step_equals_host_driven(ibm, shape, form):
    case = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    more = dict(precision=2, vel_precision=1) if form == "mixed" else {}
    fields = []
    for graph in (0, 1):
        s = ibm.Solver(case, ibm.solver_params(use_graph=graph, mg_coarse_max=640, **GROUPED, **more))
        for _ in range(2):
            s.step(1.0)
        fields.append(s.fields())
        s.close()
    for x, y in zip(*fields):
        assert np.array_equal(x.view(np.uint64), y.view(np.uint64))
