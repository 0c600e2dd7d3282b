"""Within a solve the finest FP32 level (nx a multiple of 8) keeps x and b by
colour and takes four points a thread; one point at a time on the joined arrays
(mg_quads 0) is the same arithmetic, so captured steps and host-driven solves
must agree bit for bit. One, two and three octets a line (no inner octets, one),
32 inner octets, partial runs, one sweep each way, levels below and above the
size where the transfers have launches of their own, FP32 and FP64 Krylov bases
(their input and output)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(8, 8, 8), (16, 9, 8), (24, 12, 12), (136, 13, 12), (272, 13, 11), (328, 47, 48)]
MG = dict(p_pc=1, p_pc_rap_type=0, p_pc_relax_type=2, mg_nu_coarse=2, mg_omega=1.0, mg_group_ratio=1.5, mg_coarse_max=64)


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("nu", [1, 3])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_split_equals_joined(ibm, shape, nu, precision):
    case = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    fluid = case.array("fluid_p").astype(bool)
    b = np.random.default_rng(5).standard_normal(fluid.size) * fluid
    b -= fluid * (b.sum() / fluid.sum())
    out = []
    for quads in (1, 0):
        s = ibm.Solver(case, ibm.solver_params(mg_quads=quads, mg_nu1=nu, mg_nu2=nu, precision=precision, use_graph=1,
                                               p_tol=1e-6, **MG))
        s.step(1.0)
        s.step(1.0)
        x, st = s.solve(ibm.FIELD_P, b)
        assert st.status == ibm.IBM_OK
        out.append(list(s.fields()) + [x])
        s.close()
    for x, y in zip(*out):
        assert np.all(np.isfinite(x))
        assert np.array_equal(x.view(np.uint64), y.view(np.uint64))
