"""Within a solve the finest FP64 level (nx a multiple of 4) keeps x and b by
colour and takes two points a thread; one point at a time on the joined arrays
(mg_quads 0) is the same arithmetic, so captured steps and host-driven solves
must agree bit for bit. Levels of 300000 points take this form: just below it,
and above it one, two and three quads a line (no inner quads, one), 32 and 33
inner quads, one sweep each way, below and above the size where the transfers
have launches of their own, classed and plain records. (One
sweep each way does not converge on the flattest box; both forms must say so.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(4, 276, 276), (8, 201, 200), (12, 160, 161), (136, 46, 48), (136, 47, 48), (140, 47, 47), (328, 47, 48)]
MG = dict(p_pc=1, p_pc_rap_type=0, p_pc_relax_type=2, mg_nu_coarse=2, mg_omega=1.0, mg_group_ratio=1.5, mg_coarse_max=64)


@pytest.mark.parametrize("classes", [0, 1])
@pytest.mark.parametrize("nu", [1, 3])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_split_equals_joined(ibm, shape, nu, classes):
    case = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    fluid = case.array("fluid_p").astype(bool)
    b = np.random.default_rng(6).standard_normal(fluid.size) * fluid
    b -= fluid * (b.sum() / fluid.sum())
    out = []
    for quads in (1, 0):
        s = ibm.Solver(case, ibm.solver_params(mg_quads=quads, mg_nu1=nu, mg_nu2=nu, row_classes=classes, use_graph=1,
                                               p_tol=1e-6, **MG))
        s.step(1.0)
        s.step(1.0)
        x, st = s.solve(ibm.FIELD_P, b)
        out.append(list(s.fields()) + [x, np.array([float(st.status), float(st.iters)])])
        s.close()
    for x, y in zip(*out):
        assert np.all(np.isfinite(x))
        assert np.array_equal(x.view(np.uint64), y.view(np.uint64))
