"""Hierarchies that are the dense level alone: a box of at most mg_coarse_max
cells, or one level allowed. The preconditioner is then the exact inverse, as the
oracle's V-cycle is, whatever the relaxation (even and odd nx, which decide the
relaxation's layout), with and without the symmetrizer; a pressure solve takes
an iteration or two, on its own and within a step, host-driven and captured."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HOW = {"coarse-max": dict(mg_coarse_max=4096), "one-level": dict(mg_max_levels=1)}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("options", [3, 0])
@pytest.mark.parametrize("relax", [1, 2])
@pytest.mark.parametrize("how", HOW)
@pytest.mark.parametrize("shape", [(8, 8, 8), (9, 8, 8), (12, 7, 9)], ids=lambda s: "x".join(map(str, s)))
def test_dense_level_alone(ibm, pyoracle, shape, how, relax, options, precision):
    case = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    omega = 1.0 if relax == 2 else 2.0 / 3.0
    orc = pyoracle.Oracle(case, mg_rap=0, mg_relax=relax, mg_group_ratio=1.5, mg_omega=omega, mg_options=options,
                          mg_nu1=3, mg_nu2=3, **HOW[how])
    r = np.random.default_rng(3).standard_normal(orc.box_sizes()[3])
    zo = orc.mg_vcycle(r)
    b = r * case.array("fluid_p").astype(bool)
    for graph in (0, 1):
        s = ibm.Solver(case, ibm.solver_params(precision=precision, use_graph=graph, p_pc_rap_type=0,
                                               p_pc_relax_type=relax, mg_group_ratio=1.5, mg_omega=omega,
                                               mg_options=options, mg_nu1=3, mg_nu2=3, **HOW[how]))
        try:
            z = s.apply_preconditioner(ibm.FIELD_P, r)
            # FP64 and FP32 rounding of the products with the inverse, as for a whole V-cycle
            assert np.abs(z - zo).max() <= (1e-10, 1e-4)[precision] * np.abs(zo).max()
            if precision == 0:
                x, st = s.solve(ibm.FIELD_P, b)
                assert st.status == ibm.IBM_OK and st.iters <= 2
                step = s.step(1.0)
                assert step.p.status == ibm.IBM_OK and step.p.iters <= 2
        finally:
            s.close()
