"""The dense kernels take the coefficients that most faces, rows and cells share
from their parameters, where flags derived from the inputs say so. New inputs
on a context that has stepped already, and an inflow profile set between
steps, must give the bits that a fresh context gives: every flag and common
value is derived anew (the grid, dt and nu are the context's own). Grids with and without a plain interior (3 cells
thick), the body moved and resized, FP64 and double-float right-hand sides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = {"fp64": {}, "mixed": dict(precision=2, vel_precision=1, p_pc=1, p_pc_rap_type=0, p_pc_relax_type=2,
                                   vel_inner_sweeps=2)}


def same_bits(a, b):
    return all(np.array_equal(x.view(np.uint64), y.view(np.uint64)) for x, y in zip(a, b))


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("shape", [(32, 12, 12), (37, 15, 13), (24, 8, 3)])
def test_new_inputs_on_a_used_context(ibm, shape, form):
    first = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    p = ibm.channel_params(*shape, Um=0.7, dt=1e-3)
    p.xcirc, p.ycirc, p.Rcirc = 1.2 * p.xcirc, 0.9 * p.ycirc, 0.8 * p.Rcirc
    second = ibm.Case(p)
    prm = ibm.solver_params(**FORMS[form])
    a = ibm.Solver(first, prm)
    fresh = ibm.Solver(second, prm)
    try:
        a.step(1.0)
        b = ibm.Solver(second, prm, _ctx=a._ctx.value)
        for ramp in (0.5, 1.0):
            b.step(ramp)
            fresh.step(ramp)
        assert same_bits(b.fields(), fresh.fields())
        assert all(np.all(np.isfinite(f)) for f in b.fields())
    finally:
        a.close()
        fresh.close()


@pytest.mark.parametrize("form", FORMS)
def test_inflow_set_between_steps(ibm, form):
    case = ibm.Case(ibm.channel_params(32, 12, 12, Um=1.0, dt=1e-3))
    prm = ibm.solver_params(**FORMS[form])
    g = 0.8 * np.ascontiguousarray(case.array("uin"), dtype=np.float64)
    a, b = ibm.Solver(case, prm), ibm.Solver(case, prm)
    try:
        a.adjoint_setup()
        b.adjoint_setup()
        a.step(1.0)
        a.set_inflow(g)
        b.set_inflow(g)
        a.set_fields(*case.initial_fields())
        a.step(1.0)
        b.step(1.0)
        assert same_bits(a.fields(), b.fields())
    finally:
        a.close()
        b.close()
