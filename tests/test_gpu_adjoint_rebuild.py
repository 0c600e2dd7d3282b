"""The captured reverse sweep holds the solvers' buffers, the multigrid levels and
the kind of force. Whatever rebuilds or changes them after a sweep was captured
(solver parameters that the transposed context does not share, an operator or
all inputs given again), before or between a step and its reverse, the next
reverse step must give what a fresh context gives with the same settings."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPE = (32, 12, 12)


def params(ibm, **kw):
    base = dict(vel_tol=1e-13, p_tol=1e-13, vel_maxit=500, p_maxit=20000, precision=0, use_graph=1, p_pc=1,
                p_pc_rap_type=0, p_pc_relax_type=2, mg_group_ratio=1.5, compute_forces=1)
    base.update(kw)
    return ibm.solver_params(**base)


def sweep(s, state, lam, between=lambda s: None):
    s.set_fields(*state)
    s.adjoint_reset()
    s.step_forward(1.0)
    between(s)
    s.adjoint_set(*lam)
    assert s.step_backward(1.0, weight=0.3).status == 0
    out = s.adjoint_get()
    return list(out[:5]) + [np.array([out[5]])]


def operator_again(ibm, case):
    v = case.array("Ap_vals")
    return lambda s: s._check(s._lib.ibm_set_operator(s._ctx, ibm.FIELD_P, C.c_void_p(v.ctypes.data), *SHAPE))


CHANGES = {"cut-force": (dict(compute_forces=1), dict(compute_forces=2)),
           "forces-on": (dict(compute_forces=0), dict(compute_forces=1)),
           "to-jacobi": (dict(p_pc=1), dict(p_pc=0)),
           "to-multigrid": (dict(p_pc=0), dict(p_pc=1)),
           "tighter-cycles": (dict(p_kdim=50), dict(p_kdim=7)),
           "to-mixed": (dict(precision=0), dict(precision=1))}


@pytest.mark.parametrize("when", ["before-the-step", "before-its-reverse"])
@pytest.mark.parametrize("change", list(CHANGES) + ["operator", "inputs"])
def test_reverse_step_after_a_change(ibm, change, when):
    case = ibm.Case(ibm.channel_params(*SHAPE, Um=1.0, dt=2e-3))
    first, second = CHANGES.get(change, ({}, {}))
    if change == "operator":
        apply = operator_again(ibm, case)
    elif change == "inputs":
        def apply(s):
            fields = s.fields()
            ibm.Solver(case, s.params, _ctx=s._ctx.value).set_fields(*fields)
    else:
        def apply(s):
            s.set_params(params(ibm, **second))
    rng = np.random.default_rng(4)
    state = case.initial_fields()
    lam = [rng.standard_normal(x.size) for x in state]
    a, b = ibm.Solver(case, params(ibm, **first)), ibm.Solver(case, params(ibm, **second))
    try:
        a.adjoint_setup()
        b.adjoint_setup()
        sweep(a, state, lam)  # captures the reverse sweep
        if when == "before-the-step":
            apply(a)
            got = [sweep(a, state, lam)]
        else:
            got = [sweep(a, state, lam, apply), sweep(a, state, lam)]
        want = sweep(b, state, lam)
        # the systems are solved to 1e-13; the sweep's sums are atomic
        for g in got:
            for x, y in zip(g, want):
                assert np.abs(x - y).max() <= 1e-8 * np.abs(y).max()
    finally:
        a.close()
        b.close()
