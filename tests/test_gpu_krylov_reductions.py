"""The FP64 Arnoldi kernels take their dot products eight basis vectors at a
time and reduce one, up to four or up to eight of them across a warp in
different ways; restart lengths around those edges must all reach the
solution of the same system."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kdim", [1, 2, 3, 4, 5, 8, 9, 16, 17, 25])
def test_restart_lengths_reach_the_solution(ibm, kdim, precision):
    # 23 x 9 x 7 leaves a partial tile of rows; a large time step makes the
    # diffusion strong enough for a few dozen Jacobi-preconditioned iterations
    case = ibm.Case(ibm.channel_params(24, 9, 7, Um=1.0, nu=0.05, dt=0.5))
    prm = ibm.solver_params(vel_tol=1e-12, vel_maxit=4000, vel_kdim=kdim, precision=precision, vel_inner_sweeps=2)
    s = ibm.Solver(case, prm)
    try:
        x = np.random.default_rng(kdim).standard_normal(23 * 9 * 7)
        b = s.apply_operator(ibm.FIELD_U, x)
        y, st = s.solve(ibm.FIELD_U, b)
        assert st.status == ibm.IBM_OK
        # the solver's own stop test, and a residual computed apart from it
        # (FP64 rounding of b - A y: about 16 eps |A| |y|)
        r = b - s.apply_operator(ibm.FIELD_U, y)
        bound = 1e-12 * np.linalg.norm(b) + 16 * 2.3e-16 * np.linalg.norm(np.abs(b) + np.abs(y))
        assert np.linalg.norm(r) <= bound
        # |A^-1| <= 1 / min over rows of (diagonal - off-diagonals) of the diagonally dominant rows
        rows = case.array("Au_vals").reshape(-1, 7)
        gap = (np.abs(rows[:, 0]) - np.abs(rows[:, 1:]).sum(1)).min()
        assert gap > 0
        assert np.abs(y - x).max() <= np.abs(r).max() / gap + 1e-14 * np.abs(x).max() / gap
    finally:
        s.close()
