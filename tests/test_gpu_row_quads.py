"""Classed rows are taken four at a time by the Jacobi sweeps where a box is a
multiple of four rows, on lines of whole quads or over the ends of lines and
planes. Plain coefficient planes (row_classes 0) are the same values in the same
order, so mixed steps must agree bit for bit. Lines of 3 to 9 rows, planes of a
multiple of four rows and not, boxes that are no multiple of four (one row at a
time)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(4, 4, 4), (6, 4, 8), (7, 6, 8), (8, 8, 8), (9, 8, 12), (10, 7, 9), (37, 15, 13), (33, 16, 12)]


@pytest.mark.parametrize("sweeps", [2, 4])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_classed_rows_equal_planes(ibm, shape, sweeps):
    case = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    fields = []
    for classes in (1, 0):
        s = ibm.Solver(case, ibm.solver_params(row_classes=classes, df_spmv=0, df_residual=0, precision=2, vel_precision=1,
                                               vel_inner_sweeps=sweeps, p_pc=1, p_pc_rap_type=0, p_pc_relax_type=2))
        for _ in range(2):
            s.step(1.0)
        fields.append(s.fields())
        s.close()
    for x, y in zip(*fields):
        assert np.all(np.isfinite(x))
        assert np.array_equal(x.view(np.uint64), y.view(np.uint64))
