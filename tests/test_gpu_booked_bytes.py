"""Algorithmic bytes booked for the colour phases of the finest FP32 level: x and
b of a phase, and a class code only for the points outside the runs of 32 units
(octets within a solve, quads of a single application) whose records are all the
most common one, which the kernels read from their parameters. Expected from
the operator's rows; three sweeps each way are 12 launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def share_outside_runs(case, unit):
    nx, ny, nz = case.shape
    a = case.array("Ap_vals").reshape(-1, 7)
    with np.errstate(divide="ignore"):
        inv = np.where(a[:, 0] != 0, 1 / a[:, 0], 0.0)
    rec = np.concatenate([inv[:, None], a[:, 1:], a[:, :1]], axis=1).astype(np.float32)
    _, code, count = np.unique(rec.view(np.uint32), axis=0, return_inverse=True, return_counts=True)
    major = (code.reshape(-1) == np.argmax(count)).reshape(ny * nz, nx // unit, unit).all(axis=2)
    # units inside the lines first, then the two at each line's ends
    order = np.concatenate([major[:, 1:-1].ravel(), major[:, [0, -1]].ravel()])
    runs = [order[q:q + 32] for q in range(0, order.size, 32)]
    return sum(r.size for r in runs if not r.all()) / order.size


@pytest.mark.parametrize("form", ["solve", "application"])
def test_bytes_of_fine_phases(ibm, form):
    case = ibm.Case(ibm.channel_params(128, 32, 32, Um=1.0, dt=1e-3))
    n = 128 * 32 * 32
    s = ibm.Solver(case, ibm.solver_params(precision=2, p_maxit=1, p_pc_rap_type=0, p_pc_relax_type=2, mg_nu1=3,
                                           mg_nu2=3, mg_group_ratio=1.5, mg_omega=1.0, mg_options=0, mg_coarse_max=64))
    try:
        b = np.random.default_rng(1).standard_normal(n) * case.array("fluid_p").astype(bool)
        s.apply_preconditioner(ibm.FIELD_P, b)  # builds the hierarchy
        k = ibm.kernel_names().index("mg_relax_fine")
        s.profile_reset()
        if form == "solve":
            s.solve(ibm.FIELD_P, b)
            # input read and b written beside the first phase, the output beside the last
            fixed, share = 12 * 6 + 6 + 2, share_outside_runs(case, 8)
        else:
            s.apply_preconditioner(ibm.FIELD_P, b)
            fixed, share = 12 * 6, share_outside_runs(case, 4)
        p = s.profile()
        assert p.launches[k] == 12
        assert 0.05 < share < 0.9
        assert abs(p.bytes[k] - n * (fixed + 12 * share)) <= 1e-9 * p.bytes[k]
    finally:
        s.close()


def common(records):
    """Which records are the most frequent one that is not all zeros."""
    _, code, count = np.unique(np.ascontiguousarray(records).view(np.uint64), axis=0, return_inverse=True,
                               return_counts=True)
    code = code.reshape(-1)
    zeros = ~records.any(axis=1)
    count[np.unique(code[zeros])] = 0
    return code == np.argmax(count)


def common_faces(case):
    """Faces between two cells whose G pair is their field's common one."""
    ptr, val = case.array("G_rowptr"), case.array("G_val")
    n, first = 0, 0
    for name in ("nqu", "nqv", "nqw"):
        rows = np.arange(first, first + case.counts[name])
        first += case.counts[name]
        two = rows[np.diff(ptr)[rows] == 2]
        n += common(np.stack([val[ptr[two]], val[ptr[two] + 1]], axis=1)).sum()
    return int(n)


def common_rows(case):
    nx, ny, nz = case.shape
    n = 0
    for f, shape, inner in (("u", (nz, ny, nx + 1), np.s_[:, :, 1:-1]), ("v", (nz, ny + 1, nx), np.s_[:, 1:-1, :]),
                            ("w", (nz + 1, ny, nx), np.s_[1:-1, :, :])):
        ids = case.array("id_" + f).reshape(shape)[inner].ravel()
        active = case.array("active_" + f).reshape(shape)[inner].ravel()
        ids = np.where(active != 0, ids, 0)
        rec = np.stack([case.array("scale_" + f)[ids], case.array(f"rhs_{f}_bc")[ids]], axis=1)
        rec[ids == 0] = 0.0
        n += int(common(rec).sum())
    return n


def test_bytes_of_dense_kernels(ibm):
    """Scale, boundary term, G and cell flags are booked only for the rows and
    faces that do not share the common ones."""
    nx, ny, nz = shape = (64, 24, 20)
    case = ibm.Case(ibm.channel_params(*shape, Um=1.0, dt=1e-3))
    s = ibm.Solver(case, ibm.solver_params())
    try:
        s.step(1.0)
        s.profile_reset()
        s.step(1.0)
        p, names = s.profile(), ibm.kernel_names()
        booked = {name: p.bytes[k] for k, name in enumerate(names)}
        faces = (nx + 1) * ny * nz + nx * (ny + 1) * nz + nx * ny * (nz + 1)
        box = (nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1)
        cells = nx * ny * nz
        pf, pr = common_faces(case), common_rows(case)
        assert 0.5 * faces < pf < faces and 0.3 * box < pr < box
        assert booked["scatter"] == 16 * faces
        assert booked["project"] == 17 * faces + 18 * (faces - pf) + 25 * cells
        assert booked["momentum_rhs"] == 8 * faces + 8 * cells + 17 * box + 16 * (box - pr) + 18 * (box - pf)
        assert 8 * faces + cells < booked["diagnostics"] < 8 * faces + 63 * cells
    finally:
        s.close()
