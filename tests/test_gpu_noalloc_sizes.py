"""ibm_residual_noalloc at the edges of its split: fewer rows than a warp, one
more or less than a warp's chunk, a block's, and a resident wave's with a
remainder, one-point-thick boxes, and coefficients aligned to 8 bytes only.
Against the same sum in numpy: a row is eight products and sums, so each side
is within 8 u of the exact row relative to its terms' magnitudes (u = 2^-53)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOXES = [(1, 1, 1), (5, 1, 1), (31, 1, 1), (1, 32, 1), (33, 1, 1), (255, 1, 1), (1, 1, 257), (7, 5, 3), (64, 8, 8),
         (641, 33, 25)]


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("box", BOXES, ids=lambda b: "x".join(map(str, b)))
def test_residual_sizes(ibm, box, offset):
    torch = pytest.importorskip("torch")
    nx, ny, nz = box
    n = nx * ny * nz
    lib = ibm._native.gpu()
    f = lib.ibm_residual_noalloc
    f.argtypes = [C.c_void_p] + [C.c_int] * 3 + [C.c_void_p] * 5
    f.restype = C.c_int
    rng = np.random.default_rng(n)
    vals, x, b = rng.standard_normal((n, 7)), rng.standard_normal(n), rng.standard_normal(n)
    x3 = x.reshape(nz, ny, nx)
    pad = np.pad(x3, 1)
    nb = [x3, pad[1:-1, 1:-1, :-2], pad[1:-1, 1:-1, 2:], pad[1:-1, :-2, 1:-1], pad[1:-1, 2:, 1:-1], pad[:-2, 1:-1, 1:-1],
          pad[2:, 1:-1, 1:-1]]
    terms = np.stack([vals[:, s] * nb[s].ravel() for s in range(7)])
    ref, mag = b - terms.sum(0), np.abs(b) + np.abs(terms).sum(0)
    buf = torch.zeros(7 * n + 1, dtype=torch.float64, device="cuda")
    dv = buf[offset:offset + 7 * n]
    dv.copy_(torch.from_numpy(vals.ravel()))
    dx, db = torch.from_numpy(x).cuda(), torch.from_numpy(b).cuda()
    r, norms = torch.full_like(db, float("nan")), torch.full((2,), float("nan"), dtype=torch.float64, device="cuda")
    rc = f(dv.data_ptr(), nx, ny, nz, dx.data_ptr(), db.data_ptr(), r.data_ptr(), norms.data_ptr(),
           torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    assert np.all(np.abs(r.cpu().numpy() - ref) <= 16 * 2.0 ** -53 * mag)
    got = norms.cpu().numpy()
    # sums of at most 2^20 squares, chains of some hundred additions
    assert abs(got[0] - np.linalg.norm(r.cpu().numpy())) <= 1e-12 * got[0]
    assert abs(got[1] - np.linalg.norm(b)) <= 1e-12 * got[1]
