"""The work that the performance of this framework is measured on.

Each case is one pass through the C ABI of include/ibm_gpu.h as a program that
keeps its fields in device memory calls it: timesteps of the channel (plain FP64
and mixed precision, host-driven and graph-captured), one pressure solve, a
forward and reverse pair of adjoint steps, a batch of independent channels, and
the allocation-free residual. Sizes are those of the benchmark, the tests and
the ensemble generator (96..256 x 16..48 x 16..48), with odd grids among them.
"""
import ctypes as C
import functools
import importlib
import math

import numpy as np
import torch

ibm = importlib.import_module("ibm-3d-fpc_gb300")

U, V, W, P = ibm.FIELD_U, ibm.FIELD_V, ibm.FIELD_W, ibm.FIELD_P


def listed():
    return [
        # the smallest call: the reference's example grid with the library's default options (FP64, host-driven loop)
        {"name": "step-default-32x12x12", "kind": "step", "form": "default", "nx": 32, "ny": 12, "nz": 12, "Um": 0.45,
         "dt": 1e-3, "steps": 1, "forces": 0},
        # the small plain run: FP64 steps at 1e-8, captured as a graph
        {"name": "step-fp64-160x32x32", "kind": "step", "form": "fp64", "nx": 160, "ny": 32, "nz": 32, "Um": 0.45,
         "dt": 1e-3, "steps": 2, "forces": 0, "tol": 1e-8},
        # a grid nobody tuned for: odd in every direction, so no pairing of points along a line
        {"name": "step-mixed-97x33x21", "kind": "step", "form": "mixed", "nx": 97, "ny": 33, "nz": 21, "Um": 1.0,
         "dt": 1e-3, "steps": 2, "forces": 0, "tol": 1e-10},
        # an ordinary run: the drag validation's grid, with the cut-surface force of every step
        {"name": "step-mixed-320x64x64", "kind": "step", "form": "mixed", "nx": 320, "ny": 64, "nz": 64, "Um": 0.45,
         "dt": 2e-3, "steps": 1, "forces": 2, "tol": 1e-10},
        # the benchmark: unsteady wake at 10.5M cells, mixed precision, at the tight tolerance of its accuracy study
        {"name": "step-mixed-640x128x128", "kind": "step", "form": "mixed", "nx": 640, "ny": 128, "nz": 128,
         "Um": 2.25, "dt": 2e-4, "steps": 1, "forces": 0, "tol": 1e-10},
        # the same step in plain FP64, the largest of the list
        {"name": "step-fp64-640x128x128", "kind": "step", "form": "fp64", "nx": 640, "ny": 128, "nz": 128,
         "Um": 2.25, "dt": 2e-4, "steps": 1, "forces": 0, "tol": 1e-8},
        # the pressure solver alone on a rough right-hand side, FP32 multigrid inside FP64 flexible GMRES at 1e-10
        {"name": "pressure-512x96x96", "kind": "solve", "form": "fp32mg", "nx": 512, "ny": 96, "nz": 96, "Um": 2.25,
         "dt": 2e-4, "tol": 1e-10},
        # sensitivities: two taped FP64 steps and their reverse steps at 1e-12, as one segment of a gradient sweep
        {"name": "adjoint-256x48x48", "kind": "adjoint", "form": "fp64", "nx": 256, "ny": 48, "nz": 48, "Um": 0.45,
         "dt": 1e-3, "steps": 2, "tol": 1e-12},
        # twelve channels of uneven size stepped together, the ensemble's sizes and solver settings at a tolerance that
        # tells the channels' own errors apart
        {"name": "ensemble-12", "kind": "batch", "form": "mixed", "channels": 12, "draw": 5, "dt": 1e-3, "steps": 2,
         "tol": 1e-12},
        # residual and norms of one operator on the caller's own buffers
        {"name": "residual-512x96x96", "kind": "residual", "nx": 512, "ny": 96, "nz": 96, "Um": 2.25, "dt": 2e-4},
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "solve", "adjoint", "batch", "residual"])
    if kind == "batch":
        return {"kind": kind, "form": rng.choice(["mixed", "fp64"]), "channels": rng.randint(3, 12),
                "draw": rng.randint(6, 10 ** 6), "dt": 1e-3, "steps": rng.randint(1, 3), "tol": 1e-12}
    top = {"step": 640, "solve": 512, "adjoint": 256, "residual": 640}[kind]
    form = {"step": rng.choice(["default", "fp64", "mixed", "mixed"]), "solve": rng.choice(["fp64", "fp32mg"]),
            "adjoint": "fp64", "residual": None}[kind]
    if form == "default":
        top = 96  # its pressure solve takes hundreds of iterations on larger grids
    nx = round(math.exp(rng.uniform(math.log(32), math.log(top))))
    ny, nz = (min(128, max(12, round(nx * rng.uniform(0.16, 0.32)))) for _ in range(2))
    um = round(rng.uniform(0.2, 2.25), 3)
    case = {"kind": kind, "form": form, "nx": nx, "ny": ny, "nz": nz, "Um": um,
            "dt": min(1e-3, round(0.3 * 2.5 / nx / um, 5))}
    cells = nx * ny * nz
    if kind in ("step", "adjoint"):
        case["steps"] = rng.randint(1, 2) if cells < 10 ** 6 else 1
    if kind == "step":
        case["forces"] = rng.choice([0, 0, 2])
    if form not in (None, "default"):
        case["tol"] = {"step": 1e-10 if form == "mixed" else 1e-8, "solve": 1e-10, "adjoint": 1e-12}[kind]
    return case


# ------------------------------------------------------------------ what a program has in hand

@functools.lru_cache(maxsize=48)
def _channel(nx, ny, nz, um, dt, yc=0.2, radius=0.05):
    """The channel's geometry, masks and operators: host set-up that a program does once per channel."""
    return ibm.Case(ibm.channel_params(nx, ny, nz, Um=um, nu=1e-3, dt=dt, ycirc=yc, Rcirc=radius))


def _ensemble(case):
    rng = np.random.default_rng(case["draw"])
    out = []
    for _ in range(case["channels"]):
        nx, ny, nz = (int(rng.integers(a, b)) * 16 for a, b in ((6, 17), (1, 4), (1, 4)))
        d, yc, um = (float(rng.uniform(a, b)) for a, b in ((0.06, 0.14), (0.15, 0.26), (0.2, 2.25)))
        out.append(_channel(nx, ny, nz, um, case["dt"], yc, d / 2))
    return out


def _channel_of(case):
    return _channel(case["nx"], case["ny"], case["nz"], case["Um"], case["dt"])


def _params(case):
    form = case["form"]
    if form == "default":
        return ibm.solver_params()
    tol = case["tol"]
    prm = ibm.solver_params(vel_tol=tol, p_tol=tol, vel_maxit=500, p_maxit=500, p_pc=1, p_pc_rap_type=0,
                            p_pc_relax_type=2, mg_nu1=3, mg_nu2=3, mg_nu_coarse=2, mg_omega=1.0, mg_group_ratio=1.5,
                            mg_coarse_max=640, vel_inner_sweeps=2, use_graph=int(case["kind"] != "solve"),
                            compute_forces=2 if case["kind"] == "adjoint" else case.get("forces", 0))
    if form == "mixed":
        prm.precision, prm.vel_precision, prm.arnoldi_passes = 2, 1, 1
    if form == "fp32mg":
        prm.precision, prm.vel_precision, prm.arnoldi_passes = 1, 1, 1
    return prm


def _fields(channel, gen):
    """A flow under way: the inlet profile led round the body, with 1e-3 N(0, 1) perturbations. Both are the curl of a
    vector potential on the cells' edges that is zero at the body, so the field is divergence-free on the grid as every
    step's end is, and the pressure is zero."""
    cp = channel.params
    nx, ny, nz = channel.shape
    dx, dy, dz = cp.Lx / nx, cp.Ly / ny, cp.Lz / nz
    profile = torch.from_numpy(channel.array("uin").copy()).cuda().view(nz, ny)

    def away(nxp, nyp, offx, offy):  # 0 at the body, 1 away from it and at the walls
        x = (torch.arange(nxp, dtype=torch.float64, device="cuda") + offx) * dx - cp.xcirc
        y = (torch.arange(nyp, dtype=torch.float64, device="cuda") + offy) * dy - cp.ycirc
        near, far = 1.15 * cp.Rcirc + max(dx, dy), 0.98 * min(cp.ycirc, cp.Ly - cp.ycirc)
        t = ((torch.hypot(x[None, :], y[:, None]) - near) / max(far - near, 0.1 * near)).clamp(0, 1)
        return t * t * (3 - 2 * t)

    def noise(shape, h):
        """1e-3 N(0, 1) on the edges in cell widths, zero on the domain's boundary planes."""
        a = 1e-3 * h * torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda")
        for d in (0, 1, 2):
            if shape[d] == (nz, ny, nx)[d] + 1:
                a.narrow(d, 0, 1).zero_()
                a.narrow(d, shape[d] - 1, 1).zero_()
        return a

    # the profile's potential: its integral over y from the body's centre
    psi = torch.cat([torch.zeros_like(profile[:, :1]), torch.cumsum(profile, 1) * dy], 1)
    at = cp.ycirc / dy - math.floor(cp.ycirc / dy)
    j = int(cp.ycirc / dy)
    psi = psi - ((1 - at) * psi[:, j:j + 1] + at * psi[:, j + 1:j + 2])
    az = (psi[:, :, None] + noise((nz, ny + 1, nx + 1), min(dx, dy))) * away(nx + 1, ny + 1, 0.0, 0.0)
    ax = noise((nz + 1, ny + 1, nx), min(dy, dz)) * away(nx, ny + 1, 0.5, 0.0)
    ay = noise((nz + 1, ny, nx + 1), min(dx, dz)) * away(nx + 1, ny, 0.0, 0.5)
    u = az.diff(dim=1) / dy - ay.diff(dim=0) / dz
    v = ax.diff(dim=0) / dz - az.diff(dim=2) / dx
    w = ay.diff(dim=2) / dx - ax.diff(dim=1) / dy
    p = torch.zeros(nx * ny * nz, dtype=torch.float64, device="cuda")
    return [u.flatten(), v.flatten(), w.flatten(), p]


def _at(*tensors):
    return [C.c_void_p(t.data_ptr()) for t in tensors]


def prepare(case, seed):
    gen = torch.Generator("cuda").manual_seed(int(seed))
    kind = case["kind"]
    state = {"case": case}
    if kind == "batch":
        channels = _ensemble(case)
        state["batch"] = ibm.Batch(channels, _params(case))
        state["solvers"] = state["batch"].solvers
        state["in"] = [_fields(c, gen) for c in channels]
    elif kind == "residual":
        n = case["nx"] * case["ny"] * case["nz"]
        state["vals"] = torch.from_numpy(_channel_of(case).array("Ap_vals").copy()).cuda()
        state["x"], state["b"] = (torch.randn(n, generator=gen, dtype=torch.float64, device="cuda") for _ in range(2))
        state["r"] = torch.empty_like(state["b"])
        state["norms"] = torch.empty(2, dtype=torch.float64, device="cuda")
        state["lib"] = importlib.import_module("ibm-3d-fpc_gb300._native").gpu()
        state["lib"].ibm_residual_noalloc.argtypes = [C.c_void_p] + [C.c_int] * 3 + [C.c_void_p] * 5
        return state
    else:
        channel = _channel_of(case)
        state["solvers"] = [ibm.Solver(channel, _params(case))]
        state["in"] = [_fields(channel, gen)]
        if kind == "solve":
            fluid = torch.from_numpy(channel.array("fluid_p").copy()).cuda().double()
            b = torch.randn(fluid.numel(), generator=gen, dtype=torch.float64, device="cuda") * fluid
            state["b"] = b - fluid * (b.sum() / fluid.sum())  # no net source over the fluid
            state["x"] = torch.empty_like(b)
            state["stream"] = torch.cuda.ExternalStream(state["solvers"][0]._lib.ibm_stream(state["solvers"][0]._ctx))
        if kind == "adjoint":
            state["solvers"][0].adjoint_setup()
            state["lambda"] = [torch.randn(t.numel(), generator=gen, dtype=torch.float64, device="cuda")
                               for t in state["in"][0]]
            sizes = [t.numel() for t in state["in"][0]] + [case["ny"] * case["nz"], 1]
            state["grad"] = [torch.empty(n, dtype=torch.float64, device="cuda") for n in sizes]
    state["out"] = [[torch.empty_like(t) for t in f] for f in state["in"]]
    torch.cuda.synchronize()
    run(state)  # a program's solver objects have their hierarchy and captured step when its time loop begins
    return state


# ------------------------------------------------------------------ one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "residual":
        rc = state["lib"].ibm_residual_noalloc(*_at(state["vals"]), case["nx"], case["ny"], case["nz"],
                                               *_at(state["x"], state["b"], state["r"], state["norms"]),
                                               C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc < 0:
            raise ibm.IBMError(rc, "ibm_residual_noalloc")
        return [state["r"], state["norms"]]
    solvers = state["solvers"]
    if kind == "solve":
        s, st = solvers[0], ibm._native.SolveStats()
        with torch.cuda.stream(state["stream"]):
            state["x"].zero_()
        s._check(s._lib.ibm_solve(s._ctx, P, *_at(state["b"], state["x"]), C.byref(st)))
        return [state["x"]]
    for s, f in zip(solvers, state["in"]):
        s._check(s._lib.ibm_set_fields(s._ctx, *_at(*f)))
    if kind == "adjoint":
        s = solvers[0]
        s.adjoint_reset()
        s._check(s._lib.ibm_adjoint_set(s._ctx, *_at(*state["lambda"])))
        for _ in range(case["steps"]):
            s.step_forward(1.0)
        for _ in range(case["steps"]):
            s.step_backward(1.0, 0.5)
        s._check(s._lib.ibm_adjoint_get(s._ctx, *_at(*state["grad"])))
        return state["grad"]
    for _ in range(case["steps"]):
        if kind == "batch":
            state["batch"].step(1.0)
        else:
            st = solvers[0].step(1.0)
    for s, f in zip(solvers, state["out"]):
        s._check(s._lib.ibm_get_fields(s._ctx, *_at(*f)))
    if kind == "batch":
        return [[t for t in f] for f in state["out"]]
    return [state["out"][0], st.force[0]] if case["forces"] else [state["out"][0]]


def work(case):
    """Every input of a pass read once and every result written once; operations of the iterations that the
    benchmark's solver settings take (three per momentum solve, seven per pressure solve)."""
    if case["kind"] == "batch":
        cells = sum(math.prod(c.shape) for c in _ensemble(case))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "residual":  # 7 coefficients, x and b in, r out
        return {"bytes": 80.0 * cells, "flops": 19.0 * cells}
    vcycle = 2 * 6 * 13 + 40  # six sweeps of the finest level, the coarser ones about a quarter of them
    pressure = 7 * (vcycle + 14 + 4 * 8)
    if case["kind"] == "solve":  # the operator and b in, x out
        return {"bytes": 72.0 * cells, "flops": float(pressure * cells)}
    # the four operators, D and G, the row scales and lifts (one pass over them at least), and the fields in and out
    step = {"bytes": (4 * 56 + 48 + 48 + 48) * cells, "flops": (3 * (60 + 3 * (14 + 14 + 4 * 3)) + pressure) * cells}
    fields = 64.0 * cells
    n = case["steps"] * (2 if case["kind"] == "adjoint" else 1)
    return {"bytes": n * step["bytes"] + fields, "flops": float(n * step["flops"])}


# ------------------------------------------------------------------ the same results in plain 64-bit torch

def _stencil(vals, x):
    """A x for row-major 7-point rows (centre, -x, +x, -y, +y, -z, +z) as seven planes; x is [nz, ny, nx]."""
    y = vals[0] * x
    y[:, :, 1:] += vals[1][:, :, 1:] * x[:, :, :-1]
    y[:, :, :-1] += vals[2][:, :, :-1] * x[:, :, 1:]
    y[:, 1:] += vals[3][:, 1:] * x[:, :-1]
    y[:, :-1] += vals[4][:, :-1] * x[:, 1:]
    y[1:] += vals[5][1:] * x[:-1]
    y[:-1] += vals[6][:-1] * x[1:]
    return y


def _planes(channel, name, nx, ny, nz):
    rows = torch.from_numpy(channel.array(name).copy()).cuda().view(nz, ny, nx, 7)
    return [rows[..., s].contiguous() for s in range(7)]


def _conjugate_gradients(vals, weight, b):
    """x of A x = b where diag(weight) A is symmetric positive definite: Jacobi-preconditioned conjugate gradients,
    refined from the true residual until that stops falling."""
    scaled = [weight * v for v in vals]
    b = weight * b
    x, best, best_x = torch.zeros_like(b), math.inf, None
    norm = float(b.norm()) or 1.0
    for _ in range(6):
        r = b - _stencil(scaled, x)
        now = float(r.norm())
        if now >= 0.5 * best or now <= 1e-16 * norm:
            break
        best, best_x = now, x.clone()
        z = r / scaled[0]
        d, rz = z.clone(), torch.dot(r.flatten(), z.flatten())
        e = torch.zeros_like(x)
        for it in range(20000):
            q = _stencil(scaled, d)
            a = rz / torch.dot(d.flatten(), q.flatten())
            e += a * d
            r -= a * q
            if it % 25 == 24 and float(r.norm()) <= 1e-9 * now:
                break
            z = r / scaled[0]
            new = torch.dot(r.flatten(), z.flatten())
            d = z + (new / rz) * d
            rz = new
        x = x + e
    r = b - _stencil(scaled, x)
    return x if best_x is None or float(r.norm()) < best else best_x


def _jacobi(vals, b):
    """x of A x = b for the diagonally dominant momentum rows: Richardson steps on the scaled residual."""
    x, last = torch.zeros_like(b), math.inf
    for _ in range(2000):
        r = (b - _stencil(vals, x)) / vals[0]
        now = float(r.norm())
        if now >= last and now <= 1e-12 * float(x.norm()):
            break
        x, last = x + r, now
    return x


def _pressure_weight(channel):
    nx, ny, nz = channel.shape
    fluid = torch.from_numpy((channel.array("fluid_p").astype(bool) & (channel.array("id_p") > 0)).copy()).cuda()
    beta = torch.from_numpy(channel.array("beta_p").astype(np.float64)).cuda()
    return torch.where(fluid, beta, torch.ones_like(beta)).view(nz, ny, nx)


class _Steps:
    """The timestep in torch: boundary cleanup, centred convection, pressure gradient, implicit diffusion of the
    three velocities, pressure equation, projection."""

    def __init__(self, channel):
        a, cp = channel.array, channel.params
        nx, ny, nz = channel.shape
        self.shape = nx, ny, nz
        self.rho, self.dt = cp.rho, cp.dt
        self.h = 2 * cp.Lx / nx, 2 * cp.Ly / ny, 2 * cp.Lz / nz  # centred differences span two cells

        def t(name, kind=None):
            return torch.from_numpy((a(name) if kind is None else a(name).astype(kind)).copy()).cuda()

        full = {"u": (nz, ny, nx + 1), "v": (nz, ny + 1, nx), "w": (nz + 1, ny, nx), "p": (nz, ny, nx)}
        self.full = full
        self.active = {f: t("active_" + f, bool).view(full[f]) for f in "uvw"}
        ids = {f: t("id_" + f, np.int64).view(full[f]) for f in "uvwp"}
        self.scale = {f: t("scale_" + f)[ids[f]] for f in "uvw"}
        self.lift = {f: t("rhs_%s_bc" % f)[ids[f]] for f in "uvw"}
        self.rows = {f: (ids[f] > 0) & self.active[f] for f in "uvw"}
        self.fluid = t("fluid_p", bool).view(full["p"]) & (ids["p"] > 0)
        self.pid = ids["p"]
        self.div_bc = t("div_bc_unit")
        self.uin = t("uin").view(nz, ny)
        self.q = [t("id_q" + f, np.int64).view(full[f]) for f in "uvw"]
        n = channel.counts
        self.nq, self.np_ = [n["nqu"], n["nqv"], n["nqw"]], n["np"]
        # rows and columns of D and G are numbered from 1; index 0 is a zero
        self.D, self.G = (self._coo(t(k + "_rowptr", np.int64), t(k + "_col", np.int64), t(k + "_val")) for k in "DG")
        boxes = {"u": (nx - 1, ny, nz), "v": (nx, ny - 1, nz), "w": (nx, ny, nz - 1), "p": (nx, ny, nz)}
        self.A = {f: _planes(channel, "A%s_vals" % f, *boxes[f]) for f in "uvwp"}
        self.weight = _pressure_weight(channel)

    @staticmethod
    def _coo(rowptr, col, val):
        row = torch.arange(1, rowptr.numel(), device="cuda")
        return torch.repeat_interleave(row, rowptr[1:] - rowptr[:-1]), col, val

    def _csr(self, M, x, n):
        row, col, val = M
        return torch.zeros(n + 1, dtype=torch.float64, device="cuda").index_add_(0, row, val * x[col])

    def gradient(self, p):
        x = torch.zeros(self.np_ + 1, dtype=torch.float64, device="cuda")
        x[self.pid[self.fluid]] = p[self.fluid]
        return self._csr(self.G, x, sum(self.nq))

    def faces(self, g):
        out, at = [], 0
        for ids, n in zip(self.q, self.nq):
            out.append(torch.where(ids > 0, g[torch.where(ids > 0, ids + at, 0)], 0.0))
            at += n
        return out

    def pack(self, fields):
        q, at = torch.zeros(sum(self.nq) + 1, dtype=torch.float64, device="cuda"), 0
        for ids, n, f in zip(self.q, self.nq, fields):
            q[ids[ids > 0] + at] = f[ids > 0]
            at += n
        return q

    def cleanup(self, u, v, w):
        u[:, :, 0] = self.uin
        u[:, :, -1] = u[:, :, -2]
        v[:, 0] = v[:, -1] = 0.0
        w[0] = w[-1] = 0.0
        u[:, :, 1:-1][~self.active["u"][:, :, 1:-1]] = 0.0
        v[:, 1:-1][~self.active["v"][:, 1:-1]] = 0.0
        w[1:-1][~self.active["w"][:-2]] = 0.0  # the mask of the plane below

    @staticmethod
    def _slope(x, dim, span):
        """Centred difference over two cells; outside the array the centre's own value."""
        n = x.shape[dim]
        up = torch.cat([x.narrow(dim, 1, n - 1), x.narrow(dim, n - 1, 1)], dim)
        down = torch.cat([x.narrow(dim, 0, 1), x.narrow(dim, 0, n - 1)], dim)
        return (up - down) / span

    @staticmethod
    def _mean(x, a, b):
        """Mean of the four values around: neighbours along dimensions a and b."""
        for d in (a, b):
            x = x.narrow(d, 0, x.shape[d] - 1) + x.narrow(d, 1, x.shape[d] - 1)
        return 0.25 * x

    def convection(self, u, v, w):
        hx, hy, hz = self.h
        c = {f: torch.zeros(self.full[f], dtype=torch.float64, device="cuda") for f in "uvw"}
        in_u, in_v, in_w = (slice(None), slice(None), slice(1, -1)), (slice(None), slice(1, -1)), (slice(1, -1),)
        du, dv, dw = ([self._slope(x, d, s) for d, s in ((2, hx), (1, hy), (0, hz))] for x in (u, v, w))
        c["u"][in_u] = (u * du[0])[in_u] + self._mean(v, 1, 2) * du[1][in_u] + self._mean(w, 0, 2) * du[2][in_u]
        c["v"][in_v] = self._mean(u, 2, 1) * dv[0][in_v] + (v * dv[1])[in_v] + self._mean(w, 0, 1) * dv[2][in_v]
        c["w"][in_w] = self._mean(u, 2, 0) * dw[0][in_w] + self._mean(v, 1, 0) * dw[1][in_w] + (w * dw[2])[in_w]
        below = torch.cat([self.active["w"][:1], self.active["w"][:-1]])
        return [torch.where(m, c[f], 0.0) for f, m in (("u", self.active["u"]), ("v", self.active["v"]), ("w", below))]

    def step(self, fields):
        u, v, w, p = (x.clone() for x in fields)
        inner = {"u": (slice(None), slice(None), slice(1, -1)), "v": (slice(None), slice(1, -1)), "w": (slice(1, -1),)}
        self.cleanup(u, v, w)
        a = self.rho / self.dt
        for f, x, conv, g in zip("uvw", (u, v, w), self.convection(u, v, w), self.faces(self.gradient(p))):
            rhs = (a * x - self.rho * conv - g + self.lift[f]) * self.scale[f]
            rhs = torch.where(self.rows[f], rhs, 0.0)[inner[f]]
            x[inner[f]] = _jacobi(self.A[f], rhs.contiguous())
        self.cleanup(u, v, w)
        q = self.pack((u, v, w))
        div = self._csr(self.D, q, self.np_)
        b = torch.where(self.fluid, -a * (div + self.div_bc)[self.pid], 0.0)
        phi = _conjugate_gradients(self.A["p"], self.weight, b)
        q = q - (self.dt / self.rho) * self.gradient(phi)
        q[0] = 0.0
        for x, ids, new in zip((u, v, w), self.q, self.faces(q)):
            x[ids > 0] = new[ids > 0]
        self.cleanup(u, v, w)
        return u, v, w, torch.where(self.fluid, p + phi, p)


def _exact_steps(channel, fields, steps):
    s = _Steps(channel)
    fields = [x.view(s.full[f]) for f, x in zip("uvwp", fields)]
    for _ in range(steps):
        fields = s.step(fields)
    return [x.flatten() for x in fields]


def exact(case, seed):
    gen = torch.Generator("cuda").manual_seed(int(seed))
    kind = case["kind"]
    if kind == "adjoint":
        return None  # a reverse sweep: there is no plain form of it to write down beside the library's own
    if kind == "batch":
        channels = _ensemble(case)
        inputs = [_fields(c, gen) for c in channels]
        return [_exact_steps(c, f, case["steps"]) for c, f in zip(channels, inputs)]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    channel = _channel_of(case)
    if kind == "residual":
        x, b = (torch.randn(nx * ny * nz, generator=gen, dtype=torch.float64, device="cuda") for _ in range(2))
        r = b - _stencil(_planes(channel, "Ap_vals", nx, ny, nz), x.view(nz, ny, nx)).flatten()
        return [r, torch.stack([r.norm(), b.norm()])]
    fields = _fields(channel, gen)
    if kind == "solve":
        fluid = torch.from_numpy(channel.array("fluid_p").copy()).cuda().double()
        b = torch.randn(fluid.numel(), generator=gen, dtype=torch.float64, device="cuda") * fluid
        b = b - fluid * (b.sum() / fluid.sum())
        return [_conjugate_gradients(_planes(channel, "Ap_vals", nx, ny, nz), _pressure_weight(channel),
                                     b.view(nz, ny, nx)).flatten()]
    out = _exact_steps(channel, fields, case["steps"])
    return [out, None] if case["forces"] else [out]
