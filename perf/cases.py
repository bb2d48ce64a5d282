"""Timed workloads of the vlp4d library, through its Python binding.

Each case is one call or one short sequence of calls that a program makes on
states it already holds on the GPU: the time loop in both precisions, the
separate sweeps that the reference's own time step calls, the moment and
field solve, the reverse mode, a batched ensemble, and the vlp4d_mpi step in
its fused and its call-by-call form.  `exact` restates each of them in 64-bit
torch from the formulas alone.

Arrays of f have shape (nvy, nvx, ny, nx), fields (ny, nx).
"""
import math

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.load_package()
v = pkg.vlp4d

TWO_PI = 2 * math.pi
MPI_L = 12.56637112  # x, y in [0, MPI_L), the box of the SLD10 deck


# ---------------------------------------------------------------- the cases
def _case(kind, n, dtype, steps=1, **more):
    nx, ny, nvx, nvy = n
    return {"kind": kind, "nx": nx, "ny": ny, "nvx": nvx, "nvy": nvy, "dtype": dtype, "steps": steps, **more}


def listed():
    return [
        # The moment, the field solve and the diagnostic of a small state: the
        # smallest calls there are (a program that drives its own time step, or
        # restarts, makes them between everything else).
        {"name": "field_16", **_case("field", (16, 16, 16, 16), "f64")},
        # A whole small run as the CPU-sized Landau configuration does it
        # (32^4, FP64, dt 0.125): initial field, time loop, energy history.
        {"name": "run_32_f64", **_case("run", (32, 32, 32, 32), "f64", 10, dt=0.125, ic="landau")},
        # The headline configuration: Landau damping 128^4, FP32 storage.
        {"name": "loop_128_f32", **_case("loop", (128, 128, 128, 128), "f32", 4, dt=0.1, ic="landau")},
        # The same in plain FP64.
        {"name": "loop_128_f64", **_case("loop", (128, 128, 128, 128), "f64", 2, dt=0.1, ic="landau")},
        # The two-stream configuration, 64 x 64 x 128 x 128.
        {"name": "loop_two_stream_f32", **_case("loop", (64, 64, 128, 128), "f32", 4, dt=0.05, ic="two_stream")},
        # A grid that is no power of two, in the even sizes people choose
        # (72 x 60 points of space, 96 x 80 of velocity).
        {"name": "loop_72x60x96x80_f32", **_case("loop", (72, 60, 96, 80), "f32", 3, dt=0.1, ic="landau")},
        # Odd extents in every dimension (an odd number of velocity points
        # puts one at v = 0): any grid the library accepts runs the same loop.
        {"name": "loop_45x39x51x43_f64", **_case("loop", (45, 39, 51, 43), "f64", 3, dt=0.1, ic="landau")},
        # One time step through the separate entry points, as the
        # reference's own onetimestep calls them (drop-in use).
        {"name": "sweeps_64_f64", **_case("sweeps", (64, 64, 64, 64), "f64", 1, dt=0.1, ic="landau")},
        # The reverse mode of the adjoint configuration (64^4, FP32, a
        # checkpoint every 8 steps): forward and backward over 16 steps.
        {"name": "reverse_64_f32", **_case("reverse", (64, 64, 64, 64), "f32", 16, dt=0.1, every=8)},
        # A batch of uneven small members in one launch, and their results.
        {"name": "ensemble_60", "kind": "ensemble", "members": 60, "grids": 11, "steps": 20, "dtype": "f32"},
        # The fused vlp4d_mpi step on the grid of its SLD10 deck.
        {"name": "mpi_step_128", **_case("mpi_step", (128, 128, 128, 128), "f64", 1, dt=0.01)},
        # The same step call by call in the reference's order and arithmetic,
        # on a ragged grid.
        {"name": "mpi_calls_48x44x40x36", **_case("mpi_calls", (48, 44, 40, 36), "f64", 1, dt=0.01)},
    ]


def _size(rng, lo, hi):
    n = math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))
    step = rng.choice((1, 1, 2, 4, 8, 16))
    return min(hi, max(lo, int(n) // step * step))


def draw(rng):
    kind = rng.choice(("field", "run", "loop", "loop", "loop", "sweeps", "reverse", "ensemble", "mpi_step", "mpi_calls"))
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(4, 62), "grids": rng.randrange(1 << 20), "steps": rng.randint(5, 25),
                "dtype": "f32"}
    lo, hi = {"field": (8, 48), "run": (8, 40), "loop": (24, 128), "sweeps": (16, 96), "reverse": (12, 64),
              "mpi_step": (12, 96), "mpi_calls": (12, 56)}[kind]
    n = tuple(_size(rng, lo, hi) for _ in range(4))
    dtype = rng.choice(("f32", "f64"))
    if kind == "field":
        return _case(kind, n, dtype)
    if kind.startswith("mpi"):
        return _case(kind, n, "f64", 1, dt=0.01)
    if kind == "reverse":
        return _case(kind, n, dtype, rng.randint(3, 12), dt=0.1, every=rng.choice((0, 4, 8)))
    steps = {"run": rng.randint(4, 12), "loop": rng.randint(1, 3), "sweeps": 1}[kind]
    return _case(kind, n, dtype, steps, dt=rng.choice((0.05, 0.1, 0.125)), ic=rng.choice(("landau", "landau", "two_stream")))


# --------------------------------------------------------------- the inputs
def _box(case):
    if case["kind"].startswith("mpi"):
        return MPI_L, 9.0
    if case.get("ic") == "two_stream":
        return 10 * math.pi, 8.0
    return 4 * math.pi, 6.0


def _domain(case):
    L, vmax = _box(case)
    # The fields of the reverse mode are those of a plain Poisson solve (case
    # 110); the other runs solve for rho - 1, as the reference's decks do.
    idcase = 110 if case["kind"] == "reverse" else 10
    return pkg.Domain([case["nx"], case["ny"], case["nvx"], case["nvy"]], [0.0, 0.0, -vmax, -vmax], [L, L, vmax, vmax],
                      case.get("dt", 0.1), max(case["steps"], 1) + 1, idcase)


def _axis(lo, hi, n):
    return lo + torch.arange(n, dtype=torch.float64) * ((hi - lo) / n)


def _f0(case, seed):
    """A perturbed equilibrium on the grid, FP64 on the GPU: density
    perturbations of random amplitude and phase in the longest modes, times
    one Maxwellian or two counter-streaming ones."""
    g = torch.Generator().manual_seed(seed)
    rnd = lambda *s: torch.rand(*s, generator=g, dtype=torch.float64)  # noqa: E731
    L, vmax = _box(case)
    nx, ny = case["nx"], case["ny"]
    x, y = _axis(0.0, L, nx)[None, :], _axis(0.0, L, ny)[:, None]
    vx, vy = _axis(-vmax, vmax, case["nvx"])[None, :], _axis(-vmax, vmax, case["nvy"])[:, None]
    maxw = lambda w: torch.exp(-0.5 * w * w) / math.sqrt(TWO_PI)  # noqa: E731
    if case.get("ic") == "two_stream":
        M = 0.5 * (maxw(vx - 2.4) + maxw(vx + 2.4)) * maxw(vy)
        top = 0.002
    else:
        M = maxw(vx) * maxw(vy)
        top = 0.08
    k = TWO_PI / L
    if case["kind"] == "reverse":
        # An amplitude field eps(x, y) on 32 x 32 points, U[0.02, 0.08].
        eps = 0.02 + 0.06 * rnd(32, 32)
        eps = eps[(torch.arange(ny) * 32) // ny][:, (torch.arange(nx) * 32) // nx]
        A = 1 + eps * (torch.cos(k * x) + torch.cos(k * y))
    else:
        A = torch.ones(ny, nx, dtype=torch.float64)
        for jx, jy in ((1, 0), (0, 1), (1, 1), (2, 0)):
            A = A + top * (0.25 + 0.75 * rnd(1)) * torch.cos(k * (jx * x + jy * y) + TWO_PI * rnd(1)) / (jx + jy)
    return M.cuda()[:, :, None, None] * A.cuda()[None, None]


def _members(case, seed):
    import random

    shape, rng = random.Random(case["grids"]), random.Random(seed)
    out = []
    for _ in range(case["members"]):
        n = [shape.choice((16, 24, 32, 48)) for _ in range(4)]
        k = shape.choice((0.3, 0.5))
        L = TWO_PI / k
        out.append(v.EnsembleMember(n, [0.0, 0.0, -6.0, -6.0], [L, L, 6.0, 6.0], 0.1, rng.uniform(0.01, 0.1), k))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        ens = v.Ensemble(_members(case, seed), case["steps"])
        ens.set_tiles(256, 64, 2)  # the tiles the library's tuner picks on a B200
        return {"kind": kind, "ens": ens}
    ctx = v.Context(_domain(case), case["dtype"])
    st = {"kind": kind, "ctx": ctx, "steps": case["steps"], "dt": case.get("dt"), "f64": case["dtype"] == "f64"}
    if kind.startswith("mpi"):
        st["a"], st["b"], st["tmp"] = ctx.mpi_empty(), ctx.mpi_empty(), None
        if kind == "mpi_calls":
            st["tmp"] = ctx.mpi_empty()
        st["a"][3:-3, 3:-3, 3:-3, 3:-3] = _f0(case, seed)
    else:
        st["a"] = _f0(case, seed).to(ctx.torch_dtype).contiguous()
        if kind in ("run", "loop", "sweeps"):
            st["b"] = torch.empty_like(st["a"])
        if kind == "reverse":
            st["grad"] = torch.empty_like(st["a"])
            st["adj"] = v.Adjoint(ctx, case["steps"], case["every"])
    st["fields"] = (ctx.rho, ctx.ex, ctx.ey)
    for t in st["fields"]:
        t.owner = ctx  # views of the context's own memory: it lives as long as they do
    return st


# ------------------------------------------------------------------ one pass
def run(st):
    kind = st["kind"]
    if kind == "ensemble":
        ens = st["ens"]
        ens.run()
        got = [ens.read(i) for i in range(len(ens.members))]
        # The energies of an FP32 run carry FP32 rounding: kept as such.
        return [f for f, _ in got], np.stack([e for _, e in got]).astype(np.float32)
    ctx = st["ctx"]
    a = st["a"]
    if kind == "field":
        ctx.field_rho(a)
        ctx.field_poisson()
        ctx.diags_compute(0)
        return st["fields"]  # phi (which replaces rho), Ex, Ey
    if kind == "reverse":
        J = st["adj"].forward(a)
        return J, st["adj"].backward(st["grad"])
    b, dt = st["b"], st["dt"]
    if kind == "run":
        ctx.field_rho(a)
        ctx.field_poisson()
        ctx.diags_compute(0)
        ctx.steps(a, b, 1, st["steps"])
        st["a"], st["b"] = b, a
        nrj, _ = ctx.diags_read(st["steps"] + 1)  # the other history, the sum of the potential, is rounding about 0
        return b, nrj if st["f64"] else nrj.astype(np.float32)
    if kind == "loop":
        # The state goes on from call to call, as in a program that saves
        # every few steps.
        ctx.steps(a, b, 1, st["steps"])
        st["a"], st["b"] = b, a
    elif kind == "sweeps":
        ctx.advect_x(a, b, 0.5 * dt)
        ctx.advect_y(b, a, 0.5 * dt)
        ctx.field_rho(a)
        ctx.field_poisson()
        ctx.diags_compute(1)
        ctx.advect_vx(a, b, dt)
        ctx.advect_vy(b, a, dt)
        ctx.advect_x(a, b, 0.5 * dt)
        ctx.advect_y(b, a, 0.5 * dt)
        b = a
    elif kind == "mpi_step":
        ctx.mpi_step(a, b, 1)
        st["a"], st["b"] = b, a
        return (b[3:-3, 3:-3, 3:-3, 3:-3],) + st["fields"][1:]
    elif kind == "mpi_calls":
        tmp = st["tmp"]
        ctx.mpi_halo_fill(a)
        ctx.mpi_spline_xy(a)
        b.copy_(a)
        ctx.mpi_advect_2d(a, tmp, 0.5 * dt)
        ctx.mpi_field(a)
        ctx.diags_compute(1)
        ctx.mpi_spline_vxvy(b)
        ctx.mpi_advect_4d(b, tmp, dt)
        ctx.mpi_field(b)
        ctx.diags_compute(1)
        ctx.mpi_l2norm(b, 1)
        st["a"], st["b"] = b, a
        inner = (slice(3, -3),) * 4
        return (a[inner], b[inner]) + st["fields"][1:]  # the half-step f, the new f, Ex, Ey
    # The mid-step field belongs to an FP32 run's results only as f does.
    return (b,) + (st["fields"][1:] if st["f64"] else ())


def work(case):
    kind, s = case["kind"], case["steps"]
    e = 8 if case["dtype"] == "f64" else 4
    if kind == "ensemble":
        cells = sum(math.prod(m.n) for m in _members(case, 0))
        return {"bytes": cells * e * (4 * s + 2), "flops": cells * 75 * s}
    cells = case["nx"] * case["ny"] * case["nvx"] * case["nvy"]
    if kind == "field":
        return {"bytes": cells * e, "flops": cells}
    if kind in ("run", "loop"):
        # Every step: x/y and its moment, then v with the field of it.
        return {"bytes": cells * e * (4 * s + (kind == "run")), "flops": cells * 75 * s}
    if kind == "sweeps":
        return {"bytes": cells * e * 13, "flops": cells * 75}
    if kind == "reverse":
        # Forward 4 transfers a step; backward reads the state and the
        # adjoint for the field gradient and moves the adjoint twice.
        return {"bytes": cells * e * 10 * s, "flops": cells * 250 * s}
    # vlp4d_mpi: the density of the half step, then the 4^4 spline with four
    # prefilters and a predictor-corrector foot; call by call every call
    # reads and writes f.
    return {"bytes": cells * 8 * (4 if kind == "mpi_step" else 14), "flops": cells * 850}


# ------------------------------------------------- the same in 64-bit torch
def _weights6(x):
    """The reference's fifth-order basis (advection.hpp:38-50) on the points
    -2 .. 3 at x in [0, 1)."""
    a, b, c = x - 1, x + 1, x - 2
    return [-x * a * a * b * c / 24, x * a * c * (5 * x * x + x - 8) / 24, -a * c * b * (5 * x * x - 3 * x - 6) / 12,
            x * b * c * (5 * x * x - 7 * x - 4) / 12, -x * a * b * (5 * x * x - 11 * x - 2) / 24, x * x * a * b * c / 24]


def _shift(f, dim, disp, lo, hi):
    """f at (x - disp) along `dim`; disp is constant along it (size 1 there)."""
    n = f.shape[dim]
    q = -disp / ((hi - lo) / n)
    m = torch.floor(q).detach()
    w = _weights6(q - m)
    shape = [1] * f.dim()
    shape[dim] = n
    i = torch.arange(n, device=f.device).view(shape) + m.to(torch.int64) - 2
    out = None
    for k in range(6):
        t = w[k] * torch.gather(f, dim, ((i + k) % n).expand(f.shape))
        out = t if out is None else out + t
    return out


class _Exact:
    def __init__(self, n, lo, hi, dt, minus_one):
        nx, ny, nvx, nvy = n
        self.lo, self.hi, self.dt, self.minus_one = lo, hi, dt, minus_one
        self.h = [(hi[k] - lo[k]) / n[k] for k in range(4)]
        self.x, self.y, self.vx, self.vy = (_axis(lo[k], hi[k], n[k]).cuda() for k in range(4))
        ix = torch.arange(nx // 2 + 1, dtype=torch.float64).cuda()
        iy = torch.arange(ny, dtype=torch.float64).cuda()
        self.kx = (TWO_PI / hi[0] * ix)[None, :].expand(ny, -1)
        self.ky = (TWO_PI / hi[1] * torch.where(iy < ny // 2 + 1, iy, iy - ny))[:, None].expand(-1, nx // 2 + 1)
        k2 = self.kx ** 2 + self.ky ** 2
        self.inv = torch.where(k2 > 0, 1 / torch.where(k2 > 0, k2, torch.ones_like(k2)), torch.zeros_like(k2))

    def xshift(self, f, dt):
        return _shift(f, 3, dt * self.vx[None, :, None, None], self.lo[0], self.hi[0])

    def yshift(self, f, dt):
        return _shift(f, 2, dt * self.vy[:, None, None, None], self.lo[1], self.hi[1])

    def moment(self, f):
        return f.sum((0, 1)) * (self.h[2] * self.h[3])

    def field(self, rho):
        s = rho.shape
        r = torch.fft.rfft2(rho - self.minus_one) * self.inv / (s[0] * s[1])
        back = lambda z: torch.fft.irfft2(z, s=s, norm="forward")  # noqa: E731
        return back(r), back(-1j * self.kx * r), back(-1j * self.ky * r)

    def energy(self, ex, ey):
        return (ex * ex + ey * ey).sum() * self.h[0] * self.h[1]

    def half(self, f):
        return self.yshift(self.xshift(f, 0.5 * self.dt), 0.5 * self.dt)

    def vpart(self, f, ex, ey):
        f = _shift(f, 1, self.dt * ex[None, None], self.lo[2], self.hi[2])
        return _shift(f, 0, self.dt * ey[None, None], self.lo[3], self.hi[3])

    def step(self, f):
        f = self.half(f)
        rho = self.moment(f)
        phi, ex, ey = self.field(rho)
        f = self.half(self.vpart(f, ex, ey))
        return f, phi, ex, ey

    def log_energy(self, ex, ey):
        return float(torch.log(torch.sqrt(self.energy(ex, ey))))


def _exact_of(case, minus_one):
    d = _domain(case)
    return _Exact(d.nxmax, d.min_phy, d.max_phy, d.dt, minus_one)


def _spline_line(n):
    """The (n + 6) x n matrix that takes a periodic line to its cubic spline
    coefficients at -3 .. n + 2: the boundary sums of eight terms and the two
    first-order recursions of the prefilter."""
    s3 = math.sqrt(3.0)
    al = s3 - 2.0
    be = s3 * (1.0 - al * al)
    e = np.zeros((n + 6, n))
    eye = np.eye(n)
    for p in range(-2, n + 2):
        e[p + 3] = eye[p % n]
    for j in range(1, 9):
        e[0] += al ** j * eye[(-2 - j) % n]
        e[n + 5] += al ** j * eye[(n + 1 + j) % n]
    L = n + 4
    right = e[L + 1] + sum(al ** k * e[L - k] for k in range(L))
    t = [e[0] + e[1]]
    for k in range(1, L - 1):
        t.append(e[1 + k] + al * t[-1])
    c = s3 * right
    e[L] = c
    for i in range(L - 1, 0, -1):
        c = be * t[i - 1] + al * c
        e[i] = c
    return torch.from_numpy(e).cuda()


def _along(P, f, dim):
    return torch.movedim(torch.tensordot(P, f, dims=([1], [dim])), 0, dim)


def _bspline4(w):
    return [(1 - w) ** 3 / 6, (4 - 6 * w ** 2 + 3 * w ** 3) / 6, (1 + 3 * w + 3 * w ** 2 - 3 * w ** 3) / 6, w ** 3 / 6]


def _exact_mpi(case, f):
    E = _exact_of(case, 1.0)
    nvy, nvx, ny, nx = f.shape
    h, lo, hi, dt = E.h, E.lo, E.hi, E.dt
    C = _along(_spline_line(nx), f, 3)
    C = _along(_spline_line(ny), C, 2)  # (nvy, nvx, ny + 6, nx + 6)
    half = torch.empty_like(f)
    # The half step's x/y shift is constant over an (x, y) plane.
    fx, fy = -0.5 * dt * E.vx / h[0], -0.5 * dt * E.vy / h[1]
    mx, my = torch.floor(fx), torch.floor(fy)
    wx, wy = torch.stack(_bspline4(fx - mx)), torch.stack(_bspline4(fy - my))
    for j in range(nvy):
        acc = None
        for ky in range(4):
            y0 = int(my[j]) - 1 + ky + 3
            for kx in range(4):
                at = (torch.arange(nx, device="cuda")[None, :] + mx.to(torch.int64)[:, None] - 1 + kx + 3)
                row = torch.gather(C[j, :, y0:y0 + ny], 2, at[:, None, :].expand(nvx, ny, nx))
                t = wy[ky, j] * wx[kx][:, None, None] * row
                acc = t if acc is None else acc + t
        half[j] = acc
    _, ex, ey = E.field(E.moment(half))
    C = _along(_spline_line(nvx), C, 1)
    C = _along(_spline_line(nvy), C, 0).contiguous()
    st = (1, nx + 6, (nx + 6) * (ny + 6), (nx + 6) * (ny + 6) * (nvx + 6))
    flat = C.view(-1)
    out = torch.empty_like(f)
    gx, gy = torch.arange(nx, device="cuda", dtype=torch.float64), torch.arange(ny, device="cuda", dtype=torch.float64)
    lag3 = lambda p: (0.5 * (p - 1) * (p - 2), -p * (p - 2), 0.5 * p * (p - 1))  # noqa: E731
    for j in range(nvy):
        vx, vy = E.vx[:, None, None], E.vy[j]
        # Half-step predictor, the field there (3 x 3 Lagrange), full foot.
        px = (gx - 0.5 * dt / h[0] * vx).expand(nvx, ny, nx)
        py = (gy[:, None] - 0.5 * dt / h[1] * vy).expand(nvx, ny, nx)
        bx, by = torch.round(px) - 1, torch.round(py) - 1
        cx, cy = lag3(px - bx), lag3(py - by)
        ix, iy = bx.to(torch.int64), by.to(torch.int64)
        e1 = e2 = 0.0
        for ky in range(3):
            for kx in range(3):
                q = (ix + kx) % nx + nx * ((iy + ky) % ny)
                w = cx[kx] * cy[ky]
                e1 = e1 + w * ex.reshape(-1)[q]
                e2 = e2 + w * ey.reshape(-1)[q]
        foot = (gx - dt / h[0] * (vx - 0.5 * dt * e1), gy[:, None] - dt / h[1] * (vy - 0.5 * dt * e2),
                ((vx - dt * e1).clamp(lo[2], hi[2]) - lo[2]) / h[2], ((vy - dt * e2).clamp(lo[3], hi[3]) - lo[3]) / h[3])
        base, w = 0, []
        for d in range(4):
            m = torch.floor(foot[d])
            w.append(_bspline4(foot[d] - m))
            base = base + (m.to(torch.int64) + 2) * st[d]
        acc = 0.0
        for k3 in range(4):
            for k2 in range(4):
                s2 = 0.0
                for k1 in range(4):
                    s1 = 0.0
                    for k0 in range(4):
                        s1 = s1 + w[0][k0] * flat[base + (k0 + k1 * st[1] + k2 * st[2] + k3 * st[3])]
                    s2 = s2 + w[1][k1] * s1
                acc = acc + w[2][k2] * w[3][k3] * s2
        out[j] = acc
    _, ex, ey = E.field(E.moment(out))
    return half, out, ex, ey


def _exact_reverse(case, f0):
    from torch.utils.checkpoint import checkpoint

    E = _exact_of(case, 0.0)
    f0 = f0.clone().requires_grad_(True)
    f = f0
    for _ in range(case["steps"]):
        f = checkpoint(lambda g: E.step(g)[0], f, use_reentrant=False)
    _, ex, ey = E.field(E.moment(f))
    J = E.energy(ex, ey)
    (grad,) = torch.autograd.grad(J, f0)
    return float(J), grad


def exact(case, seed):
    kind, s = case["kind"], case["steps"]
    if kind == "ensemble":
        fs, hist = [], []
        for m in _members(case, seed):
            E = _Exact(m.n, m.min_phy, m.max_phy, m.dt, 0.0)
            maxw = lambda w: torch.exp(-0.5 * w * w) / math.sqrt(TWO_PI)  # noqa: E731
            A = 1 + m.amp * (torch.cos(m.k * E.x)[None, :] + torch.cos(m.k * E.y)[:, None])
            f = (maxw(E.vy)[:, None] * maxw(E.vx)[None, :])[:, :, None, None] * A
            _, ex, ey = E.field(E.moment(f))
            e = [E.log_energy(ex, ey)]
            for _ in range(s):
                f, _, ex, ey = E.step(f)
                e.append(E.log_energy(ex, ey))
            fs.append(f)
            hist.append(e)
        return fs, np.array(hist)
    dtype = torch.float64 if case["dtype"] == "f64" else torch.float32
    f = _f0(case, seed).to(dtype).to(torch.float64)
    if kind == "mpi_step":
        return _exact_mpi(case, f)[1:]
    if kind == "mpi_calls":
        return _exact_mpi(case, f)
    if kind == "reverse":
        return _exact_reverse(case, f)
    E = _exact_of(case, 1.0)
    if kind == "field":
        return E.field(E.moment(f))
    _, ex, ey = E.field(E.moment(f))
    nrj = [E.log_energy(ex, ey)]
    for _ in range(s):
        f, _, ex, ey = E.step(f)
        nrj.append(E.log_energy(ex, ey))
    if kind == "run":
        return f, np.array(nrj)
    return (f, ex, ey) if case["dtype"] == "f64" else (f,)
