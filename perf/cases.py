"""Performance cases of the time step and of the forms built on it.

Each case is a grid and a form, taken through the calls a program makes every time step:
``Context.step`` (FP64 path and FP32 form), ``Context.step_tracers``, ``Ensemble.step``,
``euler_steps`` with its backward pass, and the unfused ``compute_tendencies`` /
``apply_tendencies`` pair. ``exact`` evaluates the same scheme in plain torch, 64 bits,
written from the scheme's equations (cell-average reconstruction, WENO blending, ADER time
series, upwind characteristic flux) with tables derived here.
"""
import math

import numpy as np
import torch

from awflcloud_b200 import capi
from awflcloud_b200.adjoint import euler_steps

GRAV, CP, RD, P0 = 9.81, 1004.0, 287.0, 1.0e5
C0, GAMMA = 27.5629410929725921310572974482, 1.40027894002789400278940027894
THETA0 = 300.0
LEN = (20000.0, 20000.0, 10000.0)  # the domain of the benchmark, metres
NGLL = {5: 3, 9: 5}
R, U, V, W, T = range(5)
# operations of one cell and time step (three splits) of the scheme, by order
FLOPS_PER_CELL_STEP = {5: 7153, 9: 24191}


# ---------------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest grid in use: quick looks, regression runs, one member of an ensemble.
        # Every launch is short, so latency and launches count
        _case("fp64_step_32x32x16", nx=32, ny=32, nz=16),
        # a small production grid in the FP32 form
        _case("fp32_step_64x64x32", nx=64, ny=64, nz=32, fp32=True),
        # ragged sizes, closed box, a new CFL time step before every step
        _case("fp64_walls_97x61x45_cfl", nx=97, ny=61, nz=45, walls=True, adaptive=True),
        # the reference's 2-D mode: a density-current sized x-z slice
        _case("fp64_sim2d_400x1x200", nx=400, ny=1, nz=200),
        # the headline grid in both forms
        _case("fp32_step_256x256x128", nx=256, ny=256, nz=128, fp32=True),
        _case("fp64_step_256x256x128", nx=256, ny=256, nz=128),
        # ninth order, both forms
        _case("fp32_ord9_128x128x64", nx=128, ny=128, nz=64, fp32=True, ord=9),
        _case("fp64_ord9_80x50x48", nx=80, ny=50, nz=48, ord=9),
        # the step with the driver's three tracers
        _case("fp64_tracers_128x128x64", kind="tracers", nx=128, ny=128, nz=64, ntr=3),
        # a gradient: four steps forward with checkpoints, then the adjoint of each segment
        _case("fp64_adjoint_64x64x32", kind="adjoint", nx=64, ny=64, nz=32, steps=4, every=2),
        # many small grids advanced together
        _case("fp32_ensemble_24", kind="ensemble", fp32=True, members=24, lo=32, hi=96, pick=7, steps=2),
        # the documented operator interface: tendencies, then the caller's own apply
        _case("fp64_tendencies_130x100x70", kind="tendencies", nx=130, ny=100, nz=70),
    ]


def _case(name=None, kind="step", **kw):
    c = dict(kind=kind, fp32=False, ord=5, walls=False)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid(most, ord_=5):
        while True:
            g = (size(12, 320), size(12, 320), size(10, 160))
            if 3000 <= g[0] * g[1] * g[2] <= most:
                return dict(nx=g[0], ny=g[1], nz=g[2], ord=ord_, walls=rng.random() < 0.3)

    kind = rng.choice(["step"] * 6 + ["sim2d", "ord9", "tracers", "adjoint", "ensemble", "tendencies"])
    fp32 = rng.random() < 0.5
    if kind == "step":
        return _case(fp32=fp32, adaptive=rng.random() < 0.2, **grid(8 << 20))
    if kind == "sim2d":
        return _case(fp32=fp32, nx=size(64, 1000), ny=1, nz=size(32, 500), walls=rng.random() < 0.3)
    if kind == "ord9":
        return _case(fp32=fp32, **grid(1 << 20, 9))
    if kind == "tracers":
        return _case(kind="tracers", fp32=fp32, ntr=rng.randint(1, 4), **grid(1 << 20))
    if kind == "adjoint":
        steps = rng.randint(2, 6)
        return _case(kind="adjoint", steps=steps, every=rng.randint(1, steps), **grid(1 << 18))
    if kind == "ensemble":
        return _case(kind="ensemble", fp32=fp32, members=rng.randint(4, 24), lo=16, hi=rng.randint(40, 96),
                     pick=rng.randint(0, 1 << 20), steps=rng.randint(1, 4))
    return _case(kind="tendencies", **grid(2 << 20))  # the parity path's interface


def _members(case):
    rng = np.random.default_rng(case["pick"])
    lo, hi = case["lo"], case["hi"]
    return [(int(rng.integers(lo, hi + 1)), int(rng.integers(lo, hi + 1)), int(rng.integers(lo // 2, hi // 2 + 1)))
            for _ in range(case["members"])]


def _bc(case):
    return ("wall",) * 3 if case["walls"] else ("periodic", "periodic", "wall")


def _cfl(case):
    return 0.4 if case["ord"] == 9 else 0.7


def _dt(case, n):
    return _cfl(case) * min(LEN[d] / n[d] for d in range(3)) / 370.0


def _grid(case):
    return case["nx"], case["ny"], case["nz"]


def work(case):
    o = case["ord"]
    grids = _members(case) if case["kind"] == "ensemble" else [_grid(case)]
    cells = sum(a * b * c for a, b, c in grids)
    # FP64: five values read and written; FP32: five values and their compensations
    step_b, step_f = 80 * cells, FLOPS_PER_CELL_STEP[o] * cells
    if case["kind"] == "tracers":
        return {"bytes": step_b + 16 * case["ntr"] * cells, "flops": step_f * (1 + 0.3 * case["ntr"])}
    if case["kind"] == "adjoint":  # the forward steps, their recomputation, the reverse sweep
        return {"bytes": 3 * step_b, "flops": 4 * step_f * case["steps"]}
    if case["kind"] == "ensemble":
        return {"bytes": step_b, "flops": step_f * case["steps"]}
    if case["kind"] == "tendencies":
        return {"bytes": step_b + 40 * cells, "flops": step_f}
    return {"bytes": step_b, "flops": step_f}


# ---------------------------------------------------------------------------- inputs
def _gen(seed, salt, device):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed) * 1000003 + salt)
    return g


def initial(n, o, seed, device):
    """A warm bubble with theta noise in a smooth wind, as perturbations (5, nz, ny, nx)."""
    nx, ny, nz = n
    rs = np.random.default_rng([int(seed) & 0x7FFFFFFF, nx, ny, nz])
    f8 = dict(dtype=torch.float64, device=device)
    x = ((torch.arange(nx, **f8) + 0.5) / nx)[None, None, :]
    y = ((torch.arange(ny, **f8) + 0.5) / ny)[None, :, None]
    z = ((torch.arange(nz, **f8) + 0.5) / nz)[:, None, None]
    bg = Background(n, o, device)
    rho = bg.dens_c[bg.hs:bg.hs + nz][:, None, None]
    cx, cy, cz = rs.uniform(0.35, 0.65), rs.uniform(0.35, 0.65), rs.uniform(0.2, 0.4)
    amp, rad = rs.uniform(1.0, 3.0), rs.uniform(0.12, 0.2)
    d2 = ((x - cx) ** 2 + ((z - cz) * 0.5) ** 2) / rad ** 2
    if ny > 1:
        d2 = d2 + ((y - cy) / rad) ** 2
    d = torch.sqrt(d2)
    th = amp * torch.where(d < 1, 0.5 * (1 + torch.cos(math.pi * d)), torch.zeros_like(d)).expand(nz, ny, nx)
    th = th + 0.05 * (2 * torch.rand(nz, ny, nx, generator=_gen(seed, 1, device), **f8) - 1)
    q = torch.zeros(5, nz, ny, nx, **f8)
    ph = rs.uniform(0, 2 * math.pi, 9)
    a = rs.uniform(0.5, 1.5, 5)
    wind = lambda s, p: 1 + 0.3 * torch.sin(2 * math.pi * x + p) * torch.cos(math.pi * z) + 0 * s  # noqa: E731
    q[R] = 1e-4 * rho * torch.sin(2 * math.pi * x + ph[0]) * torch.cos(2 * math.pi * y + ph[1]) * torch.cos(math.pi * z)
    q[U] = rho * 5 * a[0] * wind(y, ph[2])
    if ny > 1:
        q[V] = rho * 4 * a[1] * (torch.sin(2 * math.pi * y + ph[3]) + 0.2 * torch.cos(2 * math.pi * x + ph[4]))
    q[W] = rho * 1.5 * a[2] * torch.sin(math.pi * z) * torch.sin(2 * math.pi * x + ph[5])
    q[T] = rho * th
    return q


def initial_tracers(q, n, o, ntr):
    """rho times the driver's kinds of tracer: uniform, a smooth cone, a block, a wave."""
    nx, ny, nz = n
    bg = Background(n, o, q.device)
    rho = bg.dens_c[bg.hs:bg.hs + nz][:, None, None] + q[R]
    f8 = dict(dtype=torch.float64, device=q.device)
    x = ((torch.arange(nx, **f8) + 0.5) / nx)[None, None, :].expand(nz, ny, nx)
    z = ((torch.arange(nz, **f8) + 0.5) / nz)[:, None, None].expand(nz, ny, nx)
    cone = 2 * torch.clamp(1 - torch.sqrt(((x - 0.5) / 0.2) ** 2 + ((z - 0.4) / 0.3) ** 2), min=0)
    block = ((x > 0.4) & (x < 0.6) & (z > 0.1) & (z < 0.3)).double()
    fields = [torch.ones_like(x), cone, block, 1 + 0.5 * torch.sin(2 * math.pi * x) * torch.sin(math.pi * z)]
    return torch.stack([rho * fields[t % 4] for t in range(ntr)])


def _padded(q, hs):
    """`q` (v, nz, ny, nx) inside a zero halo."""
    out = torch.zeros(q.shape[0], *(s + 2 * hs for s in q.shape[1:]), dtype=q.dtype, device=q.device)
    out[:, hs:-hs, hs:-hs, hs:-hs] = q
    return out


def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _context(case, n):
    return capi.Context(*n, bc=_bc(case), ord_=case["ord"], precision=capi.FP32 if case["fp32"] else capi.FP64,
                        device=_device().index)


def _fill(ctx, q):
    st = ctx.new_state()
    st[:5] = _padded(q, ctx.hs).to(st.dtype)
    return st


def prepare(case, seed):
    dev, o = _device(), case["ord"]
    if case["kind"] == "ensemble":
        grids = _members(case)
        ens = capi.Ensemble([dict(nx=a, ny=b, nz=c, bc=_bc(case), ord_=o,
                                  precision=capi.FP32 if case["fp32"] else capi.FP64) for a, b, c in grids], dev.index)
        states = []
        for i, n in enumerate(grids):
            states.append(_fill(ens.members[i], initial(n, o, seed + 97 * i, dev)))
            ens.bind(i, states[-1], _dt(case, n))
        return dict(case=case, ens=ens, states=states)
    n = _grid(case)
    q = initial(n, o, seed, dev)
    ctx = _context(case, n)
    s = dict(case=case, ctx=ctx, state=_fill(ctx, q), dt=_dt(case, n))
    if case["kind"] == "tracers":
        s["tracers"] = _padded(initial_tracers(q, n, o, case["ntr"]), ctx.hs)
    if case["kind"] == "tendencies":
        s["tend"] = ctx.new_tend()
    if case["kind"] == "adjoint":
        s["target"] = s["state"].clone()
        s["state"].requires_grad_(True)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "ensemble":
        s["ens"].step(case["steps"])
        return [st[:5] for st in s["states"]]
    ctx, st = s["ctx"], s["state"]
    if kind == "step":
        if case.get("adaptive"):
            dt = ctx.cfl(st, _cfl(case))
            ctx.step(st, dt)
            return [st[:5], dt]
        ctx.step(st, s["dt"])
        return st[:5]  # the five variables (an FP32 state's second half is their rounding remainder)
    if kind == "tracers":
        ctx.step_tracers(st, s["tracers"], s["dt"])
        return [st[:5], s["tracers"]]
    if kind == "tendencies":
        for d in range(3):
            ctx.compute_tendencies(st, s["tend"], s["dt"], d)
            ctx.apply_tendencies(st, s["tend"], s["dt"])
        return [st[:5], s["tend"]]
    # adjoint: gradient of a misfit with respect to the initial state
    st.grad = None
    ctx.dimswitch = 1
    out = euler_steps(st, ctx, case["steps"], s["dt"], ckpt_every=case["every"])
    out.backward(out.detach() - s["target"])
    return [out.detach(), st.grad]


# ------------------------------------------------------------- the scheme in plain torch
def _lobatto(n):
    """Gauss-Lobatto-Legendre points in [-1/2, 1/2] and weights that sum to one."""
    p = np.polynomial.legendre.Legendre.basis(n - 1)
    x = np.concatenate([[-1.0], np.sort(p.deriv().roots().real), [1.0]])
    for _ in range(3):  # Newton on the inner points
        x[1:-1] -= p.deriv()(x[1:-1]) / p.deriv(2)(x[1:-1])
    return x / 2, 1.0 / (n * (n - 1) * p(x) ** 2)


def _theta_density(z):
    exner = 1.0 - GRAV * z / (CP * THETA0)
    return (exner ** (CP / RD) * P0 / C0) ** (1.0 / GAMMA) / THETA0


class Background:
    """The constant-theta hydrostatic columns: cell averages with halos, and GLL values."""

    def __init__(self, n, o, device):
        self.hs, g = (o - 1) // 2, NGLL[o]
        nz, dz = n[2], LEN[2] / n[2]
        x, w = _lobatto(o)
        zc = (np.arange(-self.hs, nz + self.hs)[:, None] + 0.5 + x[None, :]) * dz
        zg = (np.arange(nz)[:, None] + 0.5 + _lobatto(g)[0][None, :]) * dz
        f8 = dict(dtype=torch.float64, device=device)
        self.dens_c = torch.tensor(_theta_density(zc) @ w, **f8)
        self.dt_c = self.dens_c * THETA0
        self.dens_g = torch.tensor(_theta_density(zg), **f8)
        self.dt_g = self.dens_g * THETA0
        self.pres_g = C0 * self.dt_g ** GAMMA


class Tables:
    def __init__(self, o, device):
        hs, g = (o - 1) // 2, NGLL[o]
        f8 = dict(dtype=torch.float64, device=device)

        def coefs(first, m):  # averages of m cells, the first at `first` cells from the centre -> polynomial
            c = np.arange(first, first + m, dtype=np.float64)[:, None]
            p = np.arange(m)[None, :]
            return np.linalg.inv(((c + 0.5) ** (p + 1) - (c - 0.5) ** (p + 1)) / (p + 1))

        low = np.zeros((hs + 1, o, o))
        for i in range(hs + 1):
            low[i, :hs + 1, i:i + hs + 1] = coefs(i - hs, hs + 1)
        high = coefs(-hs, o)
        if o == 5:
            sigma, idl = 0.73564225445964, np.array([1.0, 73.564225445964, 1.0, 1584.89319246111])
        else:
            sigma = 0.0288539981181442
            idl = np.array([1.0, 2.15766927997459, 2.40224886796286, 2.15766927997459, 1.0, 1136.12697719888])
        idl = idl / idl.sum()

        def smooth(m):  # sum over derivatives of the integral of the square, its integrand cut to m terms
            q = np.zeros((m, m))
            for k in range(1, m):
                f = [math.factorial(j) / math.factorial(j - k) if j >= k else 0.0 for j in range(m)]
                for a in range(k, m):
                    for b in range(k, m):
                        d = a + b - 2 * k
                        if d <= m - 1 and d % 2 == 0:
                            q[a, b] += f[a] * f[b] * 0.5 ** d / (d + 1)
            return q

        x, w = _lobatto(g)
        vander = x[:, None] ** np.arange(o)[None, :]
        small = x[:, None] ** np.arange(g)[None, :]
        dsmall = np.arange(g)[None, :] * x[:, None] ** np.maximum(np.arange(g) - 1, 0)[None, :]
        t = lambda a: torch.tensor(a, **f8)  # noqa: E731
        # the bridge polynomial: the full one less the ideal-weighted low ones
        self.cand = t(np.concatenate([low, ((high - np.tensordot(idl[:-1], low, 1)) / idl[-1])[None]]))
        self.tv_low, self.tv_high = t(smooth(hs + 1)), t(smooth(o))
        self.idl, self.sigma, self.hs, self.ng, self.o = [float(v) for v in idl], sigma, hs, g, o
        self.c2g, self.deriv, self.wts = t(vander), t(dsmall @ np.linalg.inv(small)), t(w)

    def points(self, u):
        """GLL values of every cell from the padded line values u (..., L + 2 hs)."""
        hs, idl = self.hs, self.idl
        a = torch.einsum("kps,...s->k...p", self.cand, u.unfold(-1, self.o, 1))
        tv = []
        for k in range(hs + 2):
            m = self.tv_high if k == hs + 1 else self.tv_low
            b = a[k][..., :m.shape[0]]
            tv.append(((b @ m) * b).sum(-1))
        avg = sum(tv[:-1]) / (hs + 1)
        tv[-1] = avg + (tv[-1] - avg) * self.sigma

        def unit(w):
            s = sum(w) + 1e-20
            return [v / s for v in w]

        w = unit([d / (v * v + 1e-20) for d, v in zip(idl, tv)])
        w = unit([v * (d + d * d - 3 * d * v + v * v) / (d * d + v * (1 - 2 * d)) for d, v in zip(idl, w)])
        return sum(v[..., None] * c for v, c in zip(w, a)) @ self.c2g.T


class Scheme:
    def __init__(self, case, n, device):
        self.n, self.o, self.walls = n, case["ord"], _bc(case)
        self.tab, self.bg = Tables(self.o, device), Background(n, self.o, device)
        self.hs = self.tab.hs

    def pad(self, u, d, normal=None):
        """Lines (v, a, b, L) with their halos: a periodic copy, or the edge cell (no normal momentum)."""
        h, wall = self.hs, self.walls[d] == "wall"
        if not wall:
            return torch.cat([u[..., -h:], u, u[..., :h]], -1)
        lo, hi = u[..., :1].expand(*u.shape[:-1], h), u[..., -1:].expand(*u.shape[:-1], h)
        if normal is not None:
            keep = torch.ones(u.shape[0], 1, 1, 1, dtype=u.dtype, device=u.device)
            keep[normal] = 0
            lo, hi = lo * keep, hi * keep
        return torch.cat([lo, u, hi], -1)

    def sides(self, left, right, d):
        """States on both sides of the L + 1 faces from the cells' left and right edge values."""
        if self.walls[d] == "wall":
            return torch.cat([left[..., :1], right], -1), torch.cat([left, right[..., -1:]], -1)
        return torch.cat([right[..., -1:], right], -1), torch.cat([left, left[..., :1]], -1)

    def tendency(self, p, d, dt, a0, tr=None):
        """Time-averaged tendency of the padded lines p (5, a, b, L + 2 hs), whose first index
        along a is a0; with tr, padded tracer / density lines, the tracers' tendency too."""
        tab, bg, hs, g = self.tab, self.bg, self.hs, self.tab.ng
        length, nm, na = p.shape[-1] - 2 * hs, 1 + d, self.tab.ng
        dx = LEN[d] / self.n[d]
        wall_z = d == 2 and self.walls[2] == "wall"
        if d == 2:
            rb, tb, pb = bg.dens_g, bg.dt_g, bg.pres_g
        else:
            rows = slice(hs + a0, hs + a0 + p.shape[1])
            rb, tb, pb = bg.dens_c[rows][:, None, None, None], bg.dt_c[rows][:, None, None, None], 0.0
        inner = torch.ones(length, g, dtype=p.dtype, device=p.device)
        if wall_z:
            inner[0, 0] = inner[-1, -1] = 0
        q = [tab.points(p[v]) for v in range(5)]
        gravity = None
        if d == 2:
            gravity = [(-q[R][..., -1:] * GRAV).expand(q[R].shape)]  # the last point's value at every point
            q[W] = q[W] * inner
        q[R], q[T] = q[R] + rb, q[T] + tb
        q = [q]
        f = [[q[0][nm] * q[0][m] / q[0][R] for m in range(1, 5)]]
        gm = [q[0][T] ** GAMMA]
        for k in range(na - 1):
            flux = [q[k][nm]] + list(f[k])
            flux[nm] = flux[nm] + (C0 * gm[0] - pb if k == 0 else 0.5 * C0 * gm[k])
            new = [-(v @ tab.deriv.T) / dx / (k + 1) for v in flux]
            if d == 2:
                new[W] = (new[W] + gravity[k] / (k + 1)) * inner
                gravity.append(-new[R] * GRAV)
            q.append(new)
            fk = []
            for x in range(4):
                s = sum(q[i][nm] * q[k + 1 - i][x + 1] for i in range(k + 2))
                s = s - sum(q[i][R] * f[k + 1 - i][x] for i in range(1, k + 2))
                fk.append(s / q[0][R])
            f.append(fk)
            s = sum((k + 1 - i) * GAMMA * gm[i] * q[k + 1 - i][T] for i in range(k + 1))
            s = s - sum((k + 1 - i) * q[i][T] * gm[k + 1 - i] for i in range(1, k + 1))
            gm.append((GAMMA * gm[0] * q[k + 1][T] + s / (k + 1)) / q[0][T])

        def edges(series):
            m = [sum(v[..., e] * dt ** k / (k + 1) for k, v in enumerate(series)) for e in (0, -1)]
            return m

        e = [edges([q[k][v] for k in range(na)]) for v in range(5)]
        left, right = torch.stack([v[0] for v in e]), torch.stack([v[1] for v in e])
        ql, qr = self.sides(left, right, d)
        r = 0.5 * (ql[R] + qr[R])
        if d == 1:  # the y averages are not divided by the density
            vel, t = 0.5 * (ql[1:4] + qr[1:4]), 0.5 * (ql[T] + qr[T])
        else:
            vel, t = 0.5 * (ql[1:4] / ql[R] + qr[1:4] / qr[R]), 0.5 * (ql[T] / ql[R] + qr[T] / qr[R])
        cs = torch.sqrt(GAMMA * C0 * (r * t) ** GAMMA / r)
        vn = vel[d]
        up = torch.where(vn > 0, ql, qr)
        w5 = (vn * qr[R] - qr[nm]) / (2 * cs) + qr[T] / (2 * t)
        w6 = (ql[nm] - vn * ql[R]) / (2 * cs) + ql[T] / (2 * t)
        s = [None] * 5
        w1 = up[R] - up[T] / t
        s[R] = w1 + w5 + w6
        s[T] = t * (w5 + w6)
        for m in (U, V, W):
            if m == nm:
                s[m] = vn * w1 + (vn - cs) * w5 + (vn + cs) * w6
            else:
                s[m] = up[m] - vel[m - 1] * up[T] / t + vel[m - 1] * (w5 + w6)
        flux = [s[nm]] + [s[nm] * s[m] / s[R] for m in range(1, 5)]
        flux[nm] = flux[nm] + C0 * s[T] ** GAMMA
        if d == 2:
            flux[nm] = flux[nm] - torch.cat([bg.pres_g[:, 0], bg.pres_g[-1:, -1]])
        flux = torch.stack(flux)
        tend = -(flux[..., 1:] - flux[..., :-1]) / dx
        if d == 2:
            avg = sum(v * dt ** k / (k + 1) for k, v in enumerate(gravity))
            tend = torch.stack([tend[v] + (avg @ tab.wts if v == W else 0) for v in range(5)])
        if self.n[1] == 1:
            tend = torch.stack([tend[v] * (v != V) for v in range(5)])
        if tr is None:
            return tend, None
        ttend = []
        un = 0.5 * (ql[nm] + qr[nm])
        for c in tr:
            rt = [torch.clamp(tab.points(c) * q[0][R], min=0)]
            ru = [rt[0] * q[0][nm] / q[0][R]]
            for k in range(na - 1):
                rt.append(-(ru[k] @ tab.deriv.T) / dx / (k + 1))
                s = sum(q[i][nm] * rt[k + 1 - i] for i in range(k + 2))
                s = s - sum(q[i][R] * ru[k + 1 - i] for i in range(1, k + 2))
                ru.append(s / q[0][R])
            tl, tR = (torch.clamp(v, min=0) for v in edges(rt))
            tl, tR = self.sides(tl, tR, d)
            tf = flux[R] * torch.where(vn > 0, tl / ql[R], tR / qr[R])
            ttend.append(self.limited(tf, un, c[..., hs:hs + length], p[R][..., hs:hs + length], d, dt, a0, dx))
        return tend, torch.stack(ttend)

    def limited(self, tf, un, mix, rho, d, dt, a0, dx):
        """Positivity limiter, face after face along the line, then the divergence."""
        hs, length = self.hs, mix.shape[-1]
        if d == 2:
            dens = rho + self.bg.dens_c[hs:hs + length]
        else:
            dens = rho + self.bg.dens_c[hs + a0:hs + a0 + rho.shape[0]][:, None, None]
        mass = mix * dens
        tf = list(tf.unbind(-1))
        for k in range(length + 1):
            lo, hi = (k - 1) % length, k % length
            v = un[..., k]

            def factor(cell):
                out = dt * (torch.clamp(tf[cell + 1], min=0) - torch.clamp(tf[cell], max=0)) / dx
                return torch.clamp(mass[..., cell] / (out + 1e-10), max=1)

            tf[k] = tf[k] * torch.where(v > 0, factor(lo), torch.where(v < 0, factor(hi), torch.ones_like(v)))
        tf = torch.stack(tf, -1)
        return -(tf[..., 1:] - tf[..., :-1]) / dx

    def split(self, q, d, dt, tracers=None):
        """One split of the interior fields q (5, nz, ny, nx): the new fields, the tendency, the
        halo values along d, and the same for the tracers."""
        ax = 3 - d
        u = q.movedim(ax, -1)
        p = self.pad(u, d, 1 + d)
        t = None
        if tracers is not None:
            rho = q[R] + self.bg.dens_c[self.hs:self.hs + self.n[2]][:, None, None]
            t = self.pad((tracers / rho).movedim(ax, -1), d)
        rows = max(1, int((1 << 19) / (p.shape[2] * p.shape[3])))
        parts = [self.tendency(p[:, a:a + rows], d, dt, a, None if t is None else t[:, a:a + rows])
                 for a in range(0, p.shape[1], rows)]
        tend = torch.cat([x[0] for x in parts], 1).movedim(-1, ax)
        p = p.movedim(-1, ax)
        if tracers is None:
            return q + dt * tend, tend, p, None, None
        ttend = torch.cat([x[1] for x in parts], 1).movedim(-1, ax)
        return q + dt * tend, tend, p, tracers + dt * ttend, t.movedim(-1, ax)

    def halo(self, full, p, d):
        """Writes the halo values of the padded lines p into the state array, as a split does."""
        h, ax = self.hs, 3 - d
        lines = full[tuple([slice(None)] + [slice(None) if a == ax else slice(h, -h) for a in (1, 2, 3)])]
        for s in (slice(0, h), slice(-h, None)):
            at = tuple(s if a == ax else slice(None) for a in range(4))
            lines[at] = p[at]

    def step(self, full, dt, forward=True, tracers=None):
        """A time step of the state array (5, nz + 2 hs, ...) in place; returns the last tendency."""
        h, tend = self.hs, None
        box = (slice(None),) + (slice(h, -h),) * 3
        for d in ((0, 1, 2) if forward else (2, 1, 0)):
            if d == 1 and self.n[1] == 1:
                continue
            new, tend, p, tnew, tp = self.split(full[box].clone(), d, dt, None if tracers is None else tracers[box].clone())
            full[box] = new
            self.halo(full, p, d)
            if tracers is not None:
                tracers[box] = tnew
                self.halo(tracers, tp, d)
        return tend

    def cfl(self, full, cfl):
        h, nz = self.hs, self.n[2]
        q = full[:, h:-h, h:-h, h:-h]
        r = q[R] + self.bg.dens_c[h:h + nz][:, None, None]
        t = q[T] + self.bg.dt_c[h:h + nz][:, None, None]
        cs = torch.sqrt(GAMMA * C0 * t ** GAMMA / r)
        return min(float((cfl * (LEN[d] / self.n[d]) / ((q[1 + d] / r).abs() + cs)).min()) for d in range(3))


def _exact_state(case, q):
    hs = (case["ord"] - 1) // 2
    return _padded(q.float().double() if case["fp32"] else q, hs)


def exact(case, seed):
    dev, o, kind = _device(), case["ord"], case["kind"]
    if kind == "ensemble":
        out = []
        for i, n in enumerate(_members(case)):
            full, sch = _exact_state(case, initial(n, o, seed + 97 * i, dev)), Scheme(case, n, dev)
            for k in range(case["steps"]):
                sch.step(full, _dt(case, n), k % 2 == 0)
            out.append(full)
        return out
    n = _grid(case)
    sch, dt = Scheme(case, n, dev), _dt(case, n)
    q = initial(n, o, seed, dev)
    full = _exact_state(case, q)
    if kind == "step":
        if case.get("adaptive"):
            dt = sch.cfl(full, _cfl(case))
            sch.step(full, dt)
            return [full, dt]
        sch.step(full, dt)
        return full
    if kind == "tracers":
        tracers = _padded(initial_tracers(q, n, o, case["ntr"]), sch.hs)
        sch.step(full, dt, tracers=tracers)
        return [full, tracers]
    if kind == "tendencies":
        tend = sch.step(full, dt)
        return [full, tend]
    return _exact_adjoint(case, sch, full, dt)


def _exact_adjoint(case, sch, full, dt):
    from torch.utils.checkpoint import checkpoint
    h = sch.hs
    box = (slice(None),) + (slice(h, -h),) * 3
    start = full[box].clone().requires_grad_(True)
    q, out = start, full.clone()
    for k in range(case["steps"]):
        for d in ((0, 1, 2) if k % 2 == 0 else (2, 1, 0)):
            if d == 1 and sch.n[1] == 1:
                continue
            with torch.no_grad():
                sch.halo(out, sch.split(q.detach(), d, dt)[2], d)
            q = checkpoint(lambda x, d=d: sch.split(x, d, dt)[0], q, use_reentrant=False)
    q.backward(q.detach() - start.detach())
    out[box] = q.detach()
    return [out, _padded(start.grad, h)]
