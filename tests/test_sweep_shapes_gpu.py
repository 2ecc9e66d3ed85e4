"""The sweep's tile shapes (awfl_sweep.cuh): grids whose lines take each shape of the launch
rule, and the ends of a line in each -- full and ragged last chunks, a line of exactly one
chunk, lines shorter than a chunk, periodic and wall ends, one line per plane.

FP64 equals the CPU oracle bit for bit (states with halos, tendencies, tracers). FP32 is held
to the FP64 path: the form's bar is 1e-5 relative L2 of every variable after 100 steps; two
steps must meet it too, and a flux or an update that went to the wrong cell misses it by
orders of magnitude."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from awflcloud_b200 import capi  # noqa: E402
from oracle.pyoracle import Oracle  # noqa: E402

PPW, PPP, WWW = (0, 0, 1), (0, 0, 0), (1, 1, 1)
GRIDS = [((32, 32, 16), PPW), ((32, 16, 32), PPP), ((33, 31, 15), PPP), ((7, 64, 129), WWW), ((130, 5, 9), PPW),
         ((128, 1, 37), PPW), ((400, 1, 12), PPP), ((3, 128, 8), PPP), ((65, 48, 2), PPW), ((16, 8, 130), PPP)]
FP64_ONLY = [((150, 140, 9), PPW), ((9, 150, 140), PPP)]  # many tiles: the large grids' shapes, ragged


def _state(n, hs, seed):
    nx, ny, nz = n
    r = np.random.default_rng(seed)
    st = np.zeros((5, nz + 2 * hs, ny + 2 * hs, nx + 2 * hs))
    box = st[:, hs:hs + nz, hs:hs + ny, hs:hs + nx]
    scale = np.array([1e-3, 3.0, 2.0, 1.0, 0.3]).reshape(5, 1, 1, 1)
    x = np.arange(nx) / nx * 2 * np.pi
    box[:] = scale * (0.2 * r.standard_normal(box.shape) + np.sin(x + r.uniform(0, 6)))
    if ny == 1:
        box[2] = 0.0
    return st


def _bits(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.int64), np.ascontiguousarray(b).view(np.int64))


def _ctx(n, bc, **kw):
    return capi.Context(*n, bc=tuple("wall" if b else "periodic" for b in bc), **kw)


@pytest.mark.parametrize("n,bc", GRIDS + FP64_ONLY)
def test_fp64_shapes_equal_oracle(n, bc):
    c, o = _ctx(n, bc), Oracle(*n, bc=bc, crpow=True)
    st = _state(n, c.hs, 1)
    d = torch.from_numpy(st).cuda()
    dt = o.compute_dt(st, 0.5)
    tend = c.new_tend()
    for s in range(3):  # a step's splits through the unfused interface
        c.compute_tendencies(d, tend, dt, s)
        want = np.zeros(c.tend_shape)
        o.compute_tendencies_dir(st, want, dt, s) if not (s == 1 and n[1] == 1) else None
        assert _bits(tend.cpu().numpy(), want), s
        assert _bits(d.cpu().numpy(), st), s
        c.apply_tendencies(d, tend, dt)
        o.apply(st, want, dt)
    for _ in range(2):
        c.step(d, dt)
        o.time_step(st, dt)
        assert _bits(d.cpu().numpy(), st)


@pytest.mark.parametrize("n,bc", [g for g in GRIDS if min(g[0]) > 1][:6])
def test_fp64_tracer_shapes_equal_oracle(n, bc):
    c, o = _ctx(n, bc), Oracle(*n, bc=bc, crpow=True)
    st = _state(n, c.hs, 2)
    r = np.random.default_rng(3)
    tr = np.zeros(c.tracer_shape(2))
    h = c.hs
    tr[:, h:-h, h:-h, h:-h] = np.maximum(0, r.standard_normal((2, n[2], n[1], n[0])))
    d, t = torch.from_numpy(st).cuda(), torch.from_numpy(tr).cuda()
    dt = o.compute_dt(st, 0.5)
    for _ in range(2):
        c.step_tracers(d, t, dt, pos=[1, 0])
        o.time_step_tracers(st, tr, dt, [1, 0])
    assert _bits(d.cpu().numpy(), st)
    assert _bits(t.cpu().numpy(), tr)


@pytest.mark.parametrize("n,bc", GRIDS + [((129, 60, 50), PPW), ((128, 60, 50), WWW)])
def test_fp32_shapes_match_fp64(n, bc):
    c64, c32 = _ctx(n, bc), _ctx(n, bc, precision=capi.FP32)
    st = _state(n, c64.hs, 4)
    d32 = c32.new_state()
    d32[:5] = torch.from_numpy(st).cuda().float()
    d64 = d32[:5].double()
    dt = c64.cfl(d64, 0.5)
    for _ in range(2):
        c64.step(d64, dt)
        c32.step(d32, dt)
    h = c64.hs
    for v in range(5):
        a, b = (x[v, h:-h, h:-h, h:-h].double() for x in (d32, d64))
        norm = float(b.norm())
        assert float((a - b).norm()) <= 1e-5 * norm if norm else float(a.norm()) == 0, v


# ord 9: 32 x 4, 16 x 8, 8 x 16 and 128 x 1 in every direction, full and ragged
GRIDS9 = [((32, 32, 16), PPW), ((33, 31, 15), PPP), ((7, 64, 129), WWW), ((130, 5, 9), PPW), ((400, 1, 12), PPP),
          ((16, 8, 130), PPP), ((64, 64, 32), PPW), ((20, 200, 9), WWW), ((65, 48, 5), PPW)]


@pytest.mark.parametrize("n,bc", GRIDS9)
def test_fp64_ord9_shapes_equal_oracle(n, bc):
    c, o = _ctx(n, bc, ord_=9), Oracle(*n, bc=bc, ord_=9, crpow=True)
    st = _state(n, c.hs, 5)
    d = torch.from_numpy(st).cuda()
    dt = o.compute_dt(st, 0.5)
    for _ in range(2):
        c.step(d, dt)
        o.time_step(st, dt)
        assert _bits(d.cpu().numpy(), st)


@pytest.mark.parametrize("n,bc", GRIDS9 + [((9, 150, 140), PPP), ((200, 20, 30), WWW)])
def test_fp32_ord9_shapes_match_fp64(n, bc):
    c64, c32 = _ctx(n, bc, ord_=9), _ctx(n, bc, ord_=9, precision=capi.FP32)
    st = _state(n, c64.hs, 6)
    d32 = c32.new_state()
    d32[:5] = torch.from_numpy(st).cuda().float()
    d64 = d32[:5].double()
    dt = c64.cfl(d64, 0.5)
    for _ in range(2):
        c64.step(d64, dt)
        c32.step(d32, dt)
    h = c64.hs
    for v in range(5):
        a, b = (x[v, h:-h, h:-h, h:-h].double() for x in (d32, d64))
        norm = float(b.norm())
        assert float((a - b).norm()) <= 1e-5 * norm if norm else float(a.norm()) == 0, v
