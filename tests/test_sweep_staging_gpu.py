"""The sweep's tile shapes and its two ways of staging rows (awfl_sweep.cuh), with the shape that
a launch takes asserted (awfl_sweep_shape): a grid that a retuned rule sends elsewhere fails here
instead of testing something else. test_sweep_coverage_cpu.py holds that the grids of this file
and of test_sweep_shapes_gpu.py reach every shape of the rule."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from awflcloud_b200 import capi  # noqa: E402
from oracle.pyoracle import Oracle  # noqa: E402
from test_adjoint_gpu import base_state, unit_direction  # noqa: E402

PPW, PPP, WWW = (0, 0, 1), (0, 0, 0), (1, 1, 1)
BUBBLE = dict(kind=capi.INIT_BUBBLE, noise_amp=0.01)
# (grid, bc, {dir: shape}) that no grid of test_sweep_shapes_gpu.py takes, lines and tiles ragged
FP64 = {9: [((200, 18, 18), PPW, {1: (8, 16), 2: (8, 16)})]}
FP32 = {5: [((92, 107, 50), PPW, {0: (8, 16), 1: (8, 16), 2: (4, 32)}), ((52, 10, 130), PPP, {1: (4, 32)}),
            ((17, 28, 130), WWW, {0: (4, 32)})],
        9: [((200, 18, 18), PPP, {1: (8, 16)}), ((44, 83, 9), PPW, {2: (8, 16)})]}
RECORD = [((9, 9, 51), PPP, {0: (16, 8), 2: (128, 1)}), ((135, 45, 9), PPW, {2: (8, 16)}),
          ((9, 58, 58), WWW, {0: (8, 16), 1: (128, 1)}), ((200, 18, 18), PPP, {0: (128, 1), 1: (8, 16)}),
          ((9, 10, 9), PPP, {0: (32, 4), 1: (16, 8), 2: (16, 8)}), ((12, 18, 25), PPW, {1: (32, 4), 2: (32, 4)})]


def _ctx(n, bc, **kw):
    return capi.Context(*n, bc=tuple("wall" if b else "periodic" for b in bc), **kw)


def _state(n, hs, seed):
    nx, ny, nz = n
    r = np.random.default_rng(seed)
    st = np.zeros((5, nz + 2 * hs, ny + 2 * hs, nx + 2 * hs))
    box = st[:, hs:hs + nz, hs:hs + ny, hs:hs + nx]
    scale = np.array([1e-3, 3.0, 2.0, 1.0, 0.3]).reshape(5, 1, 1, 1)
    box[:] = scale * (0.2 * r.standard_normal(box.shape) + np.sin(np.arange(nx) / nx * 2 * np.pi))
    return st


def _bits(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.int64), np.ascontiguousarray(b).view(np.int64))


def _takes(c, shapes, form=0):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        return  # the rule weighs tiles against SMs
    for d, s in shapes.items():
        assert c.sweep_shape(d, form)[:2] == s, d


@pytest.mark.parametrize("ord_,n,bc,shapes", [(o,) + g for o in FP64 for g in FP64[o]])
def test_fp64_shapes_equal_oracle(ord_, n, bc, shapes):
    c, o = _ctx(n, bc, ord_=ord_), Oracle(*n, bc=bc, ord_=ord_, crpow=True)
    _takes(c, shapes)
    st = _state(n, c.hs, 1)
    d = torch.from_numpy(st).cuda()
    dt = o.compute_dt(st, 0.5)
    for _ in range(2):
        c.step(d, dt)
        o.time_step(st, dt)
        assert _bits(d.cpu().numpy(), st)


@pytest.mark.parametrize("ord_,n,bc,shapes", [(o,) + g for o in FP32 for g in FP32[o]])
def test_fp32_shapes_match_fp64(ord_, n, bc, shapes):
    """The form's bar of 1e-5 relative L2, as for the other shapes."""
    c64, c32 = _ctx(n, bc, ord_=ord_), _ctx(n, bc, ord_=ord_, precision=capi.FP32)
    _takes(c32, shapes)
    d32 = c32.new_state()
    d32[:5] = torch.from_numpy(_state(n, c64.hs, 4)).cuda().float()
    d64 = d32[:5].double()
    dt = c64.cfl(d64, 0.5)
    for _ in range(2):
        c64.step(d64, dt)
        c32.step(d32, dt)
    h = c64.hs
    for v in range(5):
        a, b = (x[v, h:-h, h:-h, h:-h].double() for x in (d32, d64))
        assert float((a - b).norm()) <= 1e-5 * float(b.norm()), v


@pytest.mark.parametrize("n,bc,shapes", RECORD)
def test_fp64_tracer_shapes_equal_oracle(n, bc, shapes):
    c, o = _ctx(n, bc), Oracle(*n, bc=bc, crpow=True)
    _takes(c, shapes, 1)
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


@pytest.mark.parametrize("n,bc,shapes", RECORD)
def test_adjoint_shapes_transpose_the_tlm(n, bc, shapes):
    """The recording sweep feeds the reverse split: <w, M v> = <M^T w, v>, to the adjoint tests'
    rounding bar (a record in the wrong place is off by O(1))."""
    c = _ctx(n, bc)
    _takes(c, shapes, 2)
    s = base_state(c)
    dt = c.cfl(s, 0.5)
    gen = torch.Generator().manual_seed(7)
    v, w = unit_direction(c, gen), unit_direction(c, gen)
    both = torch.cat([s.clone(), v.clone()])
    c.dimswitch = 1
    for _ in range(3):
        c.step_tlm(both, dt)
    left = float((w * both[5:]).sum())
    c.dimswitch = 1
    lam = w.clone()
    c.step_adjoint(s, lam, 3, dt)
    right, scale = float((lam * v).sum()), float((lam * v).abs().sum())
    assert abs(left - right) <= 1e-11 * scale, (left, right, scale)


@pytest.mark.parametrize("bc", [PPW, WWW])
@pytest.mark.parametrize("tracers", [False, True])
def test_tma_staging_matches_cp_async(bc, tracers):
    """A 16-byte aligned FP32 state takes TMA in the x and y sweeps of this grid, the same state
    two floats further on cp.async: partial tiles and partial last chunks along every line.
    Both stage the same values; the two instantiations may contract differently, so the
    bound is FP32 rounding, relative L2 <= 1e-6 per variable after 4 steps (a row staged wrongly
    shows as O(1))."""
    n = (92, 107, 50)
    ca, cb = _ctx(n, bc, precision=capi.FP32), _ctx(n, bc, precision=capi.FP32)
    s = ca.new_state()
    ca.init_state(s, **BUBBLE)
    dt = ca.cfl(s, 0.8)
    buf = torch.empty(s.numel() + 2, dtype=torch.float32, device=s.device)
    u = buf[2:].view(s.shape)
    u.copy_(s)
    for d in (0, 1):
        if torch.cuda.get_device_properties(0).multi_processor_count == 148:
            assert ca.sweep_shape(d, int(tracers), s) == (8, 16, True)
        assert cb.sweep_shape(d, int(tracers), u)[2] is False
    ta = ca.new_tracers(2)
    ca.init_tracers(ta)
    tb = ta.clone()
    for _ in range(4):
        if tracers:
            ca.step_tracers(s, ta, dt)
            cb.step_tracers(u, tb, dt)
        else:
            ca.step(s, dt)
            cb.step(u, dt)
    assert torch.isfinite(s).all()
    h = ca.hs
    for x, y in zip(list(s[:5]) + list(ta), list(u[:5]) + list(tb)):
        x, y = x[h:-h, h:-h, h:-h].double(), y[h:-h, h:-h, h:-h].double()
        assert float((x - y).norm()) <= 1e-6 * float(y.norm())
    assert ca.check_state(s) == 0 and cb.check_state(u) == 0
