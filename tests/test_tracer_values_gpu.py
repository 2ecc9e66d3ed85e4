"""FP32 tracer transport over the values a tracer can have: rough fields in any unit."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from awflcloud_b200 import capi  # noqa: E402

BUBBLE = dict(kind=capi.INIT_BUBBLE, noise_amp=0.01)


@pytest.mark.parametrize("ord_", [5, 9])
@pytest.mark.parametrize("scale", [1.0, 1e4, 1e6])
def test_fp32_rough_tracers_follow_fp64(ord_, scale):
    """Random values from cell to cell, of order one to 1e6 (number concentrations): the FP32
    form's tracers agree with the FP64 path's to the form's bar of 1e-6 relative L2. An FP32
    reconstruction's error is at most 2^-24 * 1026 of the stencil's range, 6e-5 of it; the
    four steps change the field by 2e-4 of itself, so 1e-6 leaves a factor of fifty."""
    n = (32, 24, 20)
    c32, c64 = capi.Context(*n, ord_=ord_, precision=capi.FP32), capi.Context(*n, ord_=ord_)
    s32, s64 = c32.new_state(), c64.new_state()
    c32.init_state(s32, **BUBBLE)
    c64.init_state(s64, **BUBBLE)
    h = c64.hs
    box = (slice(None), slice(h, -h), slice(h, -h), slice(h, -h))
    t64 = c64.new_tracers(2)
    t64.zero_()
    gen = torch.Generator(device="cuda").manual_seed(2)
    t64[box] = scale * torch.rand(t64[box].shape, generator=gen, device="cuda", dtype=torch.float64)
    t32 = t64.clone()
    dt = c64.cfl(s64, 0.4)
    for _ in range(4):
        c64.step_tracers(s64, t64, dt, pos=[1, 0])
        c32.step_tracers(s32, t32, dt, pos=[1, 0])
    for l in range(2):
        a, b = t32[box][l], t64[box][l]
        assert float((a - b).norm()) <= 1e-6 * float(b.norm()), l


@pytest.mark.parametrize("dir_", [0, 1, 2])
@pytest.mark.parametrize("value", ["inf", "nan", "-inf"])
def test_fp32_limited_tracer_of_one_bad_cell(dir_, value):
    """A positive-definite tracer of zeros with one cell that is not a number: the edges it
    touches are clamped to zero, so the fluxes are zero and the limiter's factor min(1, r) of
    the cell decides. +inf: the factor is 1, the cell stays +inf and nothing else moves. NaN and
    -inf: the factor makes the cell's outflow a NaN, which reaches the cell and the one
    downwind of it."""
    n = (16, 12, 10)
    c = capi.Context(*n, bc=("periodic",) * 3, precision=capi.FP32)
    s = c.new_state()
    s.zero_()
    s[1 + dir_] = 20.0  # momentum along the split, everywhere
    h = c.hs
    at = [4, 5, 6]  # k, j, i
    t = c.new_tracers(1)
    t.zero_()
    t[(0,) + tuple(h + x for x in at)] = float(value)
    c.split_tracers(s, t, 0.1, dir_, pos=[1])
    got = t[0, h:-h, h:-h, h:-h].cpu()
    want = torch.zeros_like(got)
    want[tuple(at)] = float("inf") if value == "inf" else float("nan")
    if value != "inf":
        at[2 - dir_] += 1
        want[tuple(at)] = float("nan")
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.nan_to_num(nan=0.0, posinf=1.0), want.nan_to_num(nan=0.0, posinf=1.0))
