"""awfl_cfl on cells whose speed is not a number: what each form leaves out of its minimum."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from awflcloud_b200 import capi  # noqa: E402

BUBBLE = dict(kind=capi.INIT_BUBBLE, noise_amp=0.01)
NX, NY, NZ = 16, 12, 8
WIND = (150.0, -320.0, 260.0)  # of one cell, the fastest of the grid


def _dt(prec, bad):
    """The step for a state whose one fast cell has `bad` = {variable: value}, at cfl 0.5."""
    c = capi.Context(NX, NY, NZ, precision=prec)
    s = c.new_state()
    c.init_state(s, **BUBBLE)
    cell = (c.hs + 3, c.hs + 4, c.hs + 5)
    rho = float(s[(0,) + cell]) + float(c.background()["hyDensCells"][cell[0]])
    for v in range(3):
        s[(1 + v,) + cell] = WIND[v] * rho
    for v, x in bad.items():
        s[(v,) + cell] = x
    return c.cfl(s, 0.5), c


def _quiet(prec):
    c = capi.Context(NX, NY, NZ, precision=prec)
    s = c.new_state()
    c.init_state(s, **BUBBLE)
    return c.cfl(s, 0.5)


@pytest.mark.parametrize("var", [1, 2, 3])
def test_fp32_nan_momentum_hides_its_own_direction_alone(var):
    """The FP32 form takes the minimum over the directions that are numbers: with one momentum
    of the fast cell NaN, the step is that of the other two (dz < dx < dy here: 1250, 1250,
    1667 m, so z, then y bound it), below the step of the quiet grid."""
    all_, c = _dt(capi.FP32, {})
    got, _ = _dt(capi.FP32, {var: float("nan")})
    quiet = _quiet(capi.FP32)
    # the two other directions' speeds with this one at rest bound the step the same way
    rest, _ = _dt(capi.FP32, {var: 0.0})
    assert got == rest, (got, rest, all_, quiet)
    assert all_ <= got < quiet


@pytest.mark.parametrize("var,hidden", [(1, (0,)), (2, (0, 1)), (3, (0, 1, 2))])
def test_fp64_nan_momentum_hides_the_directions_before_it(var, hidden):
    """The reference's comparisons (Spatial:169-183): a NaN of direction d also hides the
    directions before d."""
    got, _ = _dt(capi.FP64, {var: float("nan")})
    rest, _ = _dt(capi.FP64, {1 + d: 0.0 for d in hidden})
    quiet = _quiet(capi.FP64)
    want = quiet if len(hidden) == 3 else min(rest, quiet)
    assert got == want, (got, rest, quiet)


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
def test_infinite_momentum_is_refused(prec):
    for var in (1, 2, 3):
        for x in (float("inf"), -float("inf")):
            with pytest.raises(Exception, match="non-finite or non-positive"):
                _dt(prec, {var: x})
