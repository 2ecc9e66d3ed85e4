"""The grids that the GPU tests sweep reach every tile shape of the launch rule (awfl_sweep.cuh),
by the rule itself on a host-only context (148 SMs): a changed cost factor cannot leave a kernel
untested without a word."""
import pytest

pytest.importorskip("torch")

import test_sweep_shapes_gpu as shapes  # noqa: E402
import test_sweep_staging_gpu as staging  # noqa: E402
from awflcloud_b200 import capi  # noqa: E402

# every shape of the rule, along x, y and z: (precision, ord) -> plain sweeps; FP64 ord 5 also recording
PLAIN = {
    (capi.FP64, 5): [{(16, 8), (8, 16), (32, 4), (128, 1)}, {(8, 16), (16, 8), (32, 4), (128, 1)},
                     {(8, 16), (16, 8), (32, 4), (128, 1)}],
    (capi.FP64, 9): [{(32, 4), (16, 8), (128, 1)}, {(8, 16), (16, 8), (32, 4), (128, 1)},
                     {(8, 16), (16, 8), (32, 4), (128, 1)}],
    (capi.FP32, 5): [{(8, 16), (4, 32), (16, 8), (32, 4), (128, 1)}, {(8, 16), (4, 32), (16, 8), (32, 4), (128, 1)},
                     {(4, 32), (8, 16), (16, 8), (32, 4), (128, 1)}],
    (capi.FP32, 9): [{(32, 4), (16, 8), (128, 1)}, {(16, 8), (8, 16), (32, 4), (128, 1)},
                     {(8, 16), (16, 8), (32, 4), (128, 1)}],
}


def _taken(grids, form, **kw):
    got = [set(), set(), set()]
    for n, bc in grids:
        c = capi.Context(*n, device=-1, **kw)
        for d in range(3):
            if not (d == 1 and n[1] == 1):  # sim2d has no y sweep
                got[d].add(c.sweep_shape(d, form)[:2])
        c.close()
    return got


def _params(fn):
    """The (n, bc) pairs of a test's own parametrisation."""
    return [p for m in fn.pytestmark if m.name == "parametrize" for p in m.args[1]]


def _grids(prec, ord_):
    own = {(capi.FP64, 5): [shapes.test_fp64_shapes_equal_oracle], (capi.FP64, 9): [shapes.test_fp64_ord9_shapes_equal_oracle],
           (capi.FP32, 5): [shapes.test_fp32_shapes_match_fp64], (capi.FP32, 9): [shapes.test_fp32_ord9_shapes_match_fp64]}
    more = (staging.FP64 if prec == capi.FP64 else staging.FP32).get(ord_, [])
    return [g for fn in own[prec, ord_] for g in _params(fn)] + [g[:2] for g in more]


@pytest.mark.parametrize("prec,ord_", list(PLAIN))
def test_every_plain_shape_is_swept(prec, ord_):
    assert _taken(_grids(prec, ord_), 0, ord_=ord_, precision=prec) == PLAIN[prec, ord_]


@pytest.mark.parametrize("form", [1, 2])
def test_every_recording_shape_is_swept(form):
    grids = [g[:2] for g in staging.RECORD]
    if form == 1:
        grids += _params(shapes.test_fp64_tracer_shapes_equal_oracle)
    got = _taken(grids, form)
    for d in range(3):
        missing = PLAIN[capi.FP64, 5][d] - got[d]
        assert not missing, (d, missing)


def test_query_refuses_what_no_sweep_takes():
    c = capi.Context(16, 12, 8, precision=capi.FP32, device=-1)
    for d, form in ((3, 0), (-1, 0), (0, 3), (0, 2)):  # the adjoint is FP64's
        with pytest.raises(Exception, match="dir must be|form must be"):
            c.sweep_shape(d, form)


@pytest.mark.parametrize("ord_,dirs", [(5, (2,)), (9, (0, 1, 2))])
@pytest.mark.parametrize("n", [(254, 256, 128), (250, 250, 128), (1022, 64, 64)])
def test_rows_that_tma_cannot_address_matter_only_where_tma_is_used(ord_, dirs, n):
    """The FP32 z sweep and every ord-9 one stage by cp.async whatever the row pitch: they take
    the shape of the next wider grid whose rows are a multiple of 16 bytes."""
    narrow = capi.Context(*n, ord_=ord_, precision=capi.FP32, device=-1)
    wide = capi.Context(n[0] + 2, *n[1:], ord_=ord_, precision=capi.FP32, device=-1)
    for d in dirs:
        assert narrow.sweep_shape(d) == wide.sweep_shape(d), d
