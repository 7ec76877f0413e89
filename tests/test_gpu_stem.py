"""Layers of few input channels on the kernel that reads the image as it is
(poplibs_b200/csrc/stem.cu), against the oracle and the general route, which a context with a
plan flag takes.  Small-integer data are exact: bit for bit.
"""
import numpy as np
import pytest

import common as T
import oracle
from poplibs_b200 import capi

pytestmark = pytest.mark.gpu

# channels in / out, images, field, kernel, stride, padding low / high: words and single
# elements, rows of odd length, strips of one and several tiles, parts of a row, more strips
# than SMs, padding that is not a multiple of the stride, odd numbers of filter columns
LAYERS = {
    "stem": (3, 64, 2, (32, 32), (7, 7), 2, (3, 3), (3, 3)),
    "odd field": (3, 64, 3, (33, 37), (7, 7), 2, (3, 3), (3, 3)),
    "wide": (3, 32, 1, (5, 420), (7, 7), 2, (3, 3), (3, 3)),
    "many strips": (3, 64, 40, (40, 46), (7, 7), 2, (3, 3), (3, 3)),
    "one channel": (1, 96, 5, (19, 23), (3, 7), 2, (1, 3), (1, 3)),
    "four channels": (4, 16, 2, (21, 18), (3, 3), 2, (1, 1), (1, 1)),
    "four, odd rows": (4, 48, 2, (17, 19), (3, 3), 2, (1, 1), (1, 1)),
    "stride 1": (3, 64, 2, (15, 28), (3, 3), 1, (1, 1), (1, 1)),
    "stride 1, two": (2, 128, 2, (9, 130), (3, 3), 1, (1, 1), (1, 1)),
    "wide output": (3, 256, 1, (12, 14), (3, 3), 1, (1, 1), (1, 1)),
    "pads differ": (3, 32, 2, (11, 14), (5, 4), 2, (1, 2), (2, 0)),
    "no padding": (3, 32, 2, (16, 17), (3, 5), 2, (0, 0), (0, 0)),
    "smallest": (1, 16, 1, (2, 2), (3, 3), 1, (1, 1), (1, 1)),
    "five columns": (2, 48, 2, (13, 20), (5, 5), 1, (2, 2), (2, 2)),
    "seven columns": (5, 16, 2, (9, 21), (2, 7), 1, (0, 3), (1, 3)),
}


@pytest.fixture(scope="module")
def general_ctx():
    ctx = capi.Context(0)
    ctx.set_plan_flags(capi.PLAN_NO_DUAL_ISSUE)
    return ctx


def layer(name, **kw):
    ci, co, images, field, kernel, stride, lo, hi = LAYERS[name]
    return capi.ConvParams.make(images, list(field), list(kernel), ci, co, stride=stride, in_pad_lo=list(lo), in_pad_hi=list(hi), **kw)


def bfloat16_bits(v):
    """(small whole numbers are exact)"""
    return (v.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)


TYPES = {"half": (capi.HALF, lambda v: v.astype(np.float16)), "bfloat16": (capi.BFLOAT16, bfloat16_bits)}


@pytest.mark.parametrize("dtype", sorted(TYPES))
@pytest.mark.parametrize("name", sorted(LAYERS))
def test_layers(gpu_ctx, general_ctx, name, dtype):
    plb, cast = TYPES[dtype]
    p = layer(name, input_type=plb, output_type=capi.HALF)
    plan = capi.conv_plan(p)
    assert (plan.kernel, plan.in_place) == (2, 1)
    ci, co, images, field, kernel = LAYERS[name][:5]
    spec = T.spec_from_params(p)
    r = T.rng(ci * 31 + co)
    x = r.integers(-2, 3, (images, ci, *field)).astype(np.float64)
    w = r.integers(-2, 3, (1, co, ci, *kernel)).astype(np.float64)
    bias = r.integers(-3, 4, co).astype(np.float32)
    for b in (bias, None):
        want = oracle.conv_fwd(spec, x, w, b)
        for ctx, launches in ((gpu_ctx, 1), (general_ctx, 2)):
            before = ctx.launch_count()
            got = T.gpu_conv_fwd(p, cast(x), cast(w), bias=b, ctx=ctx)
            assert ctx.launch_count() - before == launches
            assert (got.astype(np.float64) == want.reshape(got.shape)).all()


@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_infinite_operands_reach_their_products_only(gpu_ctx, value):
    p = capi.ConvParams.make(2, [24, 26], [7, 7], 3, 32, stride=2, padding=3)
    r = T.rng(2)
    x = r.integers(1, 3, (2, 3, 24, 26)).astype(np.float16)
    w = r.integers(1, 3, (1, 32, 3, 7, 7)).astype(np.float16)
    clean = T.gpu_conv_fwd(p, x, w).astype(np.float64)
    x[1, 2, 10, 13] = value
    got = T.gpu_conv_fwd(p, x, w).astype(np.float64)
    hit = np.zeros(clean.shape, bool)
    rows = [oh for oh in range(12) if 0 <= 10 - (2 * oh - 3) < 7]
    cols = [ow for ow in range(13) if 0 <= 13 - (2 * ow - 3) < 7]
    hit[1][:, rows[0]:rows[-1] + 1, cols[0]:cols[-1] + 1] = True
    assert (got[~hit] == clean[~hit]).all()
    assert (np.isnan(got[hit]) if np.isnan(value) else got[hit] == value).all()


@pytest.mark.parametrize("dtype", sorted(TYPES))
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_infinite_weights_and_padding(gpu_ctx, value, dtype):
    """Products with padding do not exist: an infinite weight of the first filter row leaves the
    output rows finite that meet it above the image."""
    plb, cast = TYPES[dtype]
    p = capi.ConvParams.make(2, [24, 26], [7, 7], 3, 32, stride=2, padding=3, input_type=plb, output_type=capi.HALF)
    r = T.rng(3)
    x, w = r.integers(1, 3, (2, 3, 24, 26)).astype(np.float64), r.integers(1, 3, (1, 32, 3, 7, 7)).astype(np.float64)
    clean = T.gpu_conv_fwd(p, cast(x), cast(w)).astype(np.float64)
    w[0, 5, 1, 0, 3] = value
    got = T.gpu_conv_fwd(p, cast(x), cast(w)).astype(np.float64)
    hit = np.zeros(clean.shape, bool)
    hit[:, 5, 2:] = True  # (rows 0 and 1 meet it at input rows -3 and -1)
    assert (got[~hit] == clean[~hit]).all()
    assert (np.isnan(got[hit]) if np.isnan(value) else got[hit] == value).all()
