"""Narrow channel groups and small ragged layers on the kernel that multiplies from input
patches in shared memory (poplibs_b200/csrc/patch.cuh), against the oracle and the general
route, which a context with a plan flag takes.

Small-integer data are exact in every operand type and in fp32 sums: bit for bit.
"""
import numpy as np
import pytest

import common as T
import oracle
from poplibs_b200 import capi

pytestmark = pytest.mark.gpu

TYPES = {"half": (capi.HALF, np.float16), "float": (capi.FLOAT, np.float32), "quarter": (capi.QUARTER, np.uint8)}
# groups, channels in / out, images, field, kernel, other parameters: one and several groups to
# a block, chunks that are full and not, odd and even numbers of them, rows that are tiles,
# parts and several images of one, and layers of one group that stay on the general route
LAYERS = {
    "8 to 8": (4, 8, 8, 3, (9, 7), (3, 3), dict(padding=1)),
    "32 groups": (32, 8, 8, 2, (8, 21), (3, 3), dict(padding=1)),
    "4 of 4": (2, 4, 4, 17, (13, 11), (3, 3), dict(padding=1)),
    "odd channels": (8, 9, 7, 2, (11, 13), (3, 3), dict(padding=1)),
    "24 to 24": (6, 24, 24, 2, (9, 9), (5, 5), dict(padding=2)),
    "wide row": (2, 8, 8, 1, (3, 150), (3, 3), dict(padding=1)),
    "small images": (8, 8, 8, 40, (4, 5), (3, 3), dict(padding=1)),
    "pointwise": (8, 12, 20, 3, (10, 9), (1, 1), {}),
    "one group, ragged": (1, 20, 36, 2, (13, 9), (3, 3), dict(padding=1)),
    "one group, wide": (1, 10, 100, 2, (9, 8), (3, 3), dict(padding=1)),
    "stride 2": (32, 8, 8, 2, (8, 13), (3, 3), dict(padding=1, stride=2)),
    "stride 2, pointwise": (4, 8, 8, 3, (9, 13), (1, 1), dict(stride=2)),
    "strides differ": (4, 8, 16, 2, (9, 12), (3, 2), dict(stride=[2, 1], in_pad_lo=[1, 0], in_pad_hi=[0, 1])),
    "dilated, flipped": (4, 6, 8, 2, (12, 9), (3, 3), dict(k_dilation=[2, 1], k_flip=[1, 0], padding=2)),
    "truncated": (4, 8, 8, 2, (12, 9), (3, 4), dict(k_trunc_lo=[1, 0], k_trunc_hi=[0, 1], in_trunc_lo=[1, 0], in_trunc_hi=[0, 2])),
    "padded output": (2, 8, 8, 2, (9, 9), (3, 3), dict(out_pad_lo=[1, 0], out_pad_hi=[0, 2], padding=1)),
}
GENERAL = [("24 to 24", "half")] + [(name, t) for name in ("one group, ragged", "one group, wide") for t in TYPES]
# groups, channels in / out, images, field, kernel, stride, and the types (half, float, quarter)
# whose forward pass and whose input gradient run on patches: every number of pixels (32, 64)
# and of columns (8 to 32) of an item that the planner chooses, in one and in several blocks of
# output channels, in each type and with the weights in either order
SHAPES = [
    (2, 2, 2, 1, (2, 2), 1, 2, "hfq", "hfq"),
    (8, 15, 19, 1, (2, 2), 1, 2, "hfq", "hfq"),
    (1, 36, 92, 4, (4, 3), 1, 2, "hfq", "hfq"),
    (4, 1, 1, 41, (35, 31), 3, 1, "hq", "hq"),
    (1, 59, 2, 1, (3, 2), 1, 2, "", "hfq"),
    (2, 70, 2, 1, (4, 2), 1, 2, "h", "hfq"),
    (1, 172, 4, 1, (2, 2), 1, 2, "hq", "hfq"),
    (2, 72, 4, 1, (2, 6), 1, 1, "hfq", "hfq"),
    (8, 4, 20, 37, (8, 23), 1, 1, "hfq", "hfq"),
    (16, 3, 25, 37, (7, 44), 1, 2, "hq", "hfq"),
    (3, 65, 1, 25, (11, 42), 3, 2, "", "q"),
    (2, 104, 8, 34, (10, 9), 1, 1, "fq", "q"),
    (16, 12, 2, 38, (3, 58), 7, 2, "", "hq"),
    (2, 68, 8, 13, (22, 22), 1, 1, "", "h"),
    (8, 57, 2, 37, (32, 7), 7, 2, "", "hq"),
    (16, 2, 22, 37, (12, 41), 3, 1, "hq", "f"),
    (3, 40, 4, 62, (14, 30), 7, 2, "", "hq"),
    (8, 1, 77, 17, (22, 16), 7, 1, "hq", ""),
    (2, 2, 123, 37, (6, 34), 7, 1, "hq", ""),
    (2, 178, 8, 34, (12, 37), 3, 2, "", "q"),
    (3, 8, 12, 50, (37, 30), 3, 1, "q", ""),
    (2, 72, 8, 54, (13, 29), 5, 2, "", "hq"),
    (16, 8, 56, 37, (8, 8), 3, 1, "hfq", "f"),
    (4, 8, 96, 37, (9, 30), 5, 2, "q", "hfq"),
    (1, 100, 3, 2, (14, 14), 3, 2, "", "hfq"),
    (1, 20, 36, 2, (5, 5), 3, 2, "", "hfq"),
]


@pytest.fixture(scope="module")
def general_ctx():
    ctx = capi.Context(0)
    ctx.set_plan_flags(capi.PLAN_NO_DUAL_ISSUE)
    return ctx


def ints(r, shape):
    return r.integers(-2, 3, shape).astype(np.float64)


@pytest.mark.parametrize("dtype", sorted(TYPES))
@pytest.mark.parametrize("name", sorted(LAYERS))
def test_layers(gpu_ctx, general_ctx, name, dtype):
    groups, ci, co, images, field, kernel, kw = LAYERS[name]
    plb, np_type = TYPES[dtype]
    cast = oracle.e4m3_encode if dtype == "quarter" else lambda v: v.astype(np_type)
    p = capi.ConvParams.make(images, list(field), list(kernel), ci, co, groups=groups, input_type=plb,
                             output_type=capi.FLOAT if dtype == "float" else capi.HALF, **kw)
    for pass_ in (capi.PASS_TRAINING_FWD, capi.PASS_TRAINING_BWD):
        assert (capi.conv_plan(p, pass_).kernel == 3) == ((name, dtype) not in GENERAL)
    spec = T.spec_from_params(p)
    r = T.rng(ci * 31 + co)
    x, w = ints(r, (images, groups * ci, *field)), ints(r, (groups, co, ci, *kernel))
    dy = ints(r, (images, groups * co, *p.output_field()))
    bias = r.integers(-3, 4, groups * co).astype(np.float32)
    want = oracle.conv_fwd(spec, x, w, bias)
    for ctx in (gpu_ctx, general_ctx):
        got = T.gpu_conv_fwd(p, cast(x), cast(w), bias=bias, ctx=ctx)
        assert (got.astype(np.float64) == want.reshape(got.shape)).all(), "forward"
    want = oracle.conv_bwd(spec, dy, w)
    for ctx in (gpu_ctx, general_ctx):
        got = T.gpu_conv_bwd(p, cast(dy), cast(w), ctx=ctx)
        assert (got.astype(np.float64) == want.reshape(got.shape)).all(), "input gradient"


@pytest.mark.parametrize("dtype", sorted(TYPES))
@pytest.mark.parametrize("layer", SHAPES, ids=str)
def test_shapes_of_items_and_blocks(gpu_ctx, layer, dtype):
    groups, ci, co, images, field, k, stride, fwd, bwd = layer
    plb, np_type = TYPES[dtype]
    cast = oracle.e4m3_encode if dtype == "quarter" else lambda v: v.astype(np_type)
    p = capi.ConvParams.make(images, list(field), [k, k], ci, co, groups=groups, stride=stride, padding=k // 2,
                             input_type=plb, output_type=capi.FLOAT if dtype == "float" else capi.HALF)
    spec = T.spec_from_params(p)
    r = T.rng(ci * 31 + co)
    w = ints(r, (groups, co, ci, k, k))
    for runs, pass_, shape, reference, run in (
            (fwd, capi.PASS_TRAINING_FWD, (images, groups * ci, *field), oracle.conv_fwd, T.gpu_conv_fwd),
            (bwd, capi.PASS_TRAINING_BWD, (images, groups * co, *p.output_field()), oracle.conv_bwd, T.gpu_conv_bwd)):
        if dtype[0] not in runs:
            continue
        assert capi.conv_plan(p, pass_).kernel == 3
        a = ints(r, shape)
        want = reference(spec, a, w)
        assert np.abs(want).max() <= 2048  # exact in half
        before = gpu_ctx.launch_count()
        got = run(p, cast(a), cast(w), ctx=gpu_ctx)
        assert gpu_ctx.launch_count() == before + 1
        assert (got.astype(np.float64) == want.reshape(got.shape)).all()


@pytest.mark.parametrize("dtype", sorted(TYPES))
@pytest.mark.parametrize("groups", [1, 4, 32])
def test_gradients_that_no_tap_reaches_are_zero(gpu_ctx, dtype, groups):
    """Strided layers whose filter meets padding alone have nothing to multiply; layers without
    output channels are refused."""
    plb, np_type = TYPES[dtype]
    kw = dict(groups=groups, input_type=plb, output_type=capi.FLOAT if dtype == "float" else capi.HALF)
    for field, kernel in (((1, 1), (1, 1)), ((1, 9), (1, 3))):
        p = capi.ConvParams.make(2, list(field), list(kernel), 8, 8, stride=2, padding=1, **kw)
        dy, w = np.ones((2, groups * 8, *p.output_field()), np_type), np.ones((groups, 8, 8, *kernel), np_type)
        assert (T.gpu_conv_bwd(p, dy, w) == 0).all()
    import torch
    none = capi.ConvParams.make(2, [6, 5], [3, 3], 8, 0, padding=1, **kw)
    x = torch.zeros((2, 6, 5, groups * 8), dtype=torch.float32, device="cuda")
    with pytest.raises(capi.PlbError):
        gpu_ctx.conv_bwd(none, x, x, x)


def test_narrow_groups_take_one_launch(gpu_ctx):
    r = T.rng(1)
    p = capi.ConvParams.make(2, [8, 13], [3, 3], 8, 8, groups=32, padding=1, stride=2)
    x, w = ints(r, (2, 256, 8, 13)).astype(np.float16), ints(r, (32, 8, 8, 3, 3)).astype(np.float16)
    dy = ints(r, (2, 256, *p.output_field())).astype(np.float16)
    for call in (lambda: T.gpu_conv_fwd(p, x, w), lambda: T.gpu_conv_bwd(p, dy, w)):
        before = gpu_ctx.launch_count()
        call()
        assert gpu_ctx.launch_count() == before + 1


@pytest.mark.parametrize("dtype", ["half", "float"])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_infinite_weights_and_padding(gpu_ctx, dtype, value):
    """Products with padding do not exist: an infinite weight there leaves the sum finite."""
    plb, np_type = TYPES[dtype]
    groups, c = 16, 8
    p = capi.ConvParams.make(2, [6, 7], [3, 3], c, c, groups=groups, input_type=plb, output_type=plb, padding=1)
    r = T.rng(2)
    x = r.integers(1, 3, (2, groups * c, 6, 7)).astype(np_type)
    w = r.integers(1, 3, (groups, c, c, 3, 3)).astype(np_type)
    clean = T.gpu_conv_fwd(p, x, w).astype(np.float64)
    w[3, 2, 5, 0, 1] = value  # first filter row: not read by the first output row
    got = T.gpu_conv_fwd(p, x, w).astype(np.float64)
    hit = np.zeros(clean.shape, bool)
    hit[:, 3 * c + 2, 1:] = True
    assert (got[~hit] == clean[~hit]).all()
    assert (np.isnan(got[hit]) if np.isnan(value) else got[hit] == value).all()


def test_float_layers_keep_their_precision(gpu_ctx, general_ctx):
    p = capi.ConvParams.make(2, [9, 12], [3, 3], 8, 8, groups=16, input_type=capi.FLOAT, output_type=capi.FLOAT, padding=1)
    spec = T.spec_from_params(p)
    r = T.rng(4)
    x, w = r.uniform(-1, 1, (2, 128, 9, 12)).astype(np.float32), r.uniform(-1, 1, (16, 8, 8, 3, 3)).astype(np.float32)
    want = oracle.conv_fwd(spec, x.astype(np.float64), w.astype(np.float64))
    off = [np.linalg.norm(T.gpu_conv_fwd(p, x, w, ctx=c) - want.reshape(2, 128, 9, 12)) / np.linalg.norm(want)
           for c in (gpu_ctx, general_ctx)]
    assert off[0] <= 1.1 * off[1] and off[0] < 2.0 ** -16, off


def test_wide_and_packed_layers_keep_the_general_route():
    """Layers that the tensor cores' operand rows fill: wide channels, and few channels whose taps
    share a row (the forward pass of a first layer has a kernel of its own)."""
    first = capi.ConvParams.make(256, [224, 224], [7, 7], 3, 64, padding=3, stride=2)
    assert capi.conv_plan(first, capi.PASS_TRAINING_FWD).kernel == 2
    assert capi.conv_plan(first, capi.PASS_TRAINING_BWD).kernel == 0
    for p in (capi.ConvParams.make(1, [56, 56], [3, 3], 64, 64, padding=1),
              capi.ConvParams.make(256, [28, 28], [3, 3], 128, 128, padding=1)):
        assert capi.conv_plan(p, capi.PASS_TRAINING_FWD).kernel == 0
        assert capi.conv_plan(p, capi.PASS_TRAINING_BWD).kernel == 0
