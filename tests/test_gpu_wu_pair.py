"""Weight gradients of 64 output channels whose filter rows are shared out between the two
halves of the tensor-core instruction's rows (poplibs_b200/csrc/wu_sm100.cuh), against the oracle.

Small-integer data are exact in fp32 sums: bit for bit.
"""
import numpy as np
import pytest

import common as T
import oracle
from poplibs_b200 import capi

pytestmark = pytest.mark.gpu

# images, field, kernel, channels in / out, other parameters: even and odd numbers of filter rows
# (the odd ones leave half a row of accumulators unused), steps of one and several instructions,
# rows of 16 to 64 pixels and of several images, rows of tiles that end inside a box, above it and
# below it, dilated rows, a horizontal stride, more than 64 input channels, and first layers
LAYERS = {
    "3x3": (5, (34, 48), (3, 3), 64, 64, dict(padding=1)),
    "3x3, one image": (1, (49, 64), (3, 3), 64, 64, dict(padding=1)),
    "2 rows": (24, (12, 48), (2, 1), 64, 64, {}),
    "4 rows": (6, (19, 32), (4, 3), 64, 64, dict(padding=1)),
    "5x5": (8, (12, 48), (5, 5), 64, 64, dict(padding=2)),
    "7 rows": (4, (24, 48), (7, 2), 64, 64, dict(padding=3)),
    "8 rows": (6, (24, 16), (8, 1), 64, 64, dict(in_pad_lo=[3, 0], in_pad_hi=[4, 0])),
    "many small images": (101, (13, 8), (3, 3), 64, 64, dict(padding=1)),
    "dilated": (24, (17, 32), (3, 3), 64, 64, dict(k_dilation=[3, 2], padding=[3, 2])),
    "strided columns": (32, (13, 64), (3, 3), 64, 64, dict(stride=[1, 2], padding=1)),
    "128 in": (2, (24, 32), (3, 3), 128, 64, dict(padding=1)),
    "160 in, 2 rows": (8, (24, 32), (2, 3), 160, 64, dict(padding=1)),
    "first, 7x7/2": (2, (64, 96), (7, 7), 3, 64, dict(stride=2, padding=3)),
    "first, 3x3": (8, (34, 64), (3, 3), 3, 64, dict(padding=1)),
    "no padding": (2, (33, 33), (3, 3), 64, 64, {}),
    "output truncated": (2, (32, 32), (3, 3), 64, 64, dict(padding=1, out_trunc_lo=[2, 0], out_trunc_hi=[1, 0])),
}


def _params(name):
    n, field, kernel, ci, co, kw = LAYERS[name]
    return capi.ConvParams.make(n, list(field), list(kernel), ci, co, **kw)


@pytest.mark.parametrize("name", LAYERS)
def test_wu_pair_matches_oracle(gpu_ctx, name):
    p = _params(name)
    n, field, _, ci, co, _ = LAYERS[name]
    r = T.rng(len(name))
    x = T.small_int_half(r, (n, ci) + field)
    dy = T.small_int_half(r, (n, co) + tuple(p.output_field()))
    want, _ = oracle.conv_wu(T.spec_from_params(p), x, dy)
    plan = capi.conv_wu_plan(p, capi.ConvOptions.make(split_k=1))
    assert plan.tile_m == 64
    for split in (0, 1, 3):
        _, got = T.gpu_conv_wu(p, x, dy, opt=capi.ConvOptions.make(split_k=split))  # (1: paired, 0: if it pays)
        assert (got.astype(np.float64) == want.reshape(got.shape)).all(), split


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("row", [0, 1, -2, -1])
@pytest.mark.parametrize("pad", [1, 0])
def test_wu_pair_keeps_infinities_of_edge_rows_to_their_taps(gpu_ctx, pad, row, value):
    """Rows of the walk that have output gradients for one half only give the other half nothing."""
    n, ci, co, oh, ow = 12, 64, 64, 34, 48  # (whole boxes of columns)
    height, width = oh + 2 * (1 - pad), ow + 2 * (1 - pad)
    p = capi.ConvParams.make(n, [height, width], [3, 3], ci, co, padding=pad)
    opt = capi.ConvOptions.make(split_k=2)
    assert capi.conv_wu_plan(p, opt).tile_m == 64
    r = T.rng(5)
    x = T.small_int_half(r, (n, ci, height, width))
    dy = T.small_int_half(r, (n, co, oh, ow), 1, 4)
    row %= height
    x[0, 3, row, 9] = value
    _, got = T.gpu_conv_wu(p, x, dy, opt=opt)
    finite = np.isfinite(got[0])
    assert finite[:, [c for c in range(ci) if c != 3]].all()
    for k in range(3):
        # tap k meets the input row where output row `row` + pad - k exists
        assert finite[:, 3, k].all() != (0 <= row + pad - k < oh), k


# images, field, kernel, groups, channels of each in / out, type: the other operands that the planner
# sends here: bfloat16, the pieces of floats, and groups contracted together to 64 output channels
# (all of them, with channels left over, and some of several)
FORMS = {
    "bfloat16": (5, (34, 48), (3, 3), 1, 64, 64, "bfloat16"),
    "bfloat16, 40 in, 7 rows": (3, (30, 32), (7, 3), 1, 40, 64, "bfloat16"),
    "bfloat16, groups": (6, (24, 32), (5, 5), 4, 16, 16, "bfloat16"),
    "float": (5, (34, 48), (3, 3), 1, 64, 64, "float32"),
    "float, 5 rows": (4, (24, 48), (5, 5), 1, 64, 64, "float32"),
    "float, groups": (3, (24, 32), (5, 5), 4, 16, 16, "float32"),
    "4 groups of 16": (6, (24, 32), (5, 5), 4, 16, 16, "float16"),
    "8 groups of 8": (6, (24, 32), (7, 7), 8, 8, 8, "float16"),
    "3 groups of 20": (6, (24, 32), (5, 5), 3, 20, 20, "float16"),
    "8 groups, 32 to 16": (6, (24, 32), (3, 3), 8, 32, 16, "float16"),
    "10 groups, 32 to 16": (6, (24, 32), (3, 3), 10, 32, 16, "float16"),
}


@pytest.mark.parametrize("name", FORMS)
def test_wu_pair_of_other_operands(gpu_ctx, name):
    import torch
    n, field, kernel, g, ci, co, dtype = FORMS[name]
    plb = {"float16": capi.HALF, "bfloat16": capi.BFLOAT16, "float32": capi.FLOAT}[dtype]
    pad = [k // 2 for k in kernel]
    p = capi.ConvParams.make(n, list(field), list(kernel), ci, co, groups=g, input_type=plb,
                             output_type=capi.FLOAT if plb == capi.FLOAT else capi.HALF, padding=pad)
    torch.manual_seed(len(name))
    # (floats of more bits than one piece has: the sums of their products are exact all the same)
    most = 300 if plb == capi.FLOAT else 2
    x = torch.randint(-most, most + 1, (n, *field, g * ci), device="cuda").to(getattr(torch, dtype))
    dy = torch.randint(-2, 3, (n, *field, g * co), device="cuda").to(x.dtype)
    dw = torch.full((g, *kernel, co, ci), 7.0, device="cuda")
    nchw = lambda t: t.permute(0, 3, 1, 2).double()
    want = torch.nn.grad.conv2d_weight(nchw(x), (g * co, ci, *kernel), nchw(dy), padding=pad, groups=g)
    torch.cuda.synchronize()
    for split in (1, 2):
        opt = capi.ConvOptions.make(split_k=split)
        assert capi.conv_wu_plan(p, opt).tile_m == 64
        gpu_ctx.conv_wu(p, x, dy, None, dw, opt=opt)
        gpu_ctx.synchronize()
        assert torch.equal(dw.permute(0, 3, 4, 1, 2).reshape(want.shape).double(), want), split
        dw.fill_(7.0)
        torch.cuda.synchronize()
