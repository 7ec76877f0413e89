"""Channel groups of 8 and 16 on the kernels that give a warp to a group
(poplibs_b200/csrc/rows.cu, rows_wu.cu), against the oracle.

Small-integer data are exact in fp32 sums: bit for bit.
"""
import numpy as np
import pytest

import common as T
import oracle
from poplibs_b200 import capi

pytestmark = pytest.mark.gpu

# groups, channels, images, field, kernel, other parameters: rows of less than eight pixels (two images
# side by side, an odd number of them), of parts, whole and several sixteens, tiles of part rows,
# one row, more groups than a block takes and fewer, paddings on one side, flipped and truncated
LAYERS = {
    "two images a step": (8, 8, 5, (6, 7), 3, dict(padding=1)),
    "two images a step, 16": (4, 16, 4, (9, 8), 3, dict(padding=1)),
    "9 columns": (8, 8, 3, (10, 9), 3, dict(padding=1)),
    "16 columns": (8, 8, 2, (16, 16), 3, dict(padding=1)),
    "28 columns": (32, 8, 4, (28, 28), 3, dict(padding=1)),
    "33 columns": (9, 8, 2, (21, 33), 3, dict(padding=1)),
    "112 columns": (8, 8, 1, (40, 112), 3, dict(padding=1)),
    "one row": (8, 8, 3, (1, 50), 3, dict(padding=1)),
    "tall": (16, 8, 1, (112, 16), 3, dict(padding=1)),
    "no padding": (3, 8, 3, (13, 18), 3, {}),
    "two groups": (2, 8, 9, (12, 13), 3, dict(padding=1)),
    "16 channels": (32, 16, 2, (15, 16), 3, dict(padding=1)),
    "16 channels, 30 columns": (6, 16, 3, (17, 30), 3, dict(padding=1)),
    "16 channels, two groups": (2, 16, 3, (11, 16), 3, dict(padding=1)),
    "5x5": (8, 8, 3, (14, 15), 5, dict(padding=2)),
    "5x5, 40 columns": (11, 8, 2, (23, 40), 5, dict(padding=2)),
    "5x5, two images": (8, 8, 3, (7, 5), 5, dict(padding=2)),
    "5x5, 16 channels": (8, 16, 2, (12, 20), 5, dict(padding=2)),
    "one side": (8, 8, 2, (14, 30), 3, dict(in_pad_lo=[2, 0], in_pad_hi=[0, 2])),
    "truncated": (8, 8, 2, (16, 24), 3, dict(in_trunc_lo=[1, 2], in_trunc_hi=[2, 1], padding=1)),
    "output truncated": (8, 8, 2, (16, 24), 3, dict(out_trunc_lo=[1, 2], out_trunc_hi=[2, 1], padding=1)),
}
FLIPPED = {"flipped": (8, 8, 2, (13, 17), 3, dict(padding=1, k_flip=[1, 0]))}


def _layer(name):
    g, c, n, field, k, kw = {**LAYERS, **FLIPPED}[name]
    return capi.ConvParams.make(n, list(field), [k, k], c, c, groups=g, **kw)


def _data(p, r):
    g, c, n = p.groups, p.in_chans_per_group, p.batch
    field, k = [p.field[0], p.field[1]], p.kernel[0]
    return (T.small_int_half(r, (n, g * c, *field)), T.small_int_half(r, (g, c, c, k, k), -3, 3),
            T.small_int_half(r, (n, g * c, *p.output_field())))


@pytest.mark.parametrize("name", {**LAYERS, **FLIPPED})
def test_rows_match_oracle(gpu_ctx, name):
    p = _layer(name)
    spec = T.spec_from_params(p)
    r = T.rng(len(name))
    x, w, dy = _data(p, r)
    bias = r.integers(-8, 9, p.groups * p.out_chans_per_group).astype(np.float32)
    for pass_ in (capi.PASS_TRAINING_FWD, capi.PASS_TRAINING_BWD):
        assert capi.conv_plan(p, pass_).in_place
    got = T.gpu_conv_fwd(p, x, w, bias=bias)
    assert (got.astype(np.float64) == oracle.conv_fwd(spec, x, w, bias).reshape(got.shape)).all()
    got = T.gpu_conv_bwd(p, dy, w)
    assert (got.astype(np.float64) == oracle.conv_bwd(spec, dy, w).reshape(got.shape)).all()


@pytest.mark.parametrize("name", [n for n in LAYERS if n != "5x5, 16 channels"])
def test_rows_weight_gradient_matches_oracle(gpu_ctx, name):
    p = _layer(name)
    x, _, dy = _data(p, T.rng(len(name)))
    assert capi.conv_wu_plan(p).kernel == 3
    dw16, dw32 = T.gpu_conv_wu(p, x, dy)
    want = oracle.conv_wu(T.spec_from_params(p), x, dy)[0].reshape(dw32.shape)
    assert (dw32.astype(np.float64) == want).all()
    assert (dw16 == want.astype(np.float16)).all()


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("name", ["28 columns", "two images a step", "16 channels, 30 columns", "5x5"])
def test_rows_keep_infinities_to_their_products(gpu_ctx, name, value):
    """An infinite weight meets no padding, an infinite activation no output beyond the image."""
    p = _layer(name)
    r = T.rng(3)
    x, w, dy = _data(p, r)
    k, c, (h, width), pad = p.kernel[0], p.in_chans_per_group, (p.field[0], p.field[1]), p.in_pad_lo[0]
    group = p.groups - 1
    # the tap's products exist where its input row and column do
    wi = w.copy()
    wi[group, 2, 1, 0, 0] = value
    got = T.gpu_conv_fwd(p, np.abs(x) + 1, wi)
    finite = np.isfinite(got)
    hit = np.zeros_like(finite)
    hit[:, group * c + 2, pad:, pad:] = True
    assert (finite == ~hit).all()
    # the last column's activation meets the taps whose output column exists
    xi = x.copy()
    xi[0, group * c + 1, h - 1, width - 1] = value
    _, dw = T.gpu_conv_wu(p, xi, np.abs(dy) + 1)
    finite = np.isfinite(dw)
    hit = np.zeros_like(finite)
    hit[group, :, 1, pad:, pad:] = True
    assert (finite == ~hit).all()
