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
# side by side in the weight gradient), of parts, whole and several sixteens, one row, more groups than a
# block takes and fewer, paddings on one side, flipped and truncated.  As small as this, all forward
# passes and input gradients take tiles of sixteen columns; TILES and WU_TILES below have the others.
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


def _tile(p):
    """The forward pass's tile, the one that the estimate in rows.cu takes: columns, rows, images and
    sixteens of columns that a warp walks for each row."""
    c, k, (h, w), n = p.in_chans_per_group, p.kernel[0], p.output_field(), p.batch
    up = lambda a, b: -(-a // b)
    slabs, most = up(p.groups * c, 64), 2 if c == 8 or k == 5 else 3
    products = k * (8.3 * (k // 2) + 4.2) if c == 8 else 2 * k * k * 8.3
    best = None
    for steps in range(1, 8):
        for images in (1, 2) if steps == 1 and w <= 8 else (1,):
            columns = 16 * steps // images
            row = images * up(columns + k - 1, 8) * 8 * 128
            twos = steps % 2 == 0 and k == 3
            for rows in range(1, min(h, 110 * 1024 // row - (k - 1)) + 1) if steps == 1 or 16 * (steps - 1) < w else ():
                if up(h, up(h, rows)) != rows:
                    continue
                resident = max(1, min(most, 226 * 1024 // (row * (rows + k - 1) + 1024)))
                blocks = slabs * up(w, columns) * up(h, rows) * up(n, images)
                share, here = blocks / (148 * resident), min(resident, up(blocks, 148))
                read, written = images * (rows + k - 1) * (columns + k - 1) * 128, images * rows * min(columns, w) * 128
                walked = (rows + k - 1) * steps
                busy = max(walked * (0.747 * products + (4 if twos else 14.2)) * (64 // c) * here / 4,
                           walked * (1.34 * products + (84 if twos else 168)))
                us = max(1, 0.425 * np.ceil(share) + 0.575 * share) * (1781 + here * (0.0413 * read + 0.0192 * written) + busy)
                if best is None or us < best[0]:
                    best = us, (columns, rows, images, steps)
    return best[1]


# groups, channels, images, field, kernel -> the tile: every instance of the kernel, one to seven
# sixteens of columns (whole, with a remainder, in several tiles), and pairs of images with one left over
TILES = {
    (32, 8, 32, (28, 28), 3): (32, 14, 1, 2), (2, 8, 17, (17, 20), 3): (32, 1, 1, 2), (9, 8, 64, (21, 33), 3): (48, 11, 1, 3),
    (3, 8, 129, (1, 98), 3): (64, 1, 1, 4), (9, 8, 129, (4, 70), 3): (80, 4, 1, 5), (16, 8, 129, (1, 86), 3): (96, 1, 1, 6),
    (8, 8, 161, (7, 6), 3): (8, 3, 2, 1), (2, 8, 8, (19, 1), 3): (8, 1, 2, 1),
    (32, 16, 32, (28, 28), 3): (32, 14, 1, 2), (9, 16, 129, (3, 33), 3): (48, 3, 1, 3), (2, 16, 129, (2, 102), 3): (64, 2, 1, 4),
    (9, 16, 33, (16, 66), 3): (80, 4, 1, 5), (32, 16, 33, (1, 85), 3): (96, 1, 1, 6), (8, 16, 129, (1, 112), 3): (112, 1, 1, 7),
    (4, 16, 81, (9, 8), 3): (8, 1, 2, 1), (8, 16, 321, (7, 7), 3): (8, 7, 2, 1),
    (8, 8, 161, (7, 5), 5): (8, 3, 2, 1), (3, 8, 64, (1, 96), 5): (32, 1, 1, 2), (4, 8, 129, (2, 114), 5): (64, 2, 1, 4),
    (32, 8, 129, (2, 100), 5): (112, 2, 1, 7), (4, 16, 201, (7, 7), 5): (8, 4, 2, 1), (3, 16, 64, (1, 106), 5): (32, 1, 1, 2),
    (8, 16, 64, (1, 70), 5): (48, 1, 1, 3), (32, 16, 17, (1, 100), 5): (64, 1, 1, 4),
}


def _tensors(p, seed):
    """Small integers on the device, in its layouts, and views of them as torch's functions take them."""
    import torch
    g, c, k = p.groups, p.in_chans_per_group, p.kernel[0]
    torch.manual_seed(seed)
    ints = lambda *s: torch.randint(-2, 3, s, device="cuda").half()
    x, w = ints(p.batch, p.field[0], p.field[1], g * c), ints(g, k, k, c, c)
    dy = ints(p.batch, *p.output_field(), g * c)
    torch.cuda.synchronize()
    return x, w, dy, lambda t: t.permute(0, 3, 1, 2).double(), lambda t: t.permute(0, 3, 4, 1, 2).reshape(g * c, c, k, k).double()


@pytest.mark.parametrize("layer", TILES)
def test_rows_of_every_tile(gpu_ctx, layer):
    """Exact sums of integers, and again with an infinite weight: it meets the pixels that its tap
    reaches, and no padding."""
    import torch
    g, c, n, field, k = layer
    p = capi.ConvParams.make(n, list(field), [k, k], c, c, groups=g, padding=k // 2)
    assert _tile(p) == TILES[layer] and capi.conv_plan(p).in_place and capi.conv_plan(p, capi.PASS_TRAINING_BWD).in_place
    x, w, dy, nchw, weights = _tensors(p, c + k)
    y, dx = torch.full_like(dy, 7), torch.full_like(x, 7)
    conv, back = torch.nn.functional.conv2d, torch.nn.functional.conv_transpose2d

    def run():
        torch.cuda.synchronize()
        gpu_ctx.conv_fwd(p, x, w, y)
        gpu_ctx.conv_bwd(p, dy, w, dx)
        gpu_ctx.synchronize()

    run()
    assert torch.equal(nchw(y), conv(nchw(x), weights(w), padding=k // 2, groups=g))
    assert torch.equal(nchw(dx), back(nchw(dy), weights(w), padding=k // 2, groups=g))
    x.abs_().add_(1), dy.abs_().add_(1)
    group, co, ci = g - 1, c - 1, c - 3
    w[group, 0, 0, co, ci] = np.inf
    run()
    pad, inf = k // 2, torch.zeros_like(y, dtype=torch.bool)
    inf[:, pad:, pad:, group * c + co] = True
    assert torch.equal(torch.isfinite(y), ~inf)
    inf = torch.zeros_like(inf)
    inf[:, :field[0] - pad, :field[1] - pad, group * c + ci] = True
    assert torch.equal(torch.isfinite(dx), ~inf)
    w[group, 0, 0, co, ci] = 0
    assert torch.equal(nchw(y)[:, :group * c], conv(nchw(x), weights(w), padding=pad, groups=g)[:, :group * c].half().double())


# (two images, and one to seven sixteens of columns)
WU_TILES = {
    (2, 8, 5, (4, 1), 3): (8, 2), (4, 8, 64, (1, 38), 3): (32, 1), (2, 8, 64, (3, 76), 3): (48, 1), (3, 8, 129, (1, 55), 3): (64, 1),
    (2, 8, 33, (15, 70), 3): (80, 1), (16, 8, 129, (1, 86), 3): (96, 1), (3, 8, 129, (1, 98), 3): (112, 1),
    (2, 16, 5, (1, 6), 3): (8, 2), (8, 16, 321, (7, 7), 3): (8, 2), (2, 16, 33, (1, 87), 3): (32, 1), (2, 16, 64, (1, 83), 3): (48, 1),
    (3, 16, 129, (1, 64), 3): (64, 1), (16, 16, 33, (1, 67), 3): (80, 1), (4, 16, 129, (1, 84), 3): (96, 1), (4, 16, 129, (1, 107), 3): (112, 1),
    (2, 8, 2, (10, 1), 5): (8, 2), (3, 8, 33, (1, 77), 5): (32, 1), (3, 8, 64, (1, 96), 5): (48, 1), (2, 8, 64, (2, 124), 5): (64, 1),
    (4, 8, 129, (1, 70), 5): (80, 1), (2, 8, 129, (1, 96), 5): (96, 1),
}


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("layer", WU_TILES)
def test_rows_weight_gradient_of_every_tile(gpu_ctx, layer, offset):
    """Also to gradients that start inside a vector."""
    import torch
    g, c, n, field, k = layer
    p = capi.ConvParams.make(n, list(field), [k, k], c, c, groups=g, padding=k // 2)
    plan = capi.conv_wu_plan(p)
    assert (plan.kernel, (plan.box_w, plan.box_n)) == (3, WU_TILES[layer])
    x, w, dy, nchw, weights = _tensors(p, c + k)
    half, single = (torch.full((w.numel() + 1,), 7, device="cuda", dtype=t) for t in (torch.float16, torch.float32))
    torch.cuda.synchronize()
    gpu_ctx.conv_wu(p, x, dy, half[offset:], single[offset:])
    gpu_ctx.synchronize()
    want = torch.nn.grad.conv2d_weight(nchw(x), (g * c, c, k, k), nchw(dy), padding=k // 2, groups=g)
    for got in (half, single):
        assert torch.equal(weights(got[offset:offset + w.numel()].view(w.shape)), want.to(got.dtype).double())
        assert got[0 if offset else -1] == 7


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("pixel", [(0, 0), (0, -1), (-1, -1), (5, 3)])
@pytest.mark.parametrize("name", ["28 columns", "two images a step", "16 channels, 30 columns", "5x5"])
def test_rows_weight_gradient_of_infinite_gradients(gpu_ctx, name, pixel, value):
    """As in the contraction: its output channel's sums become infinite, or NaN where the tap meets
    padding from that pixel, and no others."""
    p = _layer(name)
    x, _, dy = _data(p, T.rng(4))
    x = np.abs(x) + 1
    group, channel = p.groups - 1, 2
    dy[1, group * p.out_chans_per_group + channel, pixel[0], pixel[1]] = value
    got, general = (T.gpu_conv_wu(p, x, dy, opt=capi.ConvOptions.make(split_k=s))[1] for s in (0, 1))
    assert capi.conv_wu_plan(p).kernel == 3 and capi.conv_wu_plan(p, capi.ConvOptions.make(split_k=1)).kernel == 1
    assert (np.isnan(got) == np.isnan(general)).all() and (np.isinf(got) == np.isinf(general)).all()
    hit = np.zeros(got.shape, dtype=bool)
    hit[group, channel] = True
    assert (np.isfinite(got) == ~hit).all()


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
