"""Channel sums of few rows in one launch of clusters (poplibs_b200/csrc/channel_ops.cuh), against
float64: one block and several, rows that end inside a batch, a block and a cluster, columns that end
inside a block, and the sizes from which the other forms take over, by rows and by columns.
"""
import numpy as np
import pytest

import common as T
from poplibs_b200 import capi

pytestmark = pytest.mark.gpu

ROWS = [1, 31, 64, 255, 256, 257, 1000, 2049, 4096, 4097, 6144, 6145, 12544]
CHANS = [8, 36, 64, 72, 200, 512, 520]


@pytest.mark.parametrize("dtype", ["half", "float"])
@pytest.mark.parametrize("chans", CHANS)
@pytest.mark.parametrize("rows", ROWS)
def test_sums(gpu_ctx, rows, chans, dtype):
    import torch
    plb, np_type = (capi.HALF, np.float16) if dtype == "half" else (capi.FLOAT, np.float32)
    r = T.rng(rows + chans)
    x, y = (r.uniform(-1, 1, (rows, chans)).astype(np_type) for _ in range(2))
    bias = r.uniform(-1, 1, chans).astype(np.float32)
    dx, dy, db = T.to_dev(x), T.to_dev(y), T.to_dev(bias)
    gamma, beta = T.empty_dev((chans,), np.float32), T.empty_dev((chans,), np.float32)
    mean, inv_std = T.empty_dev((chans,), np_type), T.empty_dev((chans,), np_type)
    torch.cuda.synchronize()
    before = gpu_ctx.launch_count()
    gpu_ctx.conv_bias_update(plb, dx, rows, chans, capi.FLOAT, db, -0.5)
    small = rows <= (4095 if chans <= 16 else 6144 if chans <= 64 else 8192 if chans <= 128 else 12544) and chans % (8 if dtype == "half" else 4) == 0
    assert not small or gpu_ctx.launch_count() == before + 1
    gpu_ctx.norm_param_gradients(plb, dx, dy, rows, chans, 1.0, None, None, gamma, beta)
    gpu_ctx.norm_statistics(plb, dx, rows, chans, 1e-3, 1.0, mean, inv_std)
    gpu_ctx.synchronize()
    x64, y64 = x.astype(np.float64), y.astype(np.float64)
    # fp32 sums of up to 12544 terms below 1, in chains of 25 a thread and trees: 2^-24 of the sum of
    # magnitudes for each of some 40 additions
    bound = 40 * 2.0 ** -24 * rows
    assert np.abs(db.cpu().numpy() - (bias - 0.5 * x64.sum(0))).max() <= bound + 1e-6
    assert np.abs(gamma.cpu().numpy() - (x64 * y64).sum(0)).max() <= bound
    assert np.abs(beta.cpu().numpy() - y64.sum(0)).max() <= bound
    m, v = x64.mean(0), (x64 ** 2).mean(0)
    # one rounding to the type; the variance from a mean that has been rounded
    eps = 2.0 ** -11 if dtype == "half" else 2.0 ** -22
    assert np.abs(mean.cpu().numpy() - m).max() <= eps
    want = 1 / np.sqrt(np.maximum(v - m * m, 0) + 1e-3)
    slack = (2 * eps + 40 * 2.0 ** -24) * want ** 3 + 2 * eps * want
    assert (np.abs(inv_std.cpu().numpy() - want) <= slack).all()


# rows of more than 768 columns: one block to a column and clusters (one launch), and where those would
# come in many waves, two short launches or slabs
WIDE = [("half", 256, 16384, 1), ("half", 257, 16384, 2), ("half", 1024, 3064, 1), ("half", 1024, 3072, 2), ("float", 1024, 1536, 2),
        ("float", 1024, 4096, 2), ("half", 2560, 3072, 2), ("half", 2561, 3072, 1), ("half", 4096, 3072, 1), ("float", 2600, 1000, 1),
        ("half", 2048, 8192, 1), ("float", 128, 20000, 1)]


@pytest.mark.parametrize("dtype,rows,chans,launches", WIDE)
def test_wide_sums(gpu_ctx, dtype, rows, chans, launches):
    import torch
    plb, torch_type = (capi.HALF, torch.float16) if dtype == "half" else (capi.FLOAT, torch.float32)
    g = torch.Generator(device="cuda").manual_seed(rows + chans)
    x, y = ((torch.rand(rows, chans, device="cuda", generator=g) * 2 - 1).to(torch_type) for _ in range(2))
    bias = torch.zeros(chans, device="cuda")
    gamma, beta = torch.empty_like(bias), torch.empty_like(bias)
    torch.cuda.synchronize()
    before = gpu_ctx.launch_count()
    gpu_ctx.conv_bias_update(plb, x, rows, chans, capi.FLOAT, bias, -0.5)
    assert gpu_ctx.launch_count() == before + launches
    gpu_ctx.norm_param_gradients(plb, x, y, rows, chans, 1.0, None, None, gamma, beta)
    gpu_ctx.synchronize()
    bound = 40 * 2.0 ** -24 * rows  # (as above)
    assert (bias.double() + 0.5 * x.double().sum(0)).abs().max() <= bound
    assert (gamma.double() - (x.double() * y.double()).sum(0)).abs().max() <= bound
    assert (beta.double() - y.double().sum(0)).abs().max() <= bound
