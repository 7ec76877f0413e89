"""Per-channel sums and maps at the channel counts where their walk changes: a
row that is a fraction of, exactly, or several vectors; vectors that straddle
rows (odd counts: up to 8 rows per super-row, with 0 to 7 rows left over); one
or several column blocks; a base that is not 16-byte aligned.  Integer data:
every sum is exact in fp32 (|sum| <= 4 * 1237 * 4 < 2^24) and every mapped value
is exact in half (|x + b| <= 8), so results must match bit for bit."""
import numpy as np
import pytest

import common as T
from poplibs_b200 import capi

pytestmark = pytest.mark.gpu

CHANS = [1, 2, 3, 7, 8, 12, 20, 31, 64, 100, 136, 257, 264, 567, 1024, 2056]
ROWS = [1, 5, 64, 1237]


@pytest.mark.parametrize("dtype", ["half", "float"])
@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("chans", CHANS)
def test_channel_sums_and_maps(gpu_ctx, chans, rows, dtype):
    import torch
    ctx = T.context()
    np_t, plb_t = (np.float16, capi.HALF) if dtype == "half" else (np.float32, capi.FLOAT)
    r = T.rng(chans * 31 + rows)
    for offset in (0, 1):
        x = r.integers(-4, 5, (rows, chans)).astype(np_t)
        y = r.integers(-4, 5, (rows, chans)).astype(np_t)
        b = r.integers(-4, 5, chans).astype(np_t)
        # `offset` elements into an allocation: 2 or 4 bytes off the alignment
        def dev(a):
            t = torch.empty(a.size + offset, dtype=torch.from_numpy(a).dtype, device="cuda")
            t[offset:].copy_(torch.from_numpy(a.reshape(-1)))
            return t[offset:]
        dx, dy, db = dev(x), dev(y), dev(b)
        bias = torch.full((chans,), 3.0, device="cuda")
        ga, be = T.empty_dev([chans], np.float32), T.empty_dev([chans], np.float32)
        torch.cuda.synchronize()
        ctx.conv_bias_update(plb_t, dx, rows, chans, capi.FLOAT, bias, 0.5)
        ctx.norm_param_gradients(plb_t, dx, dy, rows, chans, 1.0, None, None, ga, be)
        capi._check(capi.lib().plb_add_bias(ctx.handle, plb_t, dy.data_ptr(), db.data_ptr(), rows, chans))
        ctx.synchronize()
        x64, y64 = x.astype(np.float64), y.astype(np.float64)
        np.testing.assert_array_equal(bias.cpu().numpy(), 3.0 + 0.5 * x64.sum(axis=0))
        np.testing.assert_array_equal(ga.cpu().numpy(), (x64 * y64).sum(axis=0))
        np.testing.assert_array_equal(be.cpu().numpy(), y64.sum(axis=0))
        np.testing.assert_array_equal(dy.cpu().numpy().reshape(rows, chans), y + b)


@pytest.mark.parametrize("dtype", ["half", "float"])
@pytest.mark.parametrize("rows", [8192, 8193, 24576, 24577])
@pytest.mark.parametrize("chans", [1, 7, 8, 64, 100, 257])
def test_sums_and_maps_where_their_route_changes(gpu_ctx, chans, rows, dtype):
    """One or two launches for the sums (by rows, for whole vectors and others), one or several
    rows per thread for the maps.  |sum| <= 24577 * 16 < 2^24."""
    import torch
    ctx = T.context()
    t_t, plb_t = (torch.float16, capi.HALF) if dtype == "half" else (torch.float32, capi.FLOAT)
    g = torch.Generator(device="cuda").manual_seed(chans + rows)
    ints = lambda *s: torch.randint(-4, 5, s, device="cuda", generator=g).to(t_t)
    x, y, a, b = ints(rows, chans), ints(rows, chans), ints(chans), ints(chans)
    bias, power = torch.full((chans,), 3.0, device="cuda"), torch.empty(chans, device="cuda")
    ga, be = torch.empty(chans, device="cuda"), torch.empty(chans, device="cuda")
    out, white, norm, grad = (torch.empty_like(x) for _ in range(4))
    one = torch.ones_like(a)
    torch.cuda.synchronize()
    ctx.conv_bias_update(plb_t, x, rows, chans, capi.FLOAT, bias, 0.5)
    ctx.norm_moments(plb_t, x, rows, chans, 1.0, None, torch.empty_like(a), power)
    ctx.norm_param_gradients(plb_t, x, y, rows, chans, 1.0, None, None, ga, be)
    ctx.norm_scale_shift(plb_t, x, a, b, rows, chans, out)
    ctx.norm_normalise(plb_t, x, a, one, b, one, rows, chans, white, norm)
    ctx.norm_statistics_gradients(plb_t, x, y, one, rows, chans, grad, var_delta=a, mean_delta=b)
    ctx.synchronize()
    x64, y64, a64, b64 = x.double(), y.double(), a.double(), b.double()
    assert torch.equal(bias.double(), 3.0 + 0.5 * x64.sum(0))
    assert torch.equal(power.double(), (x64 * x64).sum(0))
    assert torch.equal(ga.double(), (x64 * y64).sum(0)) and torch.equal(be.double(), y64.sum(0))
    assert torch.equal(out.double(), x64 * a64 + b64)
    assert torch.equal(white.double(), x64 - a64) and torch.equal(norm.double(), (x64 - a64) * b64 + 1)
    assert torch.equal(grad.double(), y64 + x64 * a64 + b64)


@pytest.mark.parametrize("count", [1, 7, 8, 9, 2047, 2048 * 8 * 148 + 13])
@pytest.mark.parametrize("dtype", ["half", "float"])
def test_scaled_add_and_cast_tails(gpu_ctx, dtype, count):
    """Whole vectors, the tail after them and a second pass of the grid."""
    import torch
    ctx = T.context()
    t_t, plb_t = (torch.float16, capi.HALF) if dtype == "half" else (torch.float32, capi.FLOAT)
    for offset in (0, 1):
        w = torch.randint(-8, 9, (count + offset,), device="cuda").to(t_t)[offset:]
        d = torch.randint(-8, 9, (count + offset,), device="cuda").float()[offset:]
        want, cast = (w.float() + 0.5 * d).to(t_t), torch.empty(count + offset, dtype=t_t, device="cuda")[offset:]
        torch.cuda.synchronize()
        ctx.scaled_add_to(plb_t, w, d, 0.5, count)
        ctx.cast_from_f32(plb_t, cast, d, count)
        ctx.synchronize()
        assert torch.equal(w, want) and torch.equal(cast, d.to(t_t))
