"""Small products on the kernel that reads its operands where they lie, from any address
and at any pitch (poplibs_b200/csrc/direct.cuh), against the oracle and against the
general route, which a context with a plan flag takes.

Small-integer data are exact in every operand type and in fp32 sums: bit for bit.
"""
import numpy as np
import pytest

import common as T
import oracle
from poplibs_b200 import capi

pytestmark = pytest.mark.gpu

TYPES = {"half": (capi.HALF, np.float16, capi.HALF, np.float16), "float": (capi.FLOAT, np.float32, capi.FLOAT, np.float32),
         "quarter": (capi.QUARTER, np.uint8, capi.HALF, np.float16)}
# remainders of the 64, 128 and 256 long K steps, one row, one column, one product; some types
# and layouts of the larger ones take the general route
SIZES = [(1, 1, 1, 1), (1, 16, 256, 32), (1, 17, 257, 33), (1, 15, 511, 31), (1, 33, 128, 64), (1, 31, 129, 65),
         (1, 132, 98, 181), (1, 64, 385, 7), (1, 65, 63, 129), (1, 300, 40, 280), (3, 47, 155, 85), (5, 112, 32, 48),
         (20, 33, 65, 17), (40, 64, 40, 64), (1, 16, 1030, 512), (2, 128, 576, 64), (1, 5, 3, 700)]
# products that are direct in every layout: together they take every block (16 x 32, 32 x 32,
# 32 x 64 and 64 x 64, with one or two teams of warps) that the planner chooses for the type
DIRECT = {
    "half": [(1, 8, 8, 8), (3, 280, 13, 261), (1, 4, 314, 5), (6, 40, 8, 288), (6, 197, 9, 296), (6, 196, 10, 395),
             (6, 275, 160, 72), (6, 80, 96, 272)],
    "float": [(1, 8, 8, 8), (2, 4, 280, 4), (6, 200, 8, 152), (6, 280, 8, 200), (6, 288, 16, 352)],
    "quarter": [(1, 4, 21, 8), (3, 5, 213, 5), (1, 7, 389, 11), (6, 175, 15, 299), (2, 228, 147, 293), (1, 8, 25, 8),
                (2, 8, 329, 8), (3, 8, 181, 40)],
}


@pytest.fixture(scope="module")
def general_ctx():
    ctx = capi.Context(0)
    ctx.set_plan_flags(capi.PLAN_NO_DUAL_ISSUE)
    return ctx


def _operand(values, dtype, offset, pitch):
    """[g][rows][cols] with rows `pitch` elements apart, `offset` elements into an allocation."""
    import torch
    g, rows, cols = values.shape
    flat = np.zeros(offset + g * rows * pitch, np.float64)
    flat[offset:].reshape(g, rows, pitch)[:, :, :cols] = values
    flat = oracle.e4m3_encode(flat) if dtype == np.uint8 else flat.astype(dtype)
    return torch.from_numpy(flat).cuda(), offset * flat.itemsize


def _run(ctx, desc, a, b, c, shape, out_dtype, ldc, offset):
    import torch
    g, m, n = shape
    d = T.empty_dev((offset + g * m * ldc,), out_dtype)
    torch.cuda.synchronize()
    ctx.matmul(desc, a[0].data_ptr() + a[1], b[0].data_ptr() + b[1], c and c[0].data_ptr() + c[1],
               d.data_ptr() + offset * d.element_size())
    ctx.synchronize()
    out = d.cpu().numpy()
    rows = out[offset:].reshape(g, m, ldc)
    # what lies before and between the rows is not written
    bits = out.view(f"u{out.itemsize}")
    poison = int.from_bytes(b"\x7d" * out.itemsize, "little")
    assert (bits[:offset] == poison).all() and (bits[offset:].reshape(g, m, ldc)[:, :, n:] == poison).all()
    return rows[:, :, :n].astype(np.float64)


@pytest.mark.parametrize("pad,offset", [(0, 0), (3, 1), (8, 16)])
@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("tb", [False, True])
@pytest.mark.parametrize("dtype", sorted(TYPES))
def test_small_products(gpu_ctx, general_ctx, dtype, ta, tb, pad, offset):
    plb_in, np_in, plb_out, np_out = TYPES[dtype]
    if dtype == "quarter" and (ta or not tb) and pad:
        pytest.skip("refused: transposed quarter operands are densely packed")
    # (floats from any address take three of the shapes)
    whole = [(20, 8, 168, 232)] if dtype == "float" and pad != 3 else []
    for g, m, k, n in SIZES + DIRECT[dtype] + whole:
        r = T.rng(m + 7 * k + n)
        av, bv = (r.integers(-2, 3, s).astype(np.float64) for s in ((g, m, k), (g, k, n)))
        want = av @ bv
        assert np.abs(want).max() <= 2048  # exact in half
        sa, sb = (av.transpose(0, 2, 1) if ta else av), (bv.transpose(0, 2, 1) if tb else bv)
        lda, ldb, ldc = sa.shape[2] + pad, sb.shape[2] + pad, n + pad
        a, b = _operand(sa, np_in, offset, lda), _operand(sb, np_in, offset, ldb)
        desc = capi.MatmulDesc.make(m, k, n, groups=g, input_type=plb_in, output_type=plb_out, transpose_a=ta,
                                    transpose_b=tb)
        desc.lda, desc.ldb, desc.ldc = lda, ldb, ldc
        assert capi.matmul_plan(desc).kernel == 3 or (g, m, k, n) in SIZES
        got = _run(gpu_ctx, desc, a, b, None, (g, m, n), np_out, ldc, offset)
        general = _run(general_ctx, desc, a, b, None, (g, m, n), np_out, ldc, offset)
        assert (got == general).all(), (g, m, k, n)
        assert (got == want).all(), (g, m, k, n)


@pytest.mark.parametrize("out", [capi.HALF, capi.FLOAT])
@pytest.mark.parametrize("n", [7, 45, 250])
def test_nothing_is_written_between_rows_of_whole_vectors(gpu_ctx, general_ctx, n, out):
    """Rows of results that start on 16 bytes and end between: a column slice of a wider matrix."""
    m, k, ldc = 150, 64, (n + 7) // 8 * 8
    r = T.rng(n)
    av, bv = (r.integers(-2, 3, s).astype(np.float64) for s in ((2, m, k), (2, k, n)))
    desc = capi.MatmulDesc.make(m, k, n, groups=2, output_type=out)
    desc.ldc = ldc
    a, b = _operand(av, np.float16, 0, k), _operand(bv, np.float16, 0, n)
    for ctx in (gpu_ctx, general_ctx):
        got = _run(ctx, desc, a, b, None, (2, m, n), np.float32 if out == capi.FLOAT else np.float16, ldc, 0)
        assert (got == av @ bv).all()


@pytest.mark.parametrize("out", [capi.HALF, capi.FLOAT])
@pytest.mark.parametrize("n", [48, 45])
def test_scaled_and_added(gpu_ctx, n, out):
    g, m, k = 3, 37, 70
    r = T.rng(n)
    av, bv, cv = (r.integers(-2, 3, s).astype(np.float64) for s in ((g, m, k), (g, k, n), (g, m, n)))
    desc = capi.MatmulDesc.make(m, k, n, groups=g, output_type=out, alpha=2.0, beta=-3.0)
    dt = np.float32 if out == capi.FLOAT else np.float16
    a, b, c = _operand(av, np.float16, 0, k), _operand(bv, np.float16, 0, n), _operand(cv, dt, 0, n)
    got = _run(gpu_ctx, desc, a, b, c, (g, m, n), dt, n, 0)
    assert (got == 2 * (av @ bv) - 3 * cv).all()


def test_impossible_pitches_are_refused(gpu_ctx):
    import torch
    x = torch.zeros(16 * 512, dtype=torch.float16, device="cuda")
    for field in ("lda", "ldb"):
        d = capi.MatmulDesc.make(16, 512, 16, transpose_b=True)
        setattr(d, field, -512)
        with pytest.raises(capi.PlbError):
            gpu_ctx.matmul(d, x, x, None, x)


def test_ragged_products_take_one_launch(gpu_ctx):
    r = T.rng(3)
    for dtype, n in ((np.float16, 181), (np.float32, 64), (np.float32, 61)):
        a, b = r.integers(-2, 3, (132, 98)).astype(dtype), r.integers(-2, 3, (98, n)).astype(dtype)
        before = gpu_ctx.launch_count()
        T.gpu_matmul(a, b, out_dtype=dtype, ctx=gpu_ctx)
        assert gpu_ctx.launch_count() == before + 1


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("k", [72, 71])
def test_float_infinities(gpu_ctx, k, value):
    """An infinity or NaN meets its row's and column's products alone, and makes no NaN of
    an infinity (the other operand's low pieces are zero here)."""
    r = T.rng(k)
    a, b = r.integers(1, 4, (40, k)).astype(np.float32), r.integers(1, 4, (k, 48)).astype(np.float32)
    a[7, 50] = value
    b[k - 1, 9] = value
    with np.errstate(invalid="ignore"):
        want = a.astype(np.float64) @ b.astype(np.float64)
    got = T.gpu_matmul(a, b, out_dtype=np.float32, ctx=gpu_ctx)
    assert np.array_equal(got.astype(np.float64), want, equal_nan=True)


def test_float_products_keep_their_precision(gpu_ctx, general_ctx):
    """Three terms per product either way: no further from 64 bits than the general route
    (within the noise of sums in another order)."""
    for m, k, n in ((128, 576, 64), (33, 700, 90)):
        r = T.rng(m)
        a, b = r.uniform(-1, 1, (m, k)).astype(np.float32), r.uniform(-1, 1, (k, n)).astype(np.float32)
        want = a.astype(np.float64) @ b.astype(np.float64)
        off = [np.linalg.norm(T.gpu_matmul(a, b, out_dtype=np.float32, ctx=c) - want) / np.linalg.norm(want)
               for c in (gpu_ctx, general_ctx)]
        assert off[0] <= 1.1 * off[1] and off[0] < 2.0 ** -16, off
