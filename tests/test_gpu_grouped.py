"""Grouped contractions, operands with ragged rows and few-channel layers, at the
sizes where the route changes: groups that fill a fraction of, exactly or more
than one 128-byte operand row; group counts whose dense blocks divide them or
not; channel counts that start a block on a 16-byte boundary only every second,
fourth or eighth group, or never; first layers of 1 to 7 channels.  Small
integer data: sums are exact in fp32 and, below 2^11, in half, so the CPU oracle's
results must come back bit for bit."""
import numpy as np
import pytest

import common as T
import oracle
from poplibs_b200 import capi

pytestmark = pytest.mark.gpu


def exact(got, want, what):
    got = np.asarray(got, dtype=np.float64)
    want = np.asarray(want, dtype=np.float64).reshape(got.shape)
    assert np.array_equal(got, want), f"{what}: {int((got != want).sum())} of {got.size} differ"


def ints(r, shape, dtype):
    return r.integers(-1, 2, shape).astype(dtype)


# groups, channels in and out per group
GROUPS = [(32, 8, 8), (32, 4, 4), (16, 5, 5), (6, 10, 6), (7, 9, 3), (2, 32, 32), (4, 16, 24), (3, 64, 64), (5, 48, 16),
          (64, 1, 1), (9, 1, 2), (8, 12, 20), (2, 136, 40), (3, 33, 17)]


@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("groups,ci,co", GROUPS)
def test_grouped_convolution(gpu_ctx, groups, ci, co, stride):
    kw = dict(batch=3, field=[9, 7], kernel=[3, 3], in_chans=ci, out_chans=co, groups=groups, padding=1, stride=stride)
    r = T.rng(groups * 100 + ci + co)
    for dtype, plb in ((np.float16, capi.HALF), (np.float32, capi.FLOAT)):
        p = capi.ConvParams.make(input_type=plb, output_type=plb, **kw)
        spec = T.spec_from_params(p)
        x = ints(r, (3, groups * ci, 9, 7), dtype)
        w = ints(r, (groups, co, ci, 3, 3), dtype)
        dy = ints(r, (3, groups * co, *p.output_field()), dtype)
        bias = r.integers(-3, 4, groups * co).astype(np.float32)
        exact(T.gpu_conv_fwd(p, x, w, bias=bias), oracle.conv_fwd(spec, x, w, bias), f"fwd {dtype}")
        exact(T.gpu_conv_bwd(p, dy, w), oracle.conv_bwd(spec, dy, w), f"bwd {dtype}")
        exact(T.gpu_conv_wu(p, x, dy)[1], oracle.conv_wu(spec, x, dy)[0], f"wu {dtype}")


@pytest.mark.parametrize("split", [0, 3])
@pytest.mark.parametrize("variant", ["resident", "pair", "halo", "halo pair"])
@pytest.mark.parametrize("kernel,chans", [((3, 3), 64), ((3, 8), 56)])
def test_resident_weights_with_groups_and_splits(gpu_ctx, kernel, chans, variant, split):
    """Residency that is asked for, with groups and with splits that are forced or (24 steps
    over rows at odd multiples of 16 bytes) the planner's own."""
    flags = (capi.PLAN_FORCE_RESIDENT_WEIGHTS | (capi.PLAN_FORCE_CTA_PAIR if "pair" in variant else 0) |
             (0 if "halo" in variant else capi.PLAN_NO_HALO))
    for groups in (1, 3):
        kw = dict(batch=2, field=[12, 12], kernel=list(kernel), in_chans=chans, out_chans=chans, groups=groups, padding=1)
        p, opt = capi.ConvParams.make(**kw), capi.ConvOptions.make(plan_flags=flags, split_k=split)
        spec = T.spec_from_params(p)
        r = T.rng(groups)
        x, w = ints(r, (2, groups * chans, 12, 12), np.float16), ints(r, (groups, chans, chans, *kernel), np.float16)
        exact(T.gpu_conv_fwd(p, x, w, opt=opt), oracle.conv_fwd(spec, x, w), f"fwd groups {groups}")


@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("groups,ci,co", [(32, 8, 8), (6, 10, 6)])
def test_infinities_stay_in_their_group(gpu_ctx, groups, ci, co, value, stride):
    """A non-finite element changes the outputs of its own group alone, although
    neighbouring groups are contracted together."""
    p = capi.ConvParams.make(batch=2, field=[8, 6], kernel=[3, 3], in_chans=ci, out_chans=co, groups=groups, padding=1,
                             stride=stride)
    r = T.rng(5)
    x = ints(r, (2, groups * ci, 8, 6), np.float16)
    w = ints(r, (groups, co, ci, 3, 3), np.float16)
    w[w == 0] = 1  # every product with the element is non-finite
    dy = ints(r, (2, groups * co, *p.output_field()), np.float16)
    y, dx = T.gpu_conv_fwd(p, x, w), T.gpu_conv_bwd(p, dy, w)
    g = groups // 2
    x2, dy2 = x.copy(), dy.copy()
    x2[1, g * ci + 1, 4, 2] = value
    dy2[1, g * co + 1, 2, 2] = value
    for got, was, c in ((T.gpu_conv_fwd(p, x2, w), y, co), (T.gpu_conv_bwd(p, dy2, w), dx, ci)):
        mine = slice(g * c, (g + 1) * c)
        assert not np.isfinite(got[1, mine]).all()
        same = np.isfinite(got[1, mine])
        exact(got[1, mine][same], was[1, mine][same], "own group, elements the value does not reach")
        got = got.copy()
        got[1, mine] = was[1, mine]
        exact(got, was, "other groups")
    # and the next call is unaffected
    exact(T.gpu_conv_fwd(p, x, w), y, "after")


PLAN_VARIANTS = {
    "streamed": capi.PLAN_NO_RESIDENT_WEIGHTS,
    "streamed no halo": capi.PLAN_NO_RESIDENT_WEIGHTS | capi.PLAN_NO_HALO,
    "streamed pair": capi.PLAN_NO_RESIDENT_WEIGHTS | capi.PLAN_FORCE_CTA_PAIR,
    "streamed no halo pair": capi.PLAN_NO_RESIDENT_WEIGHTS | capi.PLAN_NO_HALO | capi.PLAN_FORCE_CTA_PAIR,
    "resident": capi.PLAN_FORCE_RESIDENT_WEIGHTS | capi.PLAN_NO_HALO,
    "resident halo": capi.PLAN_FORCE_RESIDENT_WEIGHTS,
    "resident pair": capi.PLAN_FORCE_RESIDENT_WEIGHTS | capi.PLAN_NO_HALO | capi.PLAN_FORCE_CTA_PAIR,
    "resident halo pair": capi.PLAN_FORCE_RESIDENT_WEIGHTS | capi.PLAN_FORCE_CTA_PAIR,
}


@pytest.mark.parametrize("variant", sorted(PLAN_VARIANTS))
@pytest.mark.parametrize("dtype", ["half", "float", "quarter"])
@pytest.mark.parametrize("groups,ci,co", [(2, 32, 32), (3, 64, 64), (16, 8, 8), (5, 72, 40)])
def test_every_instance_with_groups(gpu_ctx, groups, ci, co, dtype, variant):
    """Each way the planner may run a grouped layer, on all operand types; (16, 8, 8) is
    contracted in blocks of neighbouring groups."""
    plb, cast, kind = {"half": (capi.HALF, lambda a: a.astype(np.float16), np.float16),
                       "float": (capi.FLOAT, lambda a: a.astype(np.float32), np.float32),
                       "quarter": (capi.QUARTER, oracle.e4m3_encode, np.float16)}[dtype]
    p = capi.ConvParams.make(batch=3, field=[13, 11], kernel=[3, 3], in_chans=ci, out_chans=co, groups=groups, padding=1,
                             input_type=plb, output_type=capi.FLOAT if dtype == "float" else capi.HALF)
    opt = capi.ConvOptions.make(plan_flags=PLAN_VARIANTS[variant])
    plan = capi.conv_plan(p, capi.PASS_TRAINING_FWD, opt)
    assert plan.cta_pair == (1 if "pair" in variant else 0)
    if "resident" in variant and dtype != "float" and ci <= 64:
        assert plan.resident_weights == 1
    spec, r = T.spec_from_params(p), T.rng(groups + ci)
    x = r.integers(-1, 2, (3, groups * ci, 13, 11)).astype(np.float64)
    w = r.integers(-1, 2, (groups, co, ci, 3, 3)).astype(np.float64)
    dy = r.integers(-1, 2, (3, groups * co, *p.output_field())).astype(np.float64)
    exact(T.gpu_conv_fwd(p, cast(x), cast(w), opt=opt), oracle.conv_fwd(spec, x, w), "fwd")
    exact(T.gpu_conv_bwd(p, cast(dy), cast(w), opt=opt), oracle.conv_bwd(spec, dy, w), "bwd")


@pytest.mark.parametrize("groups,ci,co", [(3, 64, 64), (5, 64, 32), (7, 64, 64), (32, 8, 8)])
def test_many_tiles_with_groups(gpu_ctx, groups, ci, co):
    """Layers large enough that the planner keeps weights resident and pairs CTAs by itself,
    with group counts that do not divide the number of SMs."""
    import torch
    p = capi.ConvParams.make(batch=128, field=[28, 28], kernel=[3, 3], in_chans=ci, out_chans=co, groups=groups, padding=1)
    # (a plan flag keeps narrow groups from the kernel that reads them in place)
    opt = capi.ConvOptions.make(plan_flags=capi.PLAN_NO_PDL if ci == 8 else 0)
    plan = capi.conv_plan(p, opt=opt)
    assert not plan.in_place and plan.resident_weights == 1 and plan.cta_pair == 1 and plan.tiles >= 2 * plan.grid
    ints = lambda *s: torch.randint(-1, 2, s, device="cuda").half()
    x, w, dy = ints(128, 28, 28, groups * ci), ints(groups, 3, 3, co, ci), ints(128, 28, 28, groups * co)
    y, dx = torch.empty_like(dy), torch.empty_like(x)
    torch.cuda.synchronize()
    T.context().conv_fwd(p, x, w, y, opt=opt)
    T.context().conv_bwd(p, dy, w, dx, opt=opt)
    T.context().synchronize()
    nchw = lambda t: t.permute(0, 3, 1, 2).double()
    w64 = w.permute(0, 3, 4, 1, 2).reshape(groups * co, ci, 3, 3).double()
    want = torch.nn.functional.conv2d(nchw(x), w64, padding=1, groups=groups)
    assert torch.equal(nchw(y), want)
    want = torch.nn.functional.conv_transpose2d(nchw(dy), w64, padding=1, groups=groups)
    assert torch.equal(nchw(dx), want)


@pytest.mark.parametrize("form", ["half, bias", "float", "quarter", "pointwise, stride 2", "transposed weights",
                                  "float, transposed weights", "quarter, transposed weights", "split"])
def test_infinities_stay_in_their_group_in_every_form(gpu_ctx, form):
    """Operand types, a bias, a sub-lattice, weights stored the other way, K splits: a NaN or an
    infinity reaches the outputs of its own group alone."""
    import torch
    groups, ci, co = 16, 8, 8
    plb = capi.FLOAT if "float" in form else capi.QUARTER if "quarter" in form else capi.HALF
    dtype = np.float32 if plb == capi.FLOAT else np.float16
    kernel, stride = (1, 2) if "pointwise" in form else (3, 1)
    swapped = "transposed" in form
    p = capi.ConvParams.make(batch=2, field=[8, 6], kernel=[kernel] * 2, in_chans=ci, out_chans=co, groups=groups,
                             padding=kernel // 2, stride=stride, input_type=plb,
                             output_type=capi.FLOAT if plb == capi.FLOAT else capi.HALF)
    r = T.rng(11)
    cast = oracle.e4m3_encode if plb == capi.QUARTER else lambda a: a.astype(dtype)
    x = cast(r.integers(-1, 2, (2, 8, 6, groups * ci)).astype(np.float64))
    w = cast(r.choice([-1.0, 1.0], (groups, kernel, kernel) + ((ci, co) if swapped else (co, ci))))
    bias = r.integers(-3, 4, groups * co).astype(np.float32) if "bias" in form else None
    opt = capi.ConvOptions.make(split_k=3) if form == "split" else None
    g = groups // 2 + 1

    def run(x):
        on = [T.to_dev(t) if t is not None else None for t in (x, w, bias)]
        y = T.empty_dev([2] + p.output_field() + [groups * co], dtype)
        torch.cuda.synchronize()
        T.context().convolution(p, on[0], on[1], y, on[2], opt, swapped)
        T.context().synchronize()
        return y.cpu().numpy().astype(np.float64)

    was = run(x)
    for value in (0x7F,) if plb == capi.QUARTER else (np.inf, np.nan):
        x2 = x.copy()
        x2[1, 4, 2, g * ci + 3] = value
        got, mine = run(x2), slice(g * co, (g + 1) * co)
        assert not np.isfinite(got[1, ..., mine]).all()
        same = np.isfinite(got[1, ..., mine])
        exact(got[1, ..., mine][same], was[1, ..., mine][same], "own group, elements the value does not reach")
        got[1, ..., mine] = was[1, ..., mine]
        exact(got, was, "other groups")
    exact(run(x), was, "after")


@pytest.mark.parametrize("groups,m,k,n", [(1, 197, 70, 103), (5, 197, 70, 103), (3, 8, 8, 8), (64, 33, 64, 130),
                                          (2, 1, 513, 1), (7, 129, 65, 257), (4, 300, 1100, 40)])
@pytest.mark.parametrize("dtype", ["half", "float", "quarter"])
def test_ragged_and_grouped_products(gpu_ctx, groups, m, k, n, dtype):
    """All operand layouts: rows of any length on both sides, one launch for all groups."""
    r = T.rng(m + k + n)
    av = r.integers(-1, 2, (groups, m, k)).astype(np.float64)
    bv = r.integers(-1, 2, (groups, k, n)).astype(np.float64)
    want = np.stack([av[g] @ bv[g] for g in range(groups)])
    cast = {"half": lambda v: v.astype(np.float16), "float": lambda v: v.astype(np.float32),
            "quarter": oracle.e4m3_encode}[dtype]
    out = np.float32 if dtype == "float" else np.float16
    for ta in (False, True):
        for tb in (False, True):
            a = cast(np.ascontiguousarray(av.transpose(0, 2, 1)) if ta else av)
            b = cast(np.ascontiguousarray(bv.transpose(0, 2, 1)) if tb else bv)
            exact(T.gpu_matmul(a, b, transpose_a=ta, transpose_b=tb, out_dtype=out), want, f"ta={ta} tb={tb}")
    if dtype == "half":
        c = ints(r, (groups, m, n), np.float32)
        exact(T.gpu_matmul(cast(av), cast(bv), c, alpha=2.0, beta=-1.0, out_dtype=np.float32), 2 * want - c, "alpha, beta")


@pytest.mark.parametrize("kernel,stride", [(7, 2), (3, 1), (3, 2), (1, 1), (5, 2)])
@pytest.mark.parametrize("chans", [1, 2, 3, 4, 5, 7, 12, 20])
def test_first_layer_weight_gradient(gpu_ctx, chans, kernel, stride):
    """Few input channels: the gradient from the rearranged input (where a folded
    filter row fits 64 elements) and from rounded-up channels (where it does not)."""
    for width, co in ((13, 64), (22, 24), (16, 136)):
        p = capi.ConvParams.make(batch=3, field=[11, width], kernel=[kernel, kernel], in_chans=chans, out_chans=co,
                                 padding=kernel // 2, stride=stride)
        spec = T.spec_from_params(p)
        r = T.rng(chans * 10 + kernel)
        x = ints(r, (3, chans, 11, width), np.float16)
        w = ints(r, (1, co, chans, kernel, kernel), np.float16)
        dy = ints(r, (3, co, *p.output_field()), np.float16)
        dw16, dw32 = T.gpu_conv_wu(p, x, dy)
        exact(dw32, oracle.conv_wu(spec, x, dy)[0], f"wu width {width} co {co}")
        exact(dw16, dw32.astype(np.float16), "half gradient")
        exact(T.gpu_conv_fwd(p, x, w), oracle.conv_fwd(spec, x, w), f"fwd width {width} co {co}")


@pytest.mark.parametrize("chans", [8, 3, 40])
@pytest.mark.parametrize("width,stride", [(4096, 2), (4097, 2), (8200, 3), (21846, 5)])
def test_unread_positions_of_long_rows_get_zero(gpu_ctx, width, stride, chans):
    """Rows that several blocks clear (4096 pixels of 8 channels each)."""
    p = capi.ConvParams.make(batch=2, field=[width], kernel=[1], in_chans=chans, out_chans=8, stride=stride)
    r = T.rng(width)
    w, dy = ints(r, (1, 8, chans, 1), np.float16), ints(r, (2, 8, *p.output_field()), np.float16)
    exact(T.gpu_conv_bwd(p, dy, w), oracle.conv_bwd(T.spec_from_params(p), dy, w), "bwd")


def test_unread_positions_of_a_row_beyond_2_gb(gpu_ctx):
    import torch
    width, chans = 2 ** 20 + 2, 1024
    p = capi.ConvParams.make(batch=1, field=[width], kernel=[1], in_chans=chans, out_chans=8, stride=2)
    dy = torch.randint(-1, 2, (1, width // 2, 8), device="cuda").half()
    w = torch.randint(-1, 2, (1, 1, 8, chans), device="cuda").half()
    dx = torch.full((1, width, chans), 7.0, dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    T.context().conv_bwd(p, dy, w, dx)
    T.context().synchronize()
    assert torch.equal(dx[0, ::2], dy[0] @ w[0, 0]) and not dx[0, 1::2].any()


@pytest.mark.parametrize("chans,co", [(3, 64), (1, 8), (20, 24), (16, 64)])
def test_weight_gradient_of_operands_at_any_address(gpu_ctx, chans, co):
    """Tensors that start at odd elements of an allocation."""
    import torch
    p = capi.ConvParams.make(batch=2, field=[11, 13], kernel=[3, 3], in_chans=chans, out_chans=co, padding=1, stride=2)
    r = T.rng(chans)
    x = ints(r, (2, chans, 11, 13), np.float16)
    dy = ints(r, (2, co, *p.output_field()), np.float16)
    want = oracle.conv_wu(T.spec_from_params(p), x, dy)[0]
    for off in ((1, 0), (0, 1), (3, 5)):
        on = []
        for t, o in zip((x, dy), off):
            a = T.acts_to_device_layout(t).ravel()
            buf = torch.zeros(a.size + o, dtype=torch.float16, device="cuda")
            buf[o:] = torch.from_numpy(a)
            on.append(buf[o:])
        dw = torch.empty((3, 3, co, chans), device="cuda")
        torch.cuda.synchronize()
        T.context().conv_wu(p, on[0], on[1], None, dw)
        T.context().synchronize()
        exact(T.weights_from_device_layout(dw.cpu().numpy()[None]), want, f"offsets {off}")


@pytest.mark.parametrize("elem", [1, 2, 4])
@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 130), (64, 64), (65, 63), (128, 96), (33, 257), (200, 4), (1000, 72)])
def test_transpose(gpu_ctx, elem, rows, cols):
    """Whole and partial tiles; rows that start on four-byte words on both sides, one or neither."""
    import torch
    dtype = {1: np.uint8, 2: np.uint16, 4: np.uint32}[elem]
    a = T.rng(rows + cols).integers(0, 256 ** elem, (3, rows, cols), dtype=np.uint64).astype(dtype)
    src = torch.from_numpy(a.view(np.uint8)).cuda()
    dst = torch.empty(a.nbytes, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    T.context().transpose_matrix(elem, 3, rows, cols, src, dst)
    T.context().synchronize()
    got = dst.cpu().numpy().view(dtype).reshape(3, cols, rows)
    assert np.array_equal(got, a.transpose(0, 2, 1))


@pytest.mark.parametrize("elem,rows", [(4, 65535 * 16), (4, 65535 * 16 + 1), (4, 65535 * 32), (2, 65535 * 32 + 5),
                                       (1, 65535 * 64 + 7)])
def test_transpose_of_tall_matrices(gpu_ctx, elem, rows):
    """More row tiles than one launch's grid holds."""
    import torch
    dtype = {1: torch.uint8, 2: torch.int16, 4: torch.int32}[elem]
    a = torch.randint(0, 100, (2, rows, 3), device="cuda").to(dtype)
    got = torch.empty((2, 3, rows), dtype=dtype, device="cuda")
    torch.cuda.synchronize()
    T.context().transpose_matrix(elem, 2, rows, 3, a, got)
    T.context().synchronize()
    assert torch.equal(got, a.transpose(1, 2))


@pytest.mark.parametrize("offset", [0, 1, 2])
@pytest.mark.parametrize("k", [1, 2, 5, 7, 8, 16, 21, 24, 42, 43, 130, 343])
def test_float_operands_are_split_in_place_order(gpu_ctx, k, offset):
    """Both pieces of a float at every alignment of the rows: elements +-1 + j / 1024
    (|j| <= 3) round to +-1 and leave j / 1024, so against integers every sum is exact."""
    import torch
    m, n, r = 37, 19, T.rng(k)
    fine = lambda *s: (r.choice([-1, 1], s) + r.integers(-3, 4, s) / 1024).astype(np.float32)
    whole = lambda *s: ints(r, s, np.float32)
    d = capi.MatmulDesc.make(m, k, n, transpose_b=True, input_type=capi.FLOAT, output_type=capi.FLOAT)
    for a, b in ((fine(m, k), whole(n, k)), (whole(m, k), fine(n, k))):
        on = [torch.zeros(x.size + offset, device="cuda") for x in (a, b)]
        for t, x in zip(on, (a, b)):
            t[offset:] = torch.from_numpy(x.ravel())
        out = torch.empty(m, n, device="cuda")
        torch.cuda.synchronize()
        T.context().matmul(d, on[0][offset:], on[1][offset:], None, out)
        T.context().synchronize()
        exact(out.cpu().numpy(), a.astype(np.float64) @ b.T.astype(np.float64), "split")


@pytest.mark.parametrize("groups,ci,field", [(2, 4, [13, 48]), (1, 8, [13, 48]), (1, 64, [14, 14])])
def test_short_tiles_launch_after_launch(gpu_ctx, groups, ci, field):
    """Layers whose tiles two threads issue in turn, on pipelines of few and of many stages, on
    operands that are not in L2 when the first copies are asked for."""
    import torch
    images = 171
    p = capi.ConvParams.make(batch=images, field=field, kernel=[3, 3], in_chans=ci, out_chans=ci, groups=groups, padding=1)
    r = T.rng(ci)
    w = ints(r, (groups, ci, ci, 3, 3), np.float16)
    dw = T.to_dev(T.weights_to_device_layout(w))
    xs = [ints(r, (images, groups * ci, *field), np.float16) for _ in range(2)]
    dx = [T.to_dev(T.acts_to_device_layout(x)) for x in xs]
    ys = [T.empty_dev([images, *field, groups * ci], np.float16) for _ in xs]
    flush = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")
    ctx = capi.Context(0)
    for plan_flags in (0, capi.PLAN_NO_PDL):
        ctx.set_plan_flags(plan_flags)
        for _ in range(20):
            flush.zero_()
            torch.cuda.synchronize()
            for _ in range(5):
                for x, y in zip(dx, ys):
                    ctx.conv_fwd(p, x, dw, y)
            ctx.synchronize()
    spec = T.spec_from_params(capi.ConvParams.make(batch=3, field=field, kernel=[3, 3], in_chans=ci, out_chans=ci,
                                                   groups=groups, padding=1))
    for x, y in zip(xs, ys):
        got = T.acts_from_device_layout(y[:3].cpu().numpy())
        exact(got, oracle.conv_fwd(spec, x[:3], w), "first images")
        got = T.acts_from_device_layout(y[-3:].cpu().numpy())
        exact(got, oracle.conv_fwd(spec, x[-3:], w), "last images")
