"""Calls captured into a CUDA graph by a context that has made none before: scratch memory cannot
grow then.  Where a kernel reads the operands where they lie it takes the call, however long it
takes; elsewhere the call is refused and the capture goes on."""
import numpy as np
import pytest

import common as T
from poplibs_b200 import capi

pytestmark = pytest.mark.gpu


def captured(call, out):
    """The bytes that replaying `call(ctx)`, a fresh context's first, leaves in `out`."""
    import torch
    stream = torch.cuda.Stream()
    ctx = capi.Context(0, stream=stream.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        call(ctx)
    out.view(torch.uint8).fill_(0x7D)
    graph.replay()
    torch.cuda.synchronize()
    return out.cpu().numpy()


def ints(r, shape, dtype):
    return T.to_dev(r.integers(-2, 3, shape).astype(dtype))


# few channels, narrow groups: layers that other kernels run more quickly, with scratch
@pytest.mark.parametrize("images,field,kernel,stride,groups,ci,co", [
    (1, (51, 51), 7, 2, 1, 3, 256), (42, (13, 13), 3, 1, 2, 32, 32), (8, (35, 35), 1, 1, 2, 32, 32)])
def test_layers(gpu_ctx, images, field, kernel, stride, groups, ci, co):
    p = capi.ConvParams.make(images, list(field), [kernel] * 2, ci, co, groups=groups, stride=stride, padding=kernel // 2)
    plan = capi.conv_plan(p)
    assert plan.in_place == 0 and plan.workspace_bytes > 0
    r = T.rng(ci)
    oh, ow = p.output_field()
    x, w = ints(r, (images, *field, groups * ci), np.float16), ints(r, (groups, kernel, kernel, co, ci), np.float16)
    y = T.empty_dev((images, oh, ow, groups * co), np.float16)
    got = captured(lambda ctx: ctx.conv_fwd(p, x, w, y), y)
    gpu_ctx.conv_fwd(p, x, w, y)
    gpu_ctx.synchronize()
    assert (got == y.cpu().numpy()).all()
    dx = T.empty_dev(tuple(x.shape), np.float16)
    if groups > 1 and capi.conv_plan(p, capi.PASS_TRAINING_BWD).in_place == 0:
        got = captured(lambda ctx: ctx.conv_bwd(p, y, w, dx), dx)
        gpu_ctx.conv_bwd(p, y, w, dx)
        gpu_ctx.synchronize()
        assert (got == dx.cpu().numpy()).all()


def test_ragged_float_product(gpu_ctx):
    m, k, n = 225, 1442, 59
    d = capi.MatmulDesc.make(m, k, n, input_type=capi.FLOAT, output_type=capi.FLOAT)
    assert capi.matmul_plan(d).in_place == 0
    r = T.rng(1)
    a, b, c = ints(r, (m, k), np.float32), ints(r, (k, n), np.float32), T.empty_dev((m, n), np.float32)
    got = captured(lambda ctx: ctx.matmul(d, a, b, None, c), c)
    assert (got == a.cpu().numpy().astype(np.float64) @ b.cpu().numpy().astype(np.float64)).all()


@pytest.mark.parametrize("dtype,rows,chans", [("float", 1024, 4096), ("half", 2048, 8192), ("half", 5000, 8)])
def test_channel_sums_of_few_rows(gpu_ctx, dtype, rows, chans):
    """Sums that other forms make more quickly, with scratch."""
    plb, np_type = (capi.HALF, np.float16) if dtype == "half" else (capi.FLOAT, np.float32)
    x = ints(T.rng(3), (rows, chans), np_type)
    beta, gamma = T.empty_dev((chans,), np.float32), T.empty_dev((chans,), np.float32)
    got = captured(lambda ctx: ctx.norm_param_gradients(plb, x, x, rows, chans, 1.0, None, None, gamma, beta), beta)
    want = x.cpu().numpy().astype(np.float64)
    assert (got == want.sum(0)).all() and (gamma.cpu().numpy() == (want * want).sum(0)).all()


def test_refused_calls_leave_the_capture(gpu_ctx):
    """A layer that needs copies of its operands, and a call that needs nothing in the same graph."""
    ragged = capi.ConvParams.make(4, [33, 29], [3, 3], 20, 36, padding=1)
    whole = capi.ConvParams.make(1, [14, 14], [3, 3], 32, 32, padding=1)
    assert capi.conv_plan(ragged).workspace_bytes > 0 and capi.conv_plan(whole).workspace_bytes == 0
    r = T.rng(2)
    x, w, y = ints(r, (1, 14, 14, 32), np.float16), ints(r, (3, 3, 32, 32), np.float16), T.empty_dev((1, 14, 14, 32), np.float16)
    big = ints(r, (4, 33, 29, 36), np.float16)

    def call(ctx):
        with pytest.raises(capi.PlbError, match="captured"):
            ctx.conv_fwd(ragged, big, w, big)
        ctx.conv_fwd(whole, x, w, y)

    got = captured(call, y)
    gpu_ctx.conv_fwd(whole, x, w, y)
    gpu_ctx.synchronize()
    assert (got == y.cpu().numpy()).all()
