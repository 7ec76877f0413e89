"""What a user of the library has it do, as cases that can be timed: matrix
products, fully connected and convolutional layers in inference and training,
and batch normalisation, through the library's public entry points
(`poplibs_b200.capi.Context`) on device-resident tensors.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw(rng)`
one more of the same ranges.  `prepare(case, seed)` makes what a program holds
before the call, `run(state)` makes ONE pass (an inference call or one training
step of the layer) and returns everything it computes.

Sizes: the convolutions and products that bench.py times, at its sizes and
around them, and generic ones (small and ragged extents, channel groups).
"""
import math

import torch

from poplibs_b200 import capi

DEVICE = 0

# A training step moves the weights by RATE * gradient.  Small enough that
# thousands of passes on one state leave the values in the range they began in.
RATE = 2.0 ** -20

_TORCH = {"half": torch.float16, "float": torch.float32}
_PLB = {"half": capi.HALF, "float": capi.FLOAT, "quarter": capi.QUARTER}
_BYTES = {"half": 2, "float": 4, "quarter": 1}
# exponents of the quarter operands' per-tensor scales (value = stored * 2^scale)
_SCALE_A, _SCALE_B = -3, -2

_context = None


def context():
    """The one library context (device, stream, scratch) of the program."""
    global _context
    if _context is None:
        _context = capi.Context(DEVICE)
    return _context


# ---------------------------------------------------------------------------- cases

def _matmul(name, m, k, n, groups=1, dtype="half", transpose_b=False):
    return {"name": name, "kind": "matmul", "dtype": dtype, "groups": groups, "m": m, "k": k, "n": n,
            "transpose_b": transpose_b}


def _fc(name, batch, inputs, outputs):
    return {"name": name, "kind": "fc_train", "dtype": "half", "batch": batch, "inputs": inputs,
            "outputs": outputs}


def _conv(name, passes, batch, height, width, kernel, chans_in, chans_out, stride=1, padding=0, groups=1,
          dtype="half"):
    """Channel counts are per group, as in the library."""
    return {"name": name, "kind": "conv", "passes": passes, "dtype": dtype, "batch": batch,
            "height": height, "width": width, "kernel": kernel, "chans_in": chans_in, "chans_out": chans_out,
            "stride": stride, "padding": padding, "groups": groups}


def _norm(name, batch, height, width, chans, dtype="half"):
    return {"name": name, "kind": "batch_norm_train", "dtype": dtype, "batch": batch, "height": height,
            "width": width, "chans": chans}


def listed():
    return [
        # The smallest call: one fully connected layer on a handful of rows, as in
        # low-latency inference.  Launch and host cost.
        _matmul("matmul_16x512x512", 16, 512, 512),
        # A product whose extents fit nothing: operands with odd row lengths.
        _matmul("matmul_ragged_197x770x1003", 197, 770, 1003),
        # Many small independent products in one call (matMulGrouped).
        _matmul("matmul_grouped_64x256x64x256", 256, 64, 256, groups=64, transpose_b=True),
        # The large 8-bit product with scaled operands; the most work of all cases.
        _matmul("matmul_quarter_8192", 8192, 8192, 8192, dtype="quarter", transpose_b=True),
        # Training step of a wide fully connected layer: output, input gradient,
        # weight gradient (both operands read along their slow axis), update.
        _fc("fc_train_2048x4096x4096", 2048, 4096, 4096),
        # One image through one 3x3 layer with a bias: inference latency.
        _conv("conv3x3_infer_n1_56x56_c64", "infer", 1, 56, 56, 3, 64, 64, padding=1),
        # Training step of a 3x3 layer on a large batch: forward with bias, both
        # gradients, weight and bias update.
        _conv("conv3x3_train_n256_28x28_c128", "train", 256, 28, 28, 3, 128, 128, padding=1),
        # Training step of an image network's first layer: three input channels,
        # no input gradient.
        _conv("conv7x7_s2_first_n256_224x224_c3_c64", "first", 256, 224, 224, 7, 3, 64, stride=2, padding=3),
        # Training step of a strided pointwise layer between two resolutions.
        _conv("conv1x1_s2_train_n256_56x56_c256_c512", "train", 256, 56, 56, 1, 256, 512, stride=2),
        # Training step of a layer with channel groups.
        _conv("conv3x3_grouped_train_n32_28x28_g32_c8", "train", 32, 28, 28, 3, 8, 8, padding=1, groups=32),
        # Training step in single precision with channel counts and extents that
        # are multiples of nothing.
        _conv("conv3x3_ragged_train_float_n4_33x29_c20_c36", "train", 4, 33, 29, 3, 20, 36, padding=1,
              dtype="float"),
        # Batch normalisation after a convolution, forward and backward.
        _norm("batch_norm_train_n32_56x56_c64", 32, 56, 56, 64),
    ]


def _log(rng, lo, hi, multiple=1):
    """An integer spread over the logarithm of [lo, hi], a multiple of `multiple`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, multiple * round(v / multiple), multiple)))


def _draw_matmul(rng):
    dtype = rng.choice(["half", "half", "half", "quarter", "float"])
    multiple = rng.choice([1, 1, 8, 64])
    while True:
        m, k, n = (_log(rng, 16, 8192, multiple) for _ in range(3))
        if 2 ** 20 <= m * k * n <= (2 ** 37 if dtype == "half" else 2 ** 36):
            break
    return _matmul("", m, k, n, dtype=dtype, transpose_b=rng.random() < 0.5)


def _draw_matmul_grouped(rng):
    multiple = rng.choice([1, 8, 16])
    return _matmul("", _log(rng, 16, 512, multiple), _log(rng, 16, 256, multiple), _log(rng, 16, 512, multiple),
                   groups=_log(rng, 2, 256), dtype=rng.choice(["half", "half", "float"]),
                   transpose_b=rng.random() < 0.5)


def _draw_fc(rng):
    multiple = rng.choice([1, 8, 64])
    return _fc("", _log(rng, 16, 4096), _log(rng, 64, 4096, multiple), _log(rng, 64, 4096, multiple))


def _draw_conv(rng):
    while True:
        kernel = rng.choice([1, 3, 3, 5])
        stride = rng.choice([1, 1, 2])
        groups = rng.choice([1, 1, 1, 2, 8, 32])
        passes = rng.choice(["infer", "train", "train"])
        dtype = rng.choice(["half", "half", "half", "half", "float", "quarter" if passes == "infer" else "half"])
        batch = _log(rng, 1, 256)
        height = _log(rng, 7, 112)
        width = rng.choice([height, _log(rng, 7, 112)])
        multiple = rng.choice([1, 8, 8, 16])
        chans_in = _log(rng, 16, 512, multiple) if groups == 1 else _log(rng, 4, 64, min(multiple, 8))
        chans_out = rng.choice([chans_in, _log(rng, 16, 512, multiple)]) if groups == 1 else chans_in
        case = _conv("", passes, batch, height, width, kernel, chans_in, chans_out, stride=stride,
                     padding=kernel // 2, groups=groups, dtype=dtype)
        elems = batch * height * width * groups * max(chans_in, chans_out)
        if elems * _BYTES[dtype] > 2 ** 27:
            continue
        flops = elems * kernel * kernel * min(chans_in, chans_out) * 2
        if 2 ** 23 <= flops <= 2 ** 35:
            return case


def _draw_first(rng):
    size = _log(rng, 32, 224)
    width = rng.choice([size, _log(rng, 32, 224)])
    kernel, stride = rng.choice([(7, 2), (7, 2), (3, 1), (3, 2)])
    batch = _log(rng, 1, max(1, 2 ** 23 // (size * width)))
    return _conv("", "first", batch, size, width, kernel, rng.choice([3, 3, 1, 4]), rng.choice([32, 64, 64, 96]),
                 stride=stride, padding=kernel // 2)


def _draw_norm(rng):
    while True:
        batch, height, chans = _log(rng, 1, 256), _log(rng, 7, 112), _log(rng, 16, 1024, rng.choice([1, 8, 32]))
        if 2 ** 14 <= batch * height * height * chans <= 2 ** 25:
            return _norm("", batch, height, height, chans, dtype=rng.choice(["half", "half", "half", "float"]))


def draw(rng):
    pick = rng.choice([_draw_matmul, _draw_matmul, _draw_matmul_grouped, _draw_fc, _draw_conv, _draw_conv,
                       _draw_conv, _draw_first, _draw_norm])
    case = pick(rng)
    del case["name"]
    return case


# ---------------------------------------------------------------------------- inputs

class _Data:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.device = torch.device("cuda", DEVICE)
        self.g = torch.Generator(device=self.device).manual_seed(int(seed))

    def uniform(self, shape, dtype, bound=1.0):
        t = torch.empty(shape, dtype=torch.float32, device=self.device)
        return t.uniform_(-bound, bound, generator=self.g).to(_TORCH[dtype])

    def normal(self, shape, dtype):
        t = torch.empty(shape, dtype=torch.float32, device=self.device)
        return t.normal_(generator=self.g).to(_TORCH[dtype])

    def quarter(self, shape, scale):
        """N(0, 1) quantised to E4M3 bytes, value = stored * 2^scale."""
        t = torch.empty(shape, dtype=torch.float32, device=self.device).normal_(generator=self.g)
        return t.mul_(2.0 ** -scale).to(torch.float8_e4m3fn).view(torch.uint8)

    def empty(self, shape, dtype):
        return torch.empty(shape, dtype=_TORCH[dtype], device=self.device)


def _result_type(dtype):
    return "float" if dtype == "float" else "half"


def _prepare_matmul(case, data):
    g, m, k, n, dtype = (case[f] for f in ("groups", "m", "k", "n", "dtype"))
    quarter, out = dtype == "quarter", _result_type(dtype)
    b_shape = (g, n, k) if case["transpose_b"] else (g, k, n)
    if quarter:
        a, b = data.quarter((g, m, k), _SCALE_A), data.quarter(b_shape, _SCALE_B)
    else:
        a, b = data.uniform((g, m, k), dtype), data.uniform(b_shape, dtype)
    desc = capi.MatmulDesc.make(m, k, n, groups=g, input_type=_PLB[dtype], output_type=_PLB[out],
                                transpose_b=case["transpose_b"], scale_a=_SCALE_A if quarter else 0,
                                scale_b=_SCALE_B if quarter else 0)
    return {"desc": desc, "a": a, "b": b, "d": data.empty((g, m, n), out)}


def _run_matmul(ctx, s):
    ctx.matmul(s["desc"], s["a"], s["b"], None, s["d"])
    return s["d"]


def _prepare_fc_train(case, data):
    batch, inputs, outputs = case["batch"], case["inputs"], case["outputs"]
    half = capi.HALF
    return {
        # y = x w,  dx = dy w^T,  dw = x^T dy, with w stored [inputs][outputs]
        "fwd": capi.MatmulDesc.make(batch, inputs, outputs, input_type=half, output_type=half),
        "bwd": capi.MatmulDesc.make(batch, outputs, inputs, input_type=half, output_type=half, transpose_b=True),
        "wu": capi.MatmulDesc.make(inputs, batch, outputs, input_type=half, output_type=capi.FLOAT,
                                   transpose_a=True),
        "x": data.uniform((batch, inputs), "half"), "dy": data.uniform((batch, outputs), "half"),
        "w": data.uniform((inputs, outputs), "half", 1.0 / math.sqrt(inputs)),
        "y": data.empty((batch, outputs), "half"), "dx": data.empty((batch, inputs), "half"),
        "dw": data.empty((inputs, outputs), "float"), "count": inputs * outputs}


def _run_fc_train(ctx, s):
    ctx.matmul(s["fwd"], s["x"], s["w"], None, s["y"])
    ctx.matmul(s["bwd"], s["dy"], s["w"], None, s["dx"])
    ctx.matmul(s["wu"], s["x"], s["dy"], None, s["dw"])
    ctx.scaled_add_to(capi.HALF, s["w"], s["dw"], -RATE, s["count"])
    return {"y": s["y"], "dx": s["dx"], "dw": s["dw"], "w": s["w"]}


def _conv_params(case):
    dtype = case["dtype"]
    return capi.ConvParams.make(case["batch"], [case["height"], case["width"]], [case["kernel"]] * 2,
                                case["chans_in"], case["chans_out"], groups=case["groups"],
                                input_type=_PLB[dtype], output_type=_PLB[_result_type(dtype)],
                                padding=case["padding"], stride=case["stride"])


def _prepare_conv(case, data):
    p = _conv_params(case)
    dtype, g = case["dtype"], case["groups"]
    ci, co, k = case["chans_in"], case["chans_out"], case["kernel"]
    oh, ow = p.output_field()
    x_shape = (case["batch"], case["height"], case["width"], g * ci)
    y_shape = (case["batch"], oh, ow, g * co)
    w_shape = (g, k, k, co, ci)
    bound = 1.0 / math.sqrt(ci * k * k)
    s = {"p": p, "opt": None, "passes": case["passes"], "dtype": _PLB[dtype], "w_count": g * k * k * co * ci,
         "pixels": case["batch"] * oh * ow, "chans": g * co,
         "bias": data.uniform((g * co,), "float"), "y": data.empty(y_shape, _result_type(dtype))}
    if dtype == "quarter":
        s["opt"] = capi.ConvOptions.make(pass_=capi.PASS_INFERENCE_FWD, scale_in=_SCALE_A, scale_weights=_SCALE_B)
        s["x"], s["w"] = data.quarter(x_shape, _SCALE_A), data.quarter(w_shape, _SCALE_B)
    else:
        s["x"], s["w"] = data.uniform(x_shape, dtype), data.uniform(w_shape, dtype, bound)
    if case["passes"] != "infer":
        s["dy"] = data.uniform(y_shape, dtype)
        s["dw"] = data.empty(w_shape, "float")
        if case["passes"] == "train":
            s["dx"] = data.empty(x_shape, dtype)
    return s


def _run_conv(ctx, s):
    p = s["p"]
    ctx.conv_fwd(p, s["x"], s["w"], s["y"], bias=s["bias"], opt=s["opt"])
    if s["passes"] == "infer":
        return s["y"]
    out = {"y": s["y"], "dw": s["dw"], "w": s["w"], "bias": s["bias"]}
    if s["passes"] == "train":
        ctx.conv_bwd(p, s["dy"], s["w"], s["dx"])
        out["dx"] = s["dx"]
    ctx.conv_wu(p, s["x"], s["dy"], None, s["dw"])
    ctx.scaled_add_to(s["dtype"], s["w"], s["dw"], -RATE, s["w_count"])
    ctx.conv_bias_update(s["dtype"], s["dy"], s["pixels"], s["chans"], capi.FLOAT, s["bias"], -RATE)
    return out


def _prepare_batch_norm_train(case, data):
    dtype, chans = case["dtype"], case["chans"]
    pixels = case["batch"] * case["height"] * case["width"]
    shape = (pixels, chans)
    s = {"dtype": _PLB[dtype], "pixels": pixels, "chans": chans,
         # a convolution's output: roughly normal, channels off centre
         "x": data.normal(shape, dtype).add_(data.uniform((chans,), dtype)), "dy": data.uniform(shape, dtype),
         "gamma": data.uniform((chans,), dtype).abs_().add_(0.5), "beta": data.uniform((chans,), dtype)}
    for f in ("whitened", "y", "dx"):
        s[f] = data.empty(shape, dtype)
    for f in ("mean", "inv_std", "dgamma", "dbeta"):
        s[f] = data.empty((chans,), dtype)
    s["grad"] = data.empty(shape, dtype)
    return s


def _run_batch_norm_train(ctx, s):
    t, n, c = s["dtype"], s["pixels"], s["chans"]
    ctx.norm_statistics(t, s["x"], n, c, 1e-3, 1.0, s["mean"], s["inv_std"])
    ctx.norm_normalise(t, s["x"], s["mean"], s["inv_std"], s["gamma"], s["beta"], n, c, s["whitened"], s["y"])
    ctx.norm_param_gradients(t, s["whitened"], s["dy"], n, c, 1.0, s["dgamma"], s["dbeta"])
    ctx.norm_scale_shift(t, s["dy"], s["gamma"], None, n, c, s["grad"])
    ctx.norm_statistics_gradients(t, s["whitened"], s["grad"], s["inv_std"], n, c, s["dx"])
    return {f: s[f] for f in ("mean", "inv_std", "whitened", "y", "dgamma", "dbeta", "grad", "dx")}


_PREPARE = {"matmul": _prepare_matmul, "fc_train": _prepare_fc_train, "conv": _prepare_conv,
            "batch_norm_train": _prepare_batch_norm_train}
_RUN = {"matmul": _run_matmul, "fc_train": _run_fc_train, "conv": _run_conv,
        "batch_norm_train": _run_batch_norm_train}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, _Data(seed))
    state["context"], state["run"] = context(), _RUN[case["kind"]]
    # the inputs were made on torch's stream, the library works on its own
    torch.cuda.synchronize(DEVICE)
    return state


def run(state):
    return state["run"](state["context"], state)


# ---------------------------------------------------------------------------- yardsticks

def work(case):
    """Operations (2 per product, products with padding not counted) and bytes
    (every input read once, every output written once) of one pass."""
    kind, es = case["kind"], _BYTES[case["dtype"]]
    out = _BYTES[_result_type(case["dtype"])]
    if kind == "matmul":
        g, m, k, n = case["groups"], case["m"], case["k"], case["n"]
        return {"bytes": g * ((m * k + k * n) * es + m * n * out), "flops": 2 * g * m * k * n}
    if kind == "fc_train":
        b, i, o = case["batch"], case["inputs"], case["outputs"]
        # x, dy, y, dx; w read and written; dw written
        return {"bytes": 2 * b * (i + o) * es + i * o * (2 * es + 4), "flops": 6 * b * i * o + 2 * i * o}
    if kind == "batch_norm_train":
        n = case["batch"] * case["height"] * case["width"] * case["chans"]
        # x, dy read; whitened, y, grad, dx written
        return {"bytes": 6 * n * es + 6 * case["chans"] * es, "flops": 20 * n}
    p = _conv_params(case)
    oh, ow = p.output_field()
    g, ci, co, k = case["groups"], case["chans_in"], case["chans_out"], case["kernel"]
    x = case["batch"] * case["height"] * case["width"] * g * ci
    y = case["batch"] * oh * ow * g * co
    w = g * k * k * ci * co
    if k == 1 and case["stride"] > 1:
        x_read = case["batch"] * oh * ow * g * ci  # a strided pointwise layer reads a sub-lattice
    else:
        x_read = x
    size = x_read * es + w * es + y * out + g * co * 4
    flops = 2 * p.macs()
    if case["passes"] != "infer":
        size += y * es + w * 4 + w * es + g * co * 4        # dy; dw, w and bias written
        flops *= 3 if case["passes"] == "train" else 2
        if case["passes"] == "train":
            size += x * es
    return {"bytes": size, "flops": flops}


def tolerance(case):
    if case["dtype"] == "float":
        # sums of fp32, products of float operands to a relative 2^-16
        return {"rel": 3e-5 if case["kind"] in ("matmul", "conv") else 1e-5}
    # one rounding to half (2^-11) of sums that may be formed in another order;
    # normalisation rounds the statistics and the whitened values on the way
    return {"rel": 2e-3 if case["kind"] == "batch_norm_train" else 1e-3}
