// C ABI entry points of the contraction path: matMul, convolution forward and
// backward-data.  Each maps its poplin-level description onto one or more
// launches of the implicit-GEMM kernel (igemm_sm100.cuh).
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <utility>
#include <vector>

#include "conv_geometry.h"
#include "direct.h"
#include "grouped.h"
#include "patch.h"
#include "runtime.h"
#include "igemm_sm100.cuh"
#include "sm100_prims.cuh"
#include "small_channel.h"
#include "stem.h"

namespace plb {

int launchScaleRows(plb_context *ctx, void *out, const void *c, float beta, bool out_f32,
                    uint32_t rows, uint32_t cols, long long ldo, long long ldc);
int convFwdSmallChannels(plb_context *ctx, const plb_conv_params &p, const plb_conv_options *opt,
                         const void *d_in, const void *d_weights, const float *d_bias,
                         void *d_out, plb_plan *plan_only);

// TMA needs 16-byte pixel strides: 8 half / 16 quarter channels.
static bool channelsFitTma(const plb_conv_params &p, uint32_t chans) {
  return (size_t(chans) * dtypeBytes(p.input_type)) % 16 == 0;
}

namespace {

int checkMatmulDesc(const plb_matmul_desc &d) {
  if (!is16BitFloat(d.input_type) && d.input_type != PLB_QUARTER && d.input_type != PLB_FLOAT)
    return fail(PLB_ERR_INVALID_PARAMS, "matMul input type must be half or quarter");
  if (d.output_type != PLB_HALF && d.output_type != PLB_FLOAT)
    return fail(PLB_ERR_INVALID_PARAMS, "matMul output type must be half or float");
  if (d.input_type == PLB_QUARTER && d.output_type != PLB_HALF)
    // lib/poplin/ConvValidation.cpp:53-69: quarter input requires half output
    return fail(PLB_ERR_INVALID_PARAMS, "Output type must be half when input type is quarter");
  if (d.partials_type != PLB_HALF && d.partials_type != PLB_FLOAT)
    return fail(PLB_ERR_INVALID_OPTION, "partialsType must be half or float");
  if (d.scale_a < -32 || d.scale_a > 31 || d.scale_b < -32 || d.scale_b > 31)
    return fail(PLB_ERR_INVALID_PARAMS, "quarter metadata scale must be in [-32, 31]");
  if ((d.format_a != PLB_F143 && d.format_a != PLB_F152) || (d.format_b != PLB_F143 && d.format_b != PLB_F152))
    return fail(PLB_ERR_INVALID_PARAMS, "quarter format must be PLB_F143 or PLB_F152");
  return PLB_OK;
}

struct Ld {
  long long a, b, c;
};

Ld leadingDims(const plb_matmul_desc &d) {
  Ld l;
  l.a = d.lda ? d.lda : (d.transpose_a ? d.m : d.k);
  l.b = d.ldb ? d.ldb : (d.transpose_b ? d.k : d.n);
  l.c = d.ldc ? d.ldc : d.n;
  return l;
}

// The igemm problem of a matrix product (all groups).  `a` is [m][k] (row stride
// lda) or, with a_is_km, [k][m]; `b` either [n][k] (b_is_nk) or [k][n].
IgemmProblem gemmProblem(const plb_matmul_desc &d, const void *a, long long lda, bool a_is_km, const void *b,
                         long long ldb, bool b_is_nk, const void *c, void *out, long long ldc) {
  IgemmProblem p;
  const size_t es = dtypeBytes(d.input_type);
  p.fp8 = d.input_type == PLB_QUARTER;
  p.bf16 = d.input_type == PLB_BFLOAT16;
  p.fmt_a = d.format_a;
  p.fmt_b = d.format_b;
  p.a_mn = a_is_km;
  p.b_mn = !b_is_nk;
  p.groups = int(d.groups);
  p.act = a;
  p.act_dims[0] = d.k;
  p.act_dims[1] = d.m;
  p.act_strides[0] = uint64_t(lda) * es;
  p.act_strides[1] = uint64_t(lda) * es * std::max<uint32_t>(a_is_km ? d.k : d.m, 1);
  p.act_strides[2] = p.act_strides[1];
  p.act_group_stride = p.act_strides[1];
  p.wgt = b;
  p.wgt_dims[0] = b_is_nk ? d.k : d.n;
  p.wgt_dims[1] = b_is_nk ? d.n : d.k;
  p.wgt_dims[2] = d.groups;
  p.wgt_strides[0] = uint64_t(ldb) * es;
  p.wgt_strides[1] = uint64_t(ldb) * es * std::max<uint64_t>(p.wgt_dims[1], 1);
  p.out_w = int(d.m);
  p.n_total = int(d.n);
  p.k_per_tap = int(d.k);
  p.out = out;
  p.ldc = ldc;
  p.out_group_stride = (long long)d.m * ldc;
  p.addend = c;
  p.ld_addend = ldc;
  p.addend_group_stride = p.out_group_stride;
  p.alpha = d.alpha;
  if (p.fp8) p.alpha *= std::ldexp(1.0f, d.scale_a + d.scale_b);
  p.beta = d.beta;
  p.out_f32 = d.output_type == PLB_FLOAT;
  return p;
}

uint64_t gemmBytes(const plb_matmul_desc &d) {
  const uint64_t es = dtypeBytes(d.input_type), os = dtypeBytes(d.output_type);
  return uint64_t(d.groups) * (uint64_t(d.m) * d.k * es + uint64_t(d.k) * d.n * es +
                               uint64_t(d.m) * d.n * os * (d.beta != 0.f ? 2 : 1));
}

// ---- convolution --------------------------------------------------------------------

struct ConvShape {
  unsigned nd;
  int H, W, OH, OW;      // input / output field as stored (H = 1 for 1-D)
  int KH, KW;            // filter taps that are used (the kernel after truncation)
  int KHs, KWs;          // filter extent as stored
  int ktH, ktW;          // kernel truncation at the low end
  // padH/padW: input padding minus output truncation minus kernel padding at
  // the low end (the high end's kernel padding for a flipped kernel), i.e.
  // output position o, used tap r reads truncated-input row
  // o*stride + r*dil - pad (may be negative: the first rows are skipped)
  int padH, padW, dilH, dilW, strH, strW, flipH, flipW;
  int tH, tW;            // input truncation at the low end (rows / columns not used)
  int He, We;            // extent of the truncated input
  int opH, opW;          // output padding at the low end (zero rows / columns)
  int OHc, OWc;          // extent of the computed (not padded) output
  bool zero_fill_out;    // the output has padded positions
  bool zero_fill_in;     // the input has truncated positions (backward pass zeroes them)
};

int igemmConvShape(const plb_conv_params &p, ConvShape *s) {
  const std::string err = validate(p);
  if (!err.empty()) return fail(PLB_ERR_INVALID_PARAMS, err);
  if (p.num_field_dims > 2)
    return fail(PLB_ERR_UNSUPPORTED, "3-D convolutions are not implemented on this path yet");
  if (!is16BitFloat(p.input_type) && p.input_type != PLB_QUARTER && p.input_type != PLB_FLOAT)
    return fail(PLB_ERR_UNSUPPORTED, "convolution input type must be half, float or quarter");
  if (p.output_type != PLB_HALF && p.output_type != PLB_FLOAT)
    return fail(PLB_ERR_INVALID_PARAMS, "convolution output type must be half or float");
  if (p.input_type == PLB_QUARTER && p.output_type != PLB_HALF)
    return fail(PLB_ERR_INVALID_PARAMS, "Output type must be half when input type is quarter");
  // Input truncation, output truncation and output padding are views and
  // offsets (below).  Input dilation only arrives through the backward pass of
  // a strided layer, which plb_conv_bwd takes in forward terms.
  // Kernel truncation selects a sub-rectangle of the taps (a sub-lattice of the
  // stored filter, setTaps), kernel padding only shifts where the taps land.
  for (unsigned d = 0; d != p.num_field_dims; ++d) {
    if (p.in_dilation[d] != 1 || p.in_flip[d])
      return fail(PLB_ERR_UNSUPPORTED,
                  "input dilation/flip are not implemented on this path yet");
  }
  s->nd = p.num_field_dims;
  const unsigned hd = p.num_field_dims == 2 ? 0 : ~0u, wd = p.num_field_dims - 1;
  auto get = [&](const uint32_t *v, unsigned d, int dflt) { return d == ~0u ? dflt : int(v[d]); };
  s->H = get(p.field, hd, 1);
  s->W = get(p.field, wd, 1);
  s->KHs = get(p.kernel, hd, 1);
  s->KWs = get(p.kernel, wd, 1);
  s->ktH = get(p.k_trunc_lo, hd, 0);
  s->ktW = get(p.k_trunc_lo, wd, 0);
  s->KH = s->KHs - s->ktH - get(p.k_trunc_hi, hd, 0);
  s->KW = s->KWs - s->ktW - get(p.k_trunc_hi, wd, 0);
  s->padH = get(p.in_pad_lo, hd, 0);
  s->padW = get(p.in_pad_lo, wd, 0);
  s->dilH = get(p.k_dilation, hd, 1);
  s->dilW = get(p.k_dilation, wd, 1);
  s->strH = get(p.stride, hd, 1);
  s->strW = get(p.stride, wd, 1);
  s->flipH = get(p.k_flip, hd, 0);
  s->flipW = get(p.k_flip, wd, 0);
  s->OH = hd == ~0u ? 1 : int(outputSize(p, hd));
  s->OW = int(outputSize(p, wd));
  s->tH = get(p.in_trunc_lo, hd, 0);
  s->tW = get(p.in_trunc_lo, wd, 0);
  s->He = s->H - s->tH - get(p.in_trunc_hi, hd, 0);
  s->We = s->W - s->tW - get(p.in_trunc_hi, wd, 0);
  s->padH -= get(p.out_trunc_lo, hd, 0) + get(s->flipH ? p.k_pad_hi : p.k_pad_lo, hd, 0);
  s->padW -= get(p.out_trunc_lo, wd, 0) + get(s->flipW ? p.k_pad_hi : p.k_pad_lo, wd, 0);
  s->opH = get(p.out_pad_lo, hd, 0);
  s->opW = get(p.out_pad_lo, wd, 0);
  s->OHc = s->OH - s->opH - get(p.out_pad_hi, hd, 0);
  s->OWc = s->OW - s->opW - get(p.out_pad_hi, wd, 0);
  s->zero_fill_out = s->OHc != s->OH || s->OWc != s->OW;
  s->zero_fill_in = s->He != s->H || s->We != s->W;
  return PLB_OK;
}

uint64_t convBytes(const plb_conv_params &p, const ConvShape &s, int pass) {
  const uint64_t es = dtypeBytes(p.input_type), os = dtypeBytes(p.output_type);
  const uint64_t in = uint64_t(p.batch) * s.H * s.W * p.groups * p.in_chans_per_group;
  const uint64_t out = uint64_t(p.batch) * s.OH * s.OW * p.groups * p.out_chans_per_group;
  const uint64_t w = uint64_t(p.groups) * s.KH * s.KW * p.in_chans_per_group * p.out_chans_per_group;
  // a 1x1 kernel with stride reads only every stride-th pixel
  uint64_t in_read = in;
  if (s.KH == 1 && s.KW == 1) in_read = uint64_t(p.batch) * s.OH * s.OW * p.groups * p.in_chans_per_group;
  switch (pass) {
    case PLB_PASS_TRAINING_BWD: return out * es + w * es + in * os;
    case PLB_PASS_TRAINING_WU: return in * es + out * es + w * es;
    default: return in_read * es + w * es + out * os;
  }
}

// The operands of a pass as the kernel reads them: the activations (or output
// gradients) with `act_pitch` channels per group and pixel, the weights as rows of
// `w_pitch` elements, and `k` channels to reduce over per tap (three times the
// layer's for float operands, whose type is then bfloat16).
struct PassOperands {
  int type;
  const void *act, *wgt;
  uint32_t k, act_pitch, w_pitch;
  bool lattice = false;  // the activations hold only the pixels a strided pointwise layer reads
};

// The filter taps of a problem: tap (r, s) is stored tile
// (first_h + r*step_h) * KWs + first_w + s*step_w of a filter of KHs x KWs.
void setTaps(IgemmProblem *r, const ConvShape &s, int first_h, int step_h, int first_w, int step_w) {
  r->tap_first_h = first_h;
  r->tap_step_h = step_h;
  r->tap_pitch_h = s.KWs;
  r->tap_first_w = first_w;
  r->tap_step_w = step_w;
  r->taps_stored = s.KHs * s.KWs;
}

// What the passes have in common: operand types, weights, options.  `w_rows` is
// the number of rows of a stored weight tile (its second dimension).
IgemmProblem passProblem(const plb_conv_params &p, const plb_conv_options *opt, const ConvShape &s,
                         const PassOperands &o, bool b_mn, uint64_t w_rows) {
  const size_t es = dtypeBytes(o.type);
  IgemmProblem r;
  r.fp8 = o.type == PLB_QUARTER;
  r.bf16 = o.type == PLB_BFLOAT16;
  r.fmt_a = opt ? opt->format_in : 0;
  r.fmt_b = opt ? opt->format_weights : 0;
  r.groups = int(p.groups);
  r.act_group_stride = uint64_t(o.act_pitch) * es;
  r.wgt = o.wgt;
  r.b_mn = b_mn;
  r.wgt_dims[0] = o.w_pitch;  // (what rows were rounded up by holds zeros)
  r.wgt_dims[1] = w_rows;
  r.wgt_dims[2] = uint64_t(p.groups) * s.KHs * s.KWs;
  r.wgt_strides[0] = uint64_t(o.w_pitch) * es;
  r.wgt_strides[1] = w_rows * o.w_pitch * es;
  r.k_per_tap = int(o.k);
  r.out_n = int(p.batch);
  r.out_f32 = p.output_type == PLB_FLOAT;
  r.force_tile_n = opt ? opt->tile_n : 0;
  r.force_split_k = opt ? opt->split_k : 0;
  r.plan_flags = opt ? opt->plan_flags : 0;
  if (r.fp8 && opt) r.alpha = std::ldexp(1.0f, opt->scale_in + opt->scale_weights);
  return r;
}

// Activations [N][H][W][G * act_pitch]: the view that starts at (h0, w0).
void setActs(IgemmProblem *r, const plb_conv_params &p, const PassOperands &o, int H, int W, int h0, int w0) {
  const size_t es = dtypeBytes(o.type);
  const uint64_t ctot = uint64_t(p.groups) * o.act_pitch;
  r->act = static_cast<const uint8_t *>(o.act) + (size_t(h0) * W + w0) * ctot * es;
  r->act_dims[0] = std::max(o.act_pitch, o.k);  // (likewise)
  r->act_strides[0] = ctot * es;
  r->act_strides[1] = uint64_t(W) * ctot * es;
  r->act_strides[2] = uint64_t(H) * W * ctot * es;
}

// A 1x1 convolution without padding reads every stride'th pixel alone.
bool pointwise(const ConvShape &s) { return s.KH == 1 && s.KW == 1 && s.padH == 0 && s.padW == 0; }
int latticeExtent(int in, int out, int stride) { return std::min(out, (in + stride - 1) / stride); }

// Forward problem (all groups).
// With `swapped_weights` the weights are stored [G][tap][Ci][Co] (the forward
// layout of the layer this convolution is the backward pass of) and are used
// with their spatial axes flipped: they are read as a K-by-N (MN-major) operand.
// With `flipped_taps` they are stored [G][flipped tap][Co][Ci].
IgemmProblem convFwdProblem(const plb_conv_params &p, const plb_conv_options *opt, const ConvShape &s,
                            const PassOperands &o, const float *bias, void *out, bool swapped_weights = false,
                            bool flipped_taps = false) {
  const size_t os = dtypeBytes(p.output_type);
  const uint64_t co = p.out_chans_per_group, cotot = uint64_t(p.groups) * co;
  IgemmProblem r = swapped_weights ? passProblem(p, opt, s, o, true, o.k) : passProblem(p, opt, s, o, false, co);
  // the truncated input is a view: same strides, shifted base, smaller extents
  setActs(&r, p, o, s.H, s.W, s.tH, s.tW);
  if (o.lattice) {
    r.act_dims[1] = uint64_t(latticeExtent(s.We, s.OWc, s.strW));
    r.act_dims[2] = uint64_t(latticeExtent(s.He, s.OHc, s.strH));
    setActs(&r, p, o, int(r.act_dims[2]), int(r.act_dims[1]), 0, 0);
  } else if (pointwise(s)) {
    // a strided 1x1 convolution reads a sub-lattice: describe only that (its
    // extent is what the input holds; outputs beyond it read zero padding)
    r.act_dims[1] = uint64_t(latticeExtent(s.We, s.OWc, s.strW));
    r.act_dims[2] = uint64_t(latticeExtent(s.He, s.OHc, s.strH));
    r.act_strides[0] *= uint64_t(s.strW);
    r.act_strides[1] *= uint64_t(s.strH);
  } else {
    r.act_dims[1] = uint64_t(s.We);
    r.act_dims[2] = uint64_t(s.He);
    r.stride_h = s.strH;
    r.stride_w = s.strW;
    r.act_elem_strides[1] = uint32_t(s.strW);
    r.act_elem_strides[2] = uint32_t(s.strH);
  }
  r.act_dims[3] = p.batch;
  // the computed part of the output is a view of the stored (padded) one
  r.out_w = s.OWc;
  r.out_h = s.OHc;
  r.n_total = int(co);
  r.taps_h = s.KH;
  r.taps_w = s.KW;
  if (flipped_taps)
    setTaps(&r, s, s.KHs - s.ktH - s.KH, 1, s.KWs - s.ktW - s.KW, 1);
  else
    setTaps(&r, s, s.ktH, 1, s.ktW, 1);
  r.pad_h = s.padH;
  r.pad_w = s.padW;
  r.dil_h = s.dilH;
  r.dil_w = s.dilW;
  r.flip_h = swapped_weights ? !s.flipH : s.flipH;
  r.flip_w = swapped_weights ? !s.flipW : s.flipW;
  r.out = static_cast<uint8_t *>(out) + (size_t(s.opH) * s.OW + s.opW) * cotot * os;
  r.ldc = (long long)cotot;
  r.out_stride_h = (long long)(cotot * s.OW);
  r.out_stride_n = (long long)(cotot * s.OW * s.OH);
  r.out_group_stride = (long long)co;
  r.bias = bias;
  return r;
}

// Backward-data problem (stride 1, all groups): the output gradients take the
// activations' role, the taps are traversed in the opposite order, the padding
// becomes (k-1)*dilation - padding, and the stored [tap][Co][Ci] weights are
// read as a K-by-N (MN-major) operand with K = Co, N = Ci.
IgemmProblem convBwdProblem(const plb_conv_params &p, const plb_conv_options *opt, const ConvShape &s,
                            const PassOperands &o, void *dx, bool weights_transposed) {
  const size_t os = dtypeBytes(p.output_type);
  const uint64_t ci = p.in_chans_per_group, ctot = uint64_t(p.groups) * ci;
  // transposed: [tap flipped][Ci][Co], a K-major operand with the taps already reversed
  IgemmProblem r = weights_transposed ? passProblem(p, opt, s, o, false, ci) : passProblem(p, opt, s, o, true, o.k);
  // computed part of the output gradients / used part of the input gradients
  setActs(&r, p, o, s.OH, s.OW, s.opH, s.opW);
  r.act_dims[1] = uint64_t(s.OWc);
  r.act_dims[2] = uint64_t(s.OHc);
  r.act_dims[3] = p.batch;
  r.flip_h = weights_transposed ? s.flipH : !s.flipH;
  r.flip_w = weights_transposed ? s.flipW : !s.flipW;
  r.out_w = s.We;
  r.out_h = s.He;
  r.n_total = int(ci);
  r.taps_h = s.KH;
  r.taps_w = s.KW;
  if (weights_transposed)
    setTaps(&r, s, s.KHs - s.ktH - s.KH, 1, s.KWs - s.ktW - s.KW, 1);
  else
    setTaps(&r, s, s.ktH, 1, s.ktW, 1);
  r.pad_h = (s.KH - 1) * s.dilH - s.padH;
  r.pad_w = (s.KW - 1) * s.dilW - s.padW;
  r.dil_h = s.dilH;
  r.dil_w = s.dilW;
  r.out = static_cast<uint8_t *>(dx) + (size_t(s.tH) * s.W + s.tW) * ctot * os;
  r.ldc = (long long)ctot;
  r.out_stride_h = (long long)(ctot * s.W);
  r.out_stride_n = (long long)(ctot * s.W * s.H);
  r.out_group_stride = (long long)ci;
  return r;
}

int runProblem(plb_context *ctx, IgemmProblem &r) {
  r.plan_flags |= ctx->plan_flags;
  plb_plan plan{};
  if (int rc = planIgemm(r, ctx->sm_count, &plan)) return rc;
  return launchIgemm(ctx, r, plan);
}

// out[pixel][c] = bias[c]: what a convolution with a fused bias leaves where
// nothing is accumulated (output padding).
template <typename T>
__global__ void fillBiasKernel(T *out, const float *__restrict__ bias, size_t total, size_t chans) {
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < total;
       i += size_t(gridDim.x) * blockDim.x)
    out[i] = T(bias[i % chans]);
}

// One dimension of the backward pass of a strided convolution, for the input
// positions i*stride + phase: which filter taps reach them and where.  Tap r
// reaches the phase iff (phase + pad - r*dil) is a multiple of the stride; with
// g = gcd(dil, stride) those taps are r0, r0 + stride/g, ... and, from one to the
// next, the output index read at a fixed i moves by dil/g.
struct BwdPhase {
  int first_tap;   // r0: smallest tap with (phase + pad - r*dil) divisible by stride
  int taps;        // J: taps r0, r0 + step, ...
  int step;        // stride / gcd(dil, stride)
  int dil;         // dil / gcd(dil, stride): dilation of the gathered sub-filter
  int offset;      // (phase + pad - r0*dil) / stride: output index read by tap r0 at i = 0
  int extent;      // input positions of this phase
};
void bwdPhase(int phase, int in_size, int kernel, int pad, int dil, int stride, BwdPhase *out) {
  int g = dil, t = stride;
  while (t) {
    const int u = g % t;
    g = t;
    t = u;
  }
  out->extent = phase < in_size ? (in_size - phase + stride - 1) / stride : 0;
  out->first_tap = -1;
  out->taps = 0;
  out->offset = 0;
  out->step = stride / g;
  out->dil = dil / g;
  for (int r = 0; r < kernel; ++r) {
    const int num = phase + pad - r * dil;
    if (((num % stride) + stride) % stride != 0) continue;
    if (out->first_tap < 0) {
      out->first_tap = r;
      out->offset = num / stride;  // exact: num is a multiple of stride (possibly negative)
    }
    ++out->taps;
  }
}

// ---- operands TMA cannot address, float operands -----------------------------------
// A pixel's channels of one group, and a row of a weight tile, must be a multiple
// of 16 bytes for the tensor maps (8 half / 16 quarter channels).  Other counts
// run on copies with the rows rounded up; the output is written as it is.  Float
// operands are split into their bfloat16 pieces by the same pass.
//
// `rows` of `cols` elements each become the activations; the weights are `w_rows`
// rows of `w_cols` elements, the reduction along their rows (w_k_rows = false) or
// along `w_k_rows` rows of each tile.
// With a lattice only its pixels are copied, if a copy is made at all (`o->lattice`).
// planOperands says what has to be copied (with null pointers: for operands as aligned
// as they need to be), prepareOperands does it.
struct Copies {
  Repack jobs[2];
  const void **operand[2];
  size_t offset[2];
  int n = 0;
  size_t bytes = 0;
  void add(const Repack &job, const void **base) {
    jobs[n] = job;
    operand[n] = base;
    offset[n++] = bytes;
    bytes += (repackBytes(job) + 255) & ~size_t(255);
  }
};

int runCopies(plb_context *ctx, Copies &c) {
  if (c.n == 0) return PLB_OK;
  void *ws = nullptr;
  if (int rc = scratch(ctx, kSlotRepacked, c.bytes + 256, &ws)) return rc;
  for (int i = 0; i < c.n; ++i) *c.operand[i] = c.jobs[i].dst = static_cast<uint8_t *>(ws) + c.offset[i];
  return repack(ctx, c.jobs, c.n);
}

Copies planOperands(int type, const void *act, uint64_t rows, uint32_t cols, const void *wgt, uint64_t w_rows,
                    uint32_t w_cols, uint64_t w_k_rows, PassOperands *o, const Repack::Lattice *lattice = nullptr) {
  const size_t es = dtypeBytes(type);
  const bool is_float = type == PLB_FLOAT;
  o->type = is_float ? PLB_BFLOAT16 : type;
  o->act = act;
  o->wgt = wgt;
  o->k = is_float ? 3 * cols : cols;
  o->act_pitch = cols;
  o->w_pitch = w_cols;
  auto unfit = [&](const void *base, uint32_t c) {
    return is_float || (c * es) % 16 != 0 || (reinterpret_cast<uintptr_t>(base) & 15) != 0;
  };
  Copies c;
  if (unfit(act, cols)) {
    o->act_pitch = is_float ? roundToRow(3 * uint64_t(cols), 2) : roundToRow(cols, es);
    Repack job{act, nullptr, rows, cols, cols, o->act_pitch, uint32_t(es), is_float ? kRepackSplitCols : kRepackCopy, false, 0, {}};
    if (lattice) {
      job.lattice = *lattice;
      job.rows = rows / (uint64_t(lattice->full_h) * lattice->full_w) * lattice->sub_h * lattice->sub_w;
      o->lattice = true;
    }
    c.add(job, &o->act);
  }
  if (unfit(wgt, w_cols)) {
    const bool along_rows = is_float && w_k_rows == 0;
    o->w_pitch = along_rows ? roundToRow(3 * uint64_t(w_cols), 2) : roundToRow(w_cols, is_float ? 2 : es);
    c.add(Repack{wgt, nullptr, w_rows, w_cols, w_cols, o->w_pitch, uint32_t(es),
                 !is_float ? kRepackCopy : along_rows ? kRepackSplitCols : kRepackSplitPlanes, true, w_k_rows, {}},
          &o->wgt);
  }
  return c;
}

// Whether the implicit-GEMM kernel can only read a copy of an operand (`k` channels of
// a group's pixel).
bool operandsCopied(const PassOperands &o, uint32_t k) {
  const size_t es = dtypeBytes(o.type);
  return o.type == PLB_FLOAT || (k * es) % 16 != 0 || (o.w_pitch * es) % 16 != 0 ||
         ((reinterpret_cast<uintptr_t>(o.act) | reinterpret_cast<uintptr_t>(o.wgt)) & 15) != 0;
}

int prepareOperands(plb_context *ctx, int type, const void *act, uint64_t rows, uint32_t cols, const void *wgt,
                    uint64_t w_rows, uint32_t w_cols, uint64_t w_k_rows, PassOperands *o,
                    const Repack::Lattice *lattice = nullptr) {
  Copies c = planOperands(type, act, rows, cols, wgt, w_rows, w_cols, w_k_rows, o, lattice);
  return runCopies(ctx, c);
}

// The same for a matrix product: rows of any pitch.  The pitches become those of what
// the kernel reads.
Copies planCopies(const plb_matmul_desc &d, const void **a, long long *lda, bool a_is_km, const void **b, long long *ldb,
                  bool b_is_nk) {
  const bool is_float = d.input_type == PLB_FLOAT;
  const size_t es = dtypeBytes(d.input_type);
  Copies c;
  // (all groups' rows are uniformly `pitch` elements apart)
  auto add = [&](const void **base, long long *pitch, uint64_t rows, uint32_t cols, bool k_along_rows, bool weights) {
    if (!is_float && (reinterpret_cast<uintptr_t>(*base) & 15) == 0 && (size_t(*pitch) * es) % 16 == 0) return;
    const int mode = !is_float ? kRepackCopy : k_along_rows ? kRepackSplitPlanes : kRepackSplitCols;
    const uint32_t pitch_out = mode == kRepackCopy ? roundToRow(cols, es)
                                                   : roundToRow(mode == kRepackSplitCols ? 3 * uint64_t(cols) : cols, 2);
    c.add(Repack{*base, nullptr, rows, cols, uint64_t(*pitch), pitch_out, uint32_t(es), mode, weights, d.k, {}}, base);
    *pitch = pitch_out;
  };
  add(a, lda, uint64_t(d.groups) * (a_is_km ? d.k : d.m), a_is_km ? d.m : d.k, a_is_km, false);
  add(b, ldb, uint64_t(d.groups) * (b_is_nk ? d.n : d.k), b_is_nk ? d.k : d.n, !b_is_nk, true);
  return c;
}

// Whether the implicit-GEMM kernel can only read a copy of an operand.
bool matmulCopies(const plb_matmul_desc &d, const void *a, const void *b) {
  const Ld ld = leadingDims(d);
  const size_t es = dtypeBytes(d.input_type);
  auto fits = [&](const void *base, long long pitch) {
    return (reinterpret_cast<uintptr_t>(base) & 15) == 0 && (size_t(pitch) * es) % 16 == 0;
  };
  return d.input_type == PLB_FLOAT || (d.input_type == PLB_QUARTER && (d.transpose_a || !d.transpose_b)) ||
         !fits(a, ld.a) || !fits(b, ld.b);
}

// The product that is contracted: float operands as three bfloat16 terms per product.
plb_matmul_desc contractionDesc(const plb_matmul_desc &d) {
  plb_matmul_desc q = d;
  if (d.input_type == PLB_FLOAT) {
    q.input_type = PLB_BFLOAT16;
    q.k = 3 * d.k;
  }
  return q;
}

// The pixels that a strided pointwise layer reads, where its input has to be copied.
bool readPixels(const plb_conv_params &p, const ConvShape &s, Repack::Lattice *sub) {
  if (!pointwise(s) || (s.strH == 1 && s.strW == 1) || s.tH != 0 || s.tW != 0) return false;
  *sub = Repack::Lattice{p.groups, uint32_t(latticeExtent(s.We, s.OWc, s.strW)),
                         uint32_t(latticeExtent(s.He, s.OHc, s.strH)), uint32_t(s.W), uint32_t(s.H),
                         uint32_t(s.strW), uint32_t(s.strH)};
  return uint64_t(p.batch) * sub->sub_h * sub->sub_w <= 0xffffffffull;
}

// Quarter weights of a pass that reduces over their rows: 8-bit operands have no
// MN-major form, so [G][tap][rows][cols] is transposed into
// [G][flipped tap][cols][rows -> pitch].
int transposedWeights(plb_context *ctx, const void *w, uint32_t groups, uint64_t taps, uint32_t rows, uint32_t cols,
                      const void **out, uint32_t *pitch) {
  *pitch = roundToRow(rows, 1);
  void *ws = nullptr;
  if (int rc = scratch(ctx, kSlotOperands, size_t(groups) * taps * cols * *pitch + 256, &ws)) return rc;
  *out = ws;
  return transposeFlipWeights(ctx, 1, groups, rows, cols, taps, *pitch, w, ws);
}

// Zeroes the pixels of [images][H][W] whose row phase (h mod str_h) or column phase
// (w mod str_w) is not in the masks, inside the window that starts at (h0, w0):
// the input positions of a strided layer that no output reads.  Only those are
// written (clearing the whole gradient first cost the layer 1x1, stride 2, 256
// images of 56x56x256 a third more bytes: 67 us of memset, now 50).  A block takes
// `each` pixels of a row: the rows of a 1-D layer are few and long.
template <typename V>
__global__ void __launch_bounds__(256)
zeroPhasesKernel(V *__restrict__ dst, uint32_t H, uint32_t W, uint32_t h0, uint32_t w0, uint32_t He, uint32_t We,
                 uint32_t str_h, uint32_t str_w, uint64_t rows_used, uint64_t cols_used, uint32_t vecs, uint32_t each) {
  // (in this order: the launches that follow write other positions and start beside
  // this one, but behind what came before it, see IgemmChain)
  pdl_wait();
  pdl_launch_dependents();
  const uint32_t h = blockIdx.x % He, n = blockIdx.x / He;
  V *row = dst + ((size_t(n) * H + h0 + h) * W + w0) * vecs;
  const bool all = !(rows_used >> (h % str_h) & 1);
  const uint32_t first = blockIdx.y * each, end = first + min(each, We - first);
  const V zero{};
  if (all) {
    for (size_t i = size_t(first) * vecs + threadIdx.x; i < size_t(end) * vecs; i += blockDim.x) row[i] = zero;
    return;
  }
  // a warp per pixel
  for (uint32_t w = first + threadIdx.x / 32; w < end; w += blockDim.x / 32)
    if (!(cols_used >> (w % str_w) & 1))
      for (uint32_t i = threadIdx.x & 31; i < vecs; i += 32) row[size_t(w) * vecs + i] = zero;
}

int zeroPhases(plb_context *ctx, void *dx, const plb_conv_params &p, const ConvShape &s, uint64_t rows_used,
               uint64_t cols_used) {
  const size_t pixel = size_t(p.groups) * p.in_chans_per_group * dtypeBytes(p.output_type);
  const uint64_t rows = uint64_t(p.batch) * s.He;
  // 64 KB a block, whole rows up to there
  const uint64_t each = std::max<uint64_t>({1, 65536 / pixel, (uint64_t(s.We) + 65534) / 65535});
  auto launch = [&](auto v) {
    using V = decltype(v);
    return launchPdl(ctx, zeroPhasesKernel<V>, dim3(unsigned(rows), unsigned((uint64_t(s.We) + each - 1) / each)), dim3(256),
                     0, static_cast<V *>(dx), uint32_t(s.H),
                     uint32_t(s.W), uint32_t(s.tH), uint32_t(s.tW), uint32_t(s.He), uint32_t(s.We), uint32_t(s.strH),
                     uint32_t(s.strW), rows_used, cols_used, uint32_t(pixel / sizeof(V)), uint32_t(each));
  };
  const size_t at = pixel | (reinterpret_cast<uintptr_t>(dx) & 15);
  if (at % 16 == 0) return launch(uint4());
  if (at % 4 == 0) return launch(uint32_t());
  return launch(uint16_t());
}

// The input gradient at the positions of phase (a, b): a stride-1 convolution of the
// output gradients with the phase's sub-filter.
IgemmProblem bwdPhaseProblem(const plb_conv_params &p, const plb_conv_options *opt, const ConvShape &s,
                             const PassOperands &o, void *dx, bool weights_transposed, int a, int b, const BwdPhase &A,
                             const BwdPhase &B) {
  const size_t os = dtypeBytes(p.output_type);
  const uint64_t ctot = uint64_t(p.groups) * p.in_chans_per_group;
  IgemmProblem r = convBwdProblem(p, opt, s, o, dx, weights_transposed);
  r.out_w = B.extent;
  r.out_h = A.extent;
  r.taps_h = A.taps;
  r.taps_w = B.taps;
  // tap j of the phase is used tap first + j*step of the (possibly flipped)
  // filter, stored where the flip, the truncation and (weights_transposed)
  // the reversal of all stored taps put it
  auto stored = [&](int used, int K, int Ks, int kt, int flip) {
    const int at = kt + (flip ? K - 1 - used : used);
    return weights_transposed ? Ks - 1 - at : at;
  };
  const int h0 = stored(A.first_tap, s.KH, s.KHs, s.ktH, s.flipH);
  const int w0 = stored(B.first_tap, s.KW, s.KWs, s.ktW, s.flipW);
  setTaps(&r, s, h0, (s.flipH != 0) != weights_transposed ? -A.step : A.step, w0,
          (s.flipW != 0) != weights_transposed ? -B.step : B.step);
  // position i of the phase reads output index i + offset - j*dil for its
  // j-th tap: a correlation with the taps reversed
  r.dil_h = A.dil;
  r.dil_w = B.dil;
  r.pad_h = (A.taps - 1) * A.dil - A.offset;
  r.pad_w = (B.taps - 1) * B.dil - B.offset;
  r.flip_h = 1;
  r.flip_w = 1;
  r.out = static_cast<uint8_t *>(dx) + (size_t(s.tH + a) * s.W + (s.tW + b)) * ctot * os;
  r.ldc = (long long)(ctot * s.strW);
  r.out_stride_h = (long long)(ctot * s.W * s.strH);
  return r;
}

// Backward pass of a strided convolution (the reference's getGradientParams
// gives the output gradients an input dilation equal to the forward stride,
// lib/poplin/ConvUtil.cpp:728-795).  Multiplying the inserted zeros would
// waste stride^2 of the work: instead the input gradient is computed per
// phase (ih mod stride_h, iw mod stride_w).  The positions of one phase see a
// fixed, evenly spaced subset of the filter taps (a sub-lattice of the stored
// filter), so each phase is a stride-1 convolution of the output gradients with
// that sub-filter, written to the strided sub-lattice of the input gradient.
// The phases write disjoint positions: they are one chain of launches (IgemmChain).
// `separate`: `p` contracts groups together; the outputs are repaired from these
// operands of the separate groups (`separate_p`).
int convBwdStrided(plb_context *ctx, const plb_conv_params &p, const plb_conv_options *opt, const ConvShape &s,
                   const PassOperands &o, void *dx, bool weights_transposed, const plb_conv_params *separate_p,
                   const PassOperands *separate) {
  const size_t os = dtypeBytes(p.output_type);
  const uint64_t ci = p.in_chans_per_group, ctot = uint64_t(p.groups) * ci;
  // phases and their taps
  std::vector<BwdPhase> ph(size_t(s.strH)), pw(size_t(s.strW));
  for (int a = 0; a < s.strH; ++a) bwdPhase(a, s.He, s.KH, s.padH, s.dilH, s.strH, &ph[size_t(a)]);
  for (int b = 0; b < s.strW; ++b) bwdPhase(b, s.We, s.KW, s.padW, s.dilW, s.strW, &pw[size_t(b)]);
  // positions no tap reaches get zero
  bool any_empty = false;
  uint64_t rows_used = 0, cols_used = 0;
  for (int a = 0; a < s.strH; ++a) {
    if (ph[size_t(a)].extent && ph[size_t(a)].taps == 0) any_empty = true;
    if (ph[size_t(a)].taps && a < 64) rows_used |= uint64_t(1) << a;
  }
  for (int b = 0; b < s.strW; ++b) {
    if (pw[size_t(b)].extent && pw[size_t(b)].taps == 0) any_empty = true;
    if (pw[size_t(b)].taps && b < 64) cols_used |= uint64_t(1) << b;
  }
  bool lead_done = false;
  if (any_empty && !s.zero_fill_in) {  // (otherwise the caller has cleared it)
    if (s.strH <= 64 && s.strW <= 64 && uint64_t(p.batch) * s.He <= 0x7fffffffull) {
      if (int rc = zeroPhases(ctx, dx, p, s, rows_used, cols_used)) return rc;
      lead_done = true;
    } else {
      PLB_CUDA(cudaMemsetAsync(dx, 0, size_t(p.batch) * s.H * s.W * ctot * os, ctx->stream));
    }
  }
  std::vector<std::pair<IgemmProblem, plb_plan>> phases;
  bool chain = true;
  for (int a = 0; a < s.strH; ++a)
    for (int b = 0; b < s.strW; ++b) {
      const BwdPhase &A = ph[size_t(a)], &B = pw[size_t(b)];
      if (A.extent == 0 || B.extent == 0 || A.taps == 0 || B.taps == 0) continue;
      IgemmProblem r = bwdPhaseProblem(p, opt, s, o, dx, weights_transposed, a, b, A, B);
      if (separate) r.nonfinite = nonfiniteFlag(ctx);
      r.plan_flags |= ctx->plan_flags;
      plb_plan plan{};
      if (int rc = planIgemm(r, ctx->sm_count, &plan)) return rc;
      if (plan.split_k > 1) chain = false;  // (the partial sums share one scratch buffer)
      phases.emplace_back(r, plan);
    }
  for (auto &[r, plan] : phases) {
    if (chain && phases.size() + (lead_done ? 1 : 0) > 1) r.chain = lead_done ? kChainFollow : kChainLead;
    lead_done = true;
    if (int rc = launchIgemm(ctx, r, plan)) return rc;
  }
  if (!separate || phases.empty()) return PLB_OK;
  return repairNonFinite(ctx, convBwdProblem(*separate_p, opt, s, *separate, dx, false), separate->type, s.strH, s.strW);
}

// Whether a pass runs on the patch kernel (patch.cu), and its problem(s); `o` are the
// caller's operands, `groups` those that the general route contracts together.
bool fwdOnPatches(int sm_count, const plb_conv_params &p, const plb_conv_options *opt, int plan_flags, const ConvShape &s,
                  const PassOperands &o, const float *bias, void *out, bool swapped, int groups, bool slower_too, IgemmProblem *r,
                  RowsTiling *rows) {
  if ((!pointwise(s) && (s.strH > 8 || s.strW > 8)) || s.KH <= 0 || s.KW <= 0) return false;
  *r = convFwdProblem(p, opt, s, o, bias, out, swapped);
  r->plan_flags |= plan_flags;
  const bool packed = p.groups == 1 && p.input_type != PLB_FLOAT && !swapped && !channelsFitTma(p, p.in_chans_per_group);
  return patchSuits(sm_count, r, 1, p.input_type, 1, groups, operandsCopied(o, p.in_chans_per_group), packed, slower_too, rows);
}
// The one-launch routes of a forward pass, tried before the others: straight from the image
// (`shape`), or on the patch kernel (`r`) or that for rows in its place (`rows`).  `slower_too`: where the others would be quicker, but
// cannot have the scratch memory that they need.
enum class FwdRoute { kOther, kStem, kPatch };
FwdRoute fwdRoute(int sm_count, const plb_conv_params &p, const plb_conv_options *opt, int plan_flags, const ConvShape &s,
                  const PassOperands &o, const float *bias, void *out, bool swapped, int groups, bool slower_too, IgemmProblem *r,
                  RowsTiling *rows, S2dShape *shape) {
  if (is16BitFloat(p.input_type) && p.groups == 1 && !channelsFitTma(p, p.in_chans_per_group) && !swapped &&
      stemLayer(sm_count, plan_flags, p, opt, out, slower_too, shape))
    return FwdRoute::kStem;
  return fwdOnPatches(sm_count, p, opt, plan_flags, s, o, bias, out, swapped, groups, slower_too, r, rows) ? FwdRoute::kPatch : FwdRoute::kOther;
}
// (the number of problems, 0 if it does not)
int bwdOnPatches(int sm_count, const plb_conv_params &p, const plb_conv_options *opt, int plan_flags, const ConvShape &s,
                 const PassOperands &o, void *dx, int groups, bool slower_too, IgemmProblem *r, RowsTiling *rows) {
  int n = 0, contractions = 0;
  if (s.strH == 1 && s.strW == 1) {
    r[n++] = convBwdProblem(p, opt, s, o, dx, false);
    contractions = 1;
  } else if (s.strH * s.strW <= kPatchMaxPhases) {
    // (a phase that no tap reaches is a sum of nothing: it is cleared by the same launch;
    // the general route clears all such phases in one)
    bool clears = false;
    for (int a = 0; a < s.strH; ++a)
      for (int b = 0; b < s.strW; ++b) {
        BwdPhase A, B;
        bwdPhase(a, s.He, s.KH, s.padH, s.dilH, s.strH, &A);
        bwdPhase(b, s.We, s.KW, s.padW, s.dilW, s.strW, &B);
        if (A.extent <= 0 || B.extent <= 0) continue;
        r[n++] = bwdPhaseProblem(p, opt, s, o, dx, false, a, b, A, B);
        if (A.taps == 0 || B.taps == 0)
          clears = true;
        else
          ++contractions;
      }
    contractions += clears ? 1 : 0;
  }
  if (n == 0) return 0;
  r[0].plan_flags |= plan_flags;
  return patchSuits(sm_count, r, n, p.input_type, contractions, groups, operandsCopied(o, p.out_chans_per_group), false, slower_too, rows) ? n : 0;
}

// Narrow channel groups are contracted together (grouped.cu): `q` = the layer of
// wider groups and its weights, [G][taps][rows][cols] made block-diagonal.
// Returns whether it applies through `together`.
int gatherGroups(plb_context *ctx, const plb_conv_params &p, const ConvShape &s, const void *weights, bool rows_are_co,
                 plb_conv_params *q, const void **out, bool *together) {
  *q = p;
  *out = weights;
  const uint32_t ci = p.in_chans_per_group, co = p.out_chans_per_group;
  const uint32_t S = groupsTogether(p.groups, ci, co, p.input_type);
  *together = S > 1;
  if (S == 1) return PLB_OK;
  q->groups = p.groups / S;
  q->in_chans_per_group = S * ci;
  q->out_chans_per_group = S * co;
  return blockDiagonalWeights(ctx, p.input_type, weights, p.groups, S, uint32_t(s.KHs * s.KWs), rows_are_co ? co : ci,
                              rows_are_co ? ci : co, out);
}

// The product by way of the implicit-GEMM kernel: operands transposed and copied as it needs them.
int matmulGeneral(plb_context *ctx, const plb_matmul_desc &d, const Ld &ld, const void *d_a, const void *d_b, const void *d_c,
                  void *d_d) {
  // Operand layouts the kernel takes directly: A as [m][k], B as [n][k], or (not
  // 8-bit) A as [k][m] and B as [k][n].  8-bit operands stored the other way go
  // through a transpose into scratch.
  const void *a = d_a, *b = d_b;
  long long lda = ld.a, ldb = ld.b;
  bool a_is_km = d.transpose_a != 0, b_is_nk = d.transpose_b != 0;
  if (d.input_type == PLB_QUARTER && (a_is_km || !b_is_nk)) {
    // (rows of whole 16-byte vectors, so that nothing has to be copied again)
    const uint64_t pitch = roundToRow(d.k, 1);
    const size_t a_bytes = a_is_km ? (size_t(d.groups) * d.m * pitch + 255) & ~size_t(255) : 0;
    const size_t b_bytes = b_is_nk ? 0 : size_t(d.groups) * d.n * pitch;
    void *ws = nullptr;
    if (int rc = scratch(ctx, kSlotOperands, a_bytes + b_bytes, &ws)) return rc;
    if (a_is_km) {
      if (int rc = transposeBatch(ctx, 1, d.groups, d.k, d.m, d_a, ws, pitch)) return rc;
      a = ws;
      lda = (long long)pitch;
      a_is_km = false;
    }
    if (!b_is_nk) {
      uint8_t *bt = static_cast<uint8_t *>(ws) + a_bytes;
      if (int rc = transposeBatch(ctx, 1, d.groups, d.k, d.n, d_b, bt, pitch)) return rc;
      b = bt;
      ldb = (long long)pitch;
      b_is_nk = true;
    }
  }
  // Operands whose rows TMA cannot address (base or row pitch not a multiple of
  // 16 bytes: n % 8 != 0, odd leading dimensions) are copied once into scratch
  // with the pitch rounded up, float operands are split into their bfloat16
  // pieces, both operands in one launch.  The output needs no such copy.
  Copies copies = planCopies(d, &a, &lda, a_is_km, &b, &ldb, b_is_nk);
  if (int rc = runCopies(ctx, copies)) return rc;
  const plb_matmul_desc q = contractionDesc(d);
  IgemmProblem p = gemmProblem(q, a, lda, a_is_km, b, ldb, b_is_nk, d_c, d_d, ld.c);
  return runProblem(ctx, p);
}

// The passes by way of the implicit-GEMM kernel: operands gathered and copied as it needs them.
int convFwdGeneral(plb_context *ctx, const plb_conv_params *p, const plb_conv_options *opt, const ConvShape &s,
                   const PassOperands &separate, const void *d_in, const void *d_weights, const float *d_bias, void *d_out,
                   bool swapped) {
  if (p->input_type != PLB_FLOAT && !channelsFitTma(*p, p->in_chans_per_group) && !swapped) {
    // few input channels (a stem): space-to-depth path, where it applies
    const int rc = convFwdSmallChannels(ctx, *p, opt, d_in, d_weights, d_bias, d_out, nullptr);
    if (rc != PLB_ERR_UNSUPPORTED) return rc;
  }
  if (s.strH > 1 || s.strW > 1) {
    if (!pointwise(s) && (s.strH > 8 || s.strW > 8))
      return fail(PLB_ERR_UNSUPPORTED, "strides above 8 are not implemented for k > 1");
  }
  if (s.KH <= 0 || s.KW <= 0) {
    // every tap is truncated away: the result is zero
    PLB_CUDA(cudaMemsetAsync(d_out, 0,
                             size_t(p->batch) * s.OH * s.OW * p->groups * p->out_chans_per_group *
                                 dtypeBytes(p->output_type),
                             ctx->stream));
    return PLB_OK;
  }
  plb_conv_params q;
  const void *w = nullptr;
  bool together = false;
  // stored [G][k][Ci][Co] when swapped, else [G][k][Co][Ci]
  if (int rc = gatherGroups(ctx, *p, s, d_weights, !swapped, &q, &w, &together)) return rc;
  const uint64_t in_rows = uint64_t(q.batch) * s.H * s.W * q.groups, tiles = uint64_t(q.groups) * s.KHs * s.KWs;
  const uint32_t ci = q.in_chans_per_group, co = q.out_chans_per_group;
  const bool transposed = swapped && q.input_type == PLB_QUARTER;  // -> [G][flipped k][Co][Ci]
  Repack::Lattice sub{};
  const Repack::Lattice *lattice = readPixels(q, s, &sub) ? &sub : nullptr;
  PassOperands o;
  if (transposed) {
    uint32_t pitch = 0;
    if (int rc = transposedWeights(ctx, w, q.groups, uint64_t(s.KHs) * s.KWs, ci, co, &w, &pitch)) return rc;
    if (int rc = prepareOperands(ctx, q.input_type, d_in, in_rows, ci, w, tiles * co, pitch, 0, &o, lattice)) return rc;
  } else if (swapped) {
    // the reduction along the rows
    if (int rc = prepareOperands(ctx, q.input_type, d_in, in_rows, ci, w, tiles * ci, co, ci, &o, lattice)) return rc;
  } else {
    if (int rc = prepareOperands(ctx, q.input_type, d_in, in_rows, ci, w, tiles * co, ci, 0, &o, lattice)) return rc;
  }
  IgemmProblem r = convFwdProblem(q, opt, s, o, d_bias, d_out, swapped && !transposed, transposed);
  if (together) r.nonfinite = nonfiniteFlag(ctx);
  if (int rc = runProblem(ctx, r)) return rc;
  if (!together) return PLB_OK;
  return repairNonFinite(ctx, convFwdProblem(*p, opt, s, separate, d_bias, d_out, swapped), p->input_type);
}

int convBwdGeneral(plb_context *ctx, const plb_conv_params *p, const plb_conv_options *opt, const ConvShape &s,
                   const PassOperands &separate, const void *d_out_grads, const void *d_weights, void *d_in_grads) {
  plb_conv_params q;
  const void *w = nullptr;
  bool together = false;
  if (int rc = gatherGroups(ctx, *p, s, d_weights, true, &q, &w, &together)) return rc;
  const uint64_t out_rows = uint64_t(q.batch) * s.OH * s.OW * q.groups, tiles = uint64_t(q.groups) * s.KHs * s.KWs;
  const uint32_t ci = q.in_chans_per_group, co = q.out_chans_per_group;
  PassOperands o;
  const bool transposed = q.input_type == PLB_QUARTER;
  if (transposed) {
    uint32_t pitch = 0;
    // [G][k][Co][Ci] -> [G][flipped k][Ci][Co]
    if (int rc = transposedWeights(ctx, w, q.groups, uint64_t(s.KHs) * s.KWs, co, ci, &w, &pitch)) return rc;
    if (int rc = prepareOperands(ctx, q.input_type, d_out_grads, out_rows, co, w, tiles * ci, pitch, 0, &o)) return rc;
  } else {
    // the reduction runs over the output channels, the rows of a weight tile
    if (int rc = prepareOperands(ctx, q.input_type, d_out_grads, out_rows, co, w, tiles * co, ci, co, &o)) return rc;
  }
  if (s.strH != 1 || s.strW != 1)
    return convBwdStrided(ctx, q, opt, s, o, d_in_grads, transposed, p, together ? &separate : nullptr);
  IgemmProblem r = convBwdProblem(q, opt, s, o, d_in_grads, transposed);
  if (together) r.nonfinite = nonfiniteFlag(ctx);
  if (int rc = runProblem(ctx, r)) return rc;
  if (!together) return PLB_OK;
  return repairNonFinite(ctx, convBwdProblem(*p, opt, s, separate, d_in_grads, false), p->input_type);
}

}  // namespace
}  // namespace plb

using namespace plb;

extern "C" {

int plb_matmul_plan(const plb_matmul_desc *desc, plb_plan *plan) {
  if (!desc || !plan) return fail(PLB_ERR_INVALID_PARAMS, "null argument");
  if (int rc = checkMatmulDesc(*desc)) return rc;
  *plan = plb_plan{};
  plan->flops = 2ull * desc->groups * desc->m * desc->k * desc->n;
  plan->bytes = gemmBytes(*desc);
  if (desc->groups == 0 || desc->m == 0 || desc->n == 0 || desc->k == 0) return PLB_OK;
  const Ld ld = leadingDims(*desc);
  const bool b_is_nk = desc->transpose_b || desc->input_type == PLB_QUARTER;
  const bool a_is_km = desc->transpose_a && desc->input_type != PLB_QUARTER;
  // quarter operands stored the other way are transposed, rows that TMA cannot address copied
  const void *a = nullptr, *b = nullptr;  // (as aligned as they need to be)
  long long lda = ld.a, ldb = ld.b;
  const uint64_t pitch = roundToRow(desc->k, 1);
  size_t transposed = 0;
  if (desc->transpose_a && !a_is_km) {
    transposed += (size_t(desc->groups) * desc->m * pitch + 255) & ~size_t(255);
    lda = (long long)pitch;
  }
  if (!desc->transpose_b && b_is_nk) {
    transposed += size_t(desc->groups) * desc->n * pitch;
    ldb = (long long)pitch;
  }
  const Copies copies = planCopies(*desc, &a, &lda, a_is_km, &b, &ldb, b_is_nk);
  const IgemmProblem p =
      gemmProblem(contractionDesc(*desc), nullptr, lda, a_is_km, nullptr, ldb, b_is_nk, nullptr, nullptr, ld.c);
  if (int rc = planIgemm(p, 148, plan)) return rc;
  plan->workspace_bytes += transposed + copies.bytes;
  const IgemmProblem direct = gemmProblem(*desc, nullptr, ld.a, desc->transpose_a != 0, nullptr, ld.b, desc->transpose_b != 0,
                                          nullptr, nullptr, ld.c);
  if (directSuits(148, direct, desc->input_type, matmulCopies(*desc, nullptr, nullptr), false)) {
    plan->kernel = 3;
    plan->in_place = 1;
  }
  return PLB_OK;
}

int plb_matmul(plb_context *ctx, const plb_matmul_desc *desc, const void *d_a, const void *d_b,
               const void *d_c, void *d_d) {
  TraceRange trace_range("plb_matmul");
  if (int rc = activate(ctx)) return rc;
  if (!desc) return fail(PLB_ERR_INVALID_PARAMS, "null descriptor");
  const plb_matmul_desc &d = *desc;
  if (int rc = checkMatmulDesc(d)) return rc;
  if (d.groups == 0 || d.m == 0 || d.n == 0) return PLB_OK;
  if (d.beta != 0.f && d_c == nullptr)
    return fail(PLB_ERR_INVALID_PARAMS, "beta != 0 needs a C matrix");
  if (d_d == nullptr || (d.k != 0 && (d_a == nullptr || d_b == nullptr)))
    return fail(PLB_ERR_INVALID_PARAMS, "null device pointer for a matrix that has elements");
  const Ld ld = leadingDims(d);
  const size_t os = dtypeBytes(d.output_type);
  if (d.k == 0) {
    // empty reduction: D = beta * C
    for (uint32_t g = 0; g < d.groups; ++g) {
      const size_t off = size_t(g) * d.m * ld.c * os;
      if (int rc = launchScaleRows(ctx, static_cast<uint8_t *>(d_d) + off,
                                   d_c ? static_cast<const uint8_t *>(d_c) + off : nullptr,
                                   d.beta, d.output_type == PLB_FLOAT, d.m, d.n, ld.c, ld.c))
        return rc;
    }
    return PLB_OK;
  }
  if (d.input_type == PLB_FLOAT && (ld.a < (long long)(d.transpose_a ? d.m : d.k) || ld.b < (long long)(d.transpose_b ? d.k : d.n)))
    return fail(PLB_ERR_INVALID_PARAMS, "leading dimension shorter than a row");
  if (d.input_type == PLB_QUARTER && d.transpose_a && ld.a != (long long)d.m)
    return fail(PLB_ERR_UNSUPPORTED, "transposed quarter A must be densely packed");
  if (d.input_type == PLB_QUARTER && !d.transpose_b && ld.b != (long long)d.n)
    return fail(PLB_ERR_UNSUPPORTED, "quarter B in [k][n] layout must be densely packed");
  // small products, and moderate ones that would need a copy, from the operands as they are
  IgemmProblem p = gemmProblem(d, d_a, ld.a, d.transpose_a != 0, d_b, ld.b, d.transpose_b != 0, d_c, d_d, ld.c);
  p.plan_flags = ctx->plan_flags;
  const bool copied = matmulCopies(d, d_a, d_b);
  if (directSuits(ctx->sm_count, p, d.input_type, copied, false)) return launchDirect(ctx, p, d.input_type);
  ctx->scratch_refused = false;
  const int rc = matmulGeneral(ctx, d, ld, d_a, d_b, d_c, d_d);
  if (rc && ctx->scratch_refused && directSuits(ctx->sm_count, p, d.input_type, copied, true)) return launchDirect(ctx, p, d.input_type);
  return rc;
}

int plb_matmul_host(plb_context *ctx, const plb_matmul_desc *desc, const void *h_a,
                    const void *h_b, const void *h_c, void *h_d) {
  if (int rc = plb_matmul_host_async(ctx, desc, h_a, h_b, h_c, h_d)) return rc;
  return plb_synchronize(ctx);
}

int plb_matmul_host_async(plb_context *ctx, const plb_matmul_desc *desc, const void *h_a,
                          const void *h_b, const void *h_c, void *h_d) {
  if (int rc = activate(ctx)) return rc;
  if (!desc) return fail(PLB_ERR_INVALID_PARAMS, "null descriptor");
  const plb_matmul_desc &d = *desc;
  if (int rc = checkMatmulDesc(d)) return rc;
  const Ld ld = leadingDims(d);
  const size_t es = dtypeBytes(d.input_type), os = dtypeBytes(d.output_type);
  const size_t a_bytes = size_t(d.groups) * (d.transpose_a ? d.k : d.m) * ld.a * es;
  const size_t b_bytes = size_t(d.groups) * (d.transpose_b ? d.n : d.k) * ld.b * es;
  const size_t c_bytes = size_t(d.groups) * d.m * ld.c * os;
  void *da = nullptr, *db = nullptr, *dc = nullptr, *dd = nullptr;
  if (int rc = scratch(ctx, kSlotHostIn, a_bytes + 16, &da)) return rc;
  if (int rc = scratch(ctx, kSlotHostWeights, b_bytes + 16, &db)) return rc;
  if (int rc = scratch(ctx, kSlotHostOut, c_bytes + 16, &dd)) return rc;
  if (d.beta != 0.f) {
    if (!h_c) return fail(PLB_ERR_INVALID_PARAMS, "beta != 0 needs a C matrix");
    if (int rc = scratch(ctx, kSlotHostBias, c_bytes + 16, &dc)) return rc;
    if (int rc = plb_memcpy_h2d(ctx, dc, h_c, c_bytes)) return rc;
  }
  if (int rc = plb_memcpy_h2d(ctx, da, h_a, a_bytes)) return rc;
  if (int rc = plb_memcpy_h2d(ctx, db, h_b, b_bytes)) return rc;
  if (int rc = plb_matmul(ctx, desc, da, db, dc, dd)) return rc;
  // enqueued only: the caller synchronises (plb_synchronize) before reading h_d
  if (c_bytes) PLB_CUDA(cudaMemcpyAsync(h_d, dd, c_bytes, cudaMemcpyDeviceToHost, ctx->stream));
  return PLB_OK;
}

// ---------------------------------------------------------------------------

int plb_conv_validate(const plb_conv_params *p) {
  if (!p) return fail(PLB_ERR_INVALID_PARAMS, "null params");
  const std::string err = validate(*p);
  return err.empty() ? PLB_OK : fail(PLB_ERR_INVALID_PARAMS, err);
}

int plb_conv_output_field(const plb_conv_params *p, uint32_t out_field[PLB_MAX_FIELD_DIMS]) {
  if (int rc = plb_conv_validate(p)) return rc;
  for (unsigned d = 0; d != p->num_field_dims; ++d) out_field[d] = uint32_t(outputSize(*p, d));
  return PLB_OK;
}

int plb_conv_input_index(const plb_conv_params *p, uint32_t dim, uint32_t out_index,
                         uint32_t kernel_index) {
  if (!p || dim >= p->num_field_dims) return -1;
  return inputIndex(*p, dim, out_index, kernel_index);
}

uint64_t plb_conv_macs(const plb_conv_params *p) { return p ? numberOfMacs(*p) : 0; }

int plb_conv_plan(const plb_conv_params *p_in, const plb_conv_options *opt, int32_t pass,
                  plb_plan *plan) {
  if (!p_in || !plan) return fail(PLB_ERR_INVALID_PARAMS, "null argument");
  if (p_in->num_field_dims == 3) return conv3dPlan(*p_in, opt, pass, plan);
  // a flipped input runs as the ordinary convolution of the reversed tensor
  plb_conv_params unflipped, undilated;
  const plb_conv_params *p = unflippedInputParams(*p_in, &unflipped) ? &unflipped : p_in;
  DilatedField df;
  // a dilated input runs as the ordinary convolution of the zero-stuffed tensor
  if (undilatedInputParams(*p, &undilated, &df)) p = &undilated;
  ConvShape s;
  if (int rc = igemmConvShape(*p, &s)) return rc;
  *plan = plb_plan{};
  const bool bwd = pass == PLB_PASS_TRAINING_BWD;
  bool rearranged = false;
  if (!bwd && p->input_type != PLB_FLOAT && !channelsFitTma(*p, p->in_chans_per_group)) {
    const int rc = convFwdSmallChannels(nullptr, *p, opt, nullptr, nullptr, nullptr, nullptr, plan);
    rearranged = rc == PLB_OK;
    if (!rearranged && rc != PLB_ERR_UNSUPPORTED) return rc;
  }
  // narrow groups run together; channel counts TMA cannot address and float operands on copies
  plb_conv_params run = *p;
  const uint32_t together = groupsTogether(p->groups, p->in_chans_per_group, p->out_chans_per_group, p->input_type);
  run.groups /= together;
  run.in_chans_per_group *= together;
  run.out_chans_per_group *= together;
  const bool transposed = bwd && run.input_type == PLB_QUARTER;
  const uint64_t tiles = uint64_t(run.groups) * s.KHs * s.KWs, pixels = uint64_t(run.batch) * run.groups;
  const uint32_t ci = run.in_chans_per_group, co = run.out_chans_per_group;
  if (!rearranged && run.batch != 0 && run.groups != 0 && ci != 0 && co != 0 && s.KH > 0 && s.KW > 0 && s.OHc > 0 && s.OWc > 0 &&
      s.He > 0 && s.We > 0) {
    PassOperands o;
    Repack::Lattice sub{};
    const uint32_t pitch = transposed ? roundToRow(co, 1) : ci;
    const Copies copies =
        bwd ? planOperands(run.input_type, nullptr, pixels * s.OH * s.OW, co, nullptr, transposed ? tiles * ci : tiles * co,
                           pitch, transposed ? 0 : co, &o)
            : planOperands(run.input_type, nullptr, pixels * s.H * s.W, ci, nullptr, tiles * co, ci, 0, &o,
                           readPixels(run, s, &sub) ? &sub : nullptr);
    const IgemmProblem q = bwd ? convBwdProblem(run, opt, s, o, nullptr, transposed)
                               : convFwdProblem(run, opt, s, o, nullptr, nullptr);
    if (int rc = planIgemm(q, 148, plan)) return rc;
    const size_t es = dtypeBytes(run.input_type);
    plan->workspace_bytes += copies.bytes;
    if (transposed) plan->workspace_bytes += tiles * ci * pitch;
    if (together > 1) plan->workspace_bytes += size_t(tiles) * ci * co * es;  // block-diagonal weights
  }
  if (plan->tiles > 0) {
    IgemmProblem r[kPatchMaxPhases];
    const PassOperands o{p->input_type, nullptr, nullptr, bwd ? p->out_chans_per_group : p->in_chans_per_group,
                         bwd ? p->out_chans_per_group : p->in_chans_per_group, p->in_chans_per_group};
    S2dShape g;
    RowsTiling rows;
    FwdRoute route = FwdRoute::kOther;
    if (!bwd)
      route = fwdRoute(148, *p, opt, 0, s, o, nullptr, nullptr, false, int(together), false, r, &rows, &g);
    else if (bwdOnPatches(148, *p, opt, 0, s, o, nullptr, int(together), false, r, &rows) > 0)
      route = FwdRoute::kPatch;
    if (route == FwdRoute::kPatch) plan->kernel = 3;
    plan->in_place = route == FwdRoute::kOther ? 0 : 1;
  }
  plan->flops = 2 * numberOfMacs(*p);
  plan->bytes = convBytes(*p, s, pass);
  return PLB_OK;
}

int plb_convolution(plb_context *ctx, const plb_conv_params *p, const plb_conv_options *opt,
                    const void *d_in, const void *d_weights, const float *d_bias, void *d_out,
                    int transpose_and_flip_weights) {
  TraceRange trace_range("plb_convolution");
  if (int rc = activate(ctx)) return rc;
  if (!p) return fail(PLB_ERR_INVALID_PARAMS, "null params");
  {
    size_t n_in, n_w, n_out;
    convElementCounts(*p, &n_in, &n_w, &n_out);
    if (n_in == 0 || n_w == 0) n_in = n_w = 0;  // nothing is read: the output is zero (or the bias)
    if (int rc = checkConvRequest(*p, false, d_in, n_out ? n_in : 0, d_weights, n_out ? n_w : 0, d_out, n_out))
      return rc;
  }
  if (p->num_field_dims == 3)
    return conv3dFwd(ctx, *p, opt, d_in, d_weights, d_bias, d_out, transpose_and_flip_weights);
  {
    // a flipped input: reverse it once, then an ordinary convolution
    plb_conv_params q;
    if (unflippedInputParams(*p, &q) && p->num_field_dims <= 2) {
      const std::string err = validate(*p);
      if (!err.empty()) return fail(PLB_ERR_INVALID_PARAMS, err);
      const bool two = p->num_field_dims == 2;
      const uint32_t H = two ? p->field[0] : 1, W = p->field[two ? 1 : 0];
      const size_t px = size_t(p->groups) * p->in_chans_per_group * dtypeBytes(p->input_type);
      void *xf = nullptr;
      if (int rc = scratch(ctx, kSlotFlipped, size_t(p->batch) * H * W * px + 256, &xf)) return rc;
      if (int rc = flipField(ctx, d_in, xf, p->batch, H, W, px, two && p->in_flip[0],
                             p->in_flip[two ? 1 : 0] != 0))
        return rc;
      return plb_convolution(ctx, &q, opt, xf, d_weights, d_bias, d_out, transpose_and_flip_weights);
    }
  }
  {
    // a dilated input: write the zero-stuffed tensor once
    plb_conv_params q;
    DilatedField df;
    if (undilatedInputParams(*p, &q, &df)) {
      const std::string err = validate(*p);
      if (!err.empty()) return fail(PLB_ERR_INVALID_PARAMS, err);
      const size_t px = size_t(p->groups) * p->in_chans_per_group * dtypeBytes(p->input_type);
      void *xd = nullptr;
      if (int rc = scratch(ctx, kSlotDilated, size_t(p->batch) * df.Hd * df.Wd * px + 256, &xd)) return rc;
      if (int rc = dilateField(ctx, d_in, xd, p->batch, df, px, false)) return rc;
      return plb_convolution(ctx, &q, opt, xd, d_weights, d_bias, d_out, transpose_and_flip_weights);
    }
  }
  ConvShape s;
  if (int rc = igemmConvShape(*p, &s)) return rc;
  if (p->batch == 0 || p->groups == 0 || p->out_chans_per_group == 0 || s.OH == 0 || s.OW == 0)
    return PLB_OK;
  if (p->in_chans_per_group == 0)
    return fail(PLB_ERR_UNSUPPORTED, "zero input channels are not implemented on this path yet");
  if (s.zero_fill_out || s.OHc <= 0 || s.OWc <= 0 || s.He <= 0 || s.We <= 0) {
    // padded output positions (and everything, if nothing is computed) hold
    // zero, or the bias alone
    const size_t chans = size_t(p->groups) * p->out_chans_per_group;
    const size_t total = size_t(p->batch) * s.OH * s.OW * chans;
    if (d_bias) {
      const int grid = int(std::min<size_t>((total + 255) / 256, size_t(ctx->sm_count) * 16));
      if (p->output_type == PLB_FLOAT)
        fillBiasKernel<float><<<grid, 256, 0, ctx->stream>>>(static_cast<float *>(d_out), d_bias, total, chans);
      else
        fillBiasKernel<__half><<<grid, 256, 0, ctx->stream>>>(static_cast<__half *>(d_out), d_bias, total, chans);
      PLB_CUDA(cudaGetLastError());
      ctx->launches++;
    } else {
      PLB_CUDA(cudaMemsetAsync(d_out, 0, total * dtypeBytes(p->output_type), ctx->stream));
    }
    if (s.OHc <= 0 || s.OWc <= 0 || s.He <= 0 || s.We <= 0) return PLB_OK;
  }
  const bool swapped = transpose_and_flip_weights != 0;
  // the caller's operands, the groups apart
  const PassOperands separate{p->input_type, d_in, d_weights, p->in_chans_per_group, p->in_chans_per_group,
                              swapped ? p->out_chans_per_group : p->in_chans_per_group};
  // in one launch, without scratch, where that is quicker, or where scratch cannot be had
  auto inPlace = [&](bool slower_too, int *rc) {
    IgemmProblem r;
    RowsTiling rows;
    S2dShape g;
    const int groups = groupsTogether(p->groups, p->in_chans_per_group, p->out_chans_per_group, p->input_type);
    const FwdRoute route =
        fwdRoute(ctx->sm_count, *p, opt, ctx->plan_flags, s, separate, d_bias, d_out, swapped, groups, slower_too, &r, &rows, &g);
    if (route == FwdRoute::kStem)
      *rc = launchStem(ctx, g, int(p->out_chans_per_group), p->input_type == PLB_BFLOAT16, d_in, d_weights, d_bias, d_out);
    else if (route == FwdRoute::kPatch)
      *rc = rows.blocks ? launchRows(ctx, r, rows) : launchPatch(ctx, &r, 1, p->input_type, groups > 1);
    return route != FwdRoute::kOther;
  };
  int done = PLB_OK;
  if (inPlace(false, &done)) return done;
  ctx->scratch_refused = false;
  const int rc = convFwdGeneral(ctx, p, opt, s, separate, d_in, d_weights, d_bias, d_out, swapped);
  if (rc == PLB_OK || !ctx->scratch_refused) return rc;
  const std::string why = plb_last_error();
  return inPlace(true, &done) ? done : fail(rc, why);
}

int plb_conv_fwd(plb_context *ctx, const plb_conv_params *p, const plb_conv_options *opt,
                 const void *d_in, const void *d_weights, const float *d_bias, void *d_out) {
  return plb_convolution(ctx, p, opt, d_in, d_weights, d_bias, d_out, 0);
}

int plb_conv_bwd(plb_context *ctx, const plb_conv_params *p, const plb_conv_options *opt,
                 const void *d_out_grads, const void *d_weights, void *d_in_grads) {
  TraceRange trace_range("plb_conv_bwd");
  if (int rc = activate(ctx)) return rc;
  if (!p) return fail(PLB_ERR_INVALID_PARAMS, "null params");
  {
    size_t n_in, n_w, n_out;
    convElementCounts(*p, &n_in, &n_w, &n_out);
    if (n_out == 0 || n_w == 0) n_out = n_w = 0;  // nothing is read: the gradient is zero
    if (int rc = checkConvRequest(*p, false, d_out_grads, n_in ? n_out : 0, d_weights, n_in ? n_w : 0,
                                  d_in_grads, n_in))
      return rc;
  }
  if (p->num_field_dims == 3) return conv3dBwd(ctx, *p, opt, d_out_grads, d_weights, d_in_grads);
  {
    // a flipped input: the gradient of the reversed input, reversed back
    plb_conv_params q;
    if (unflippedInputParams(*p, &q) && p->num_field_dims <= 2) {
      const std::string err = validate(*p);
      if (!err.empty()) return fail(PLB_ERR_INVALID_PARAMS, err);
      const bool two = p->num_field_dims == 2;
      const uint32_t H = two ? p->field[0] : 1, W = p->field[two ? 1 : 0];
      const size_t px = size_t(p->groups) * p->in_chans_per_group * dtypeBytes(p->output_type);
      void *gf = nullptr;
      if (int rc = scratch(ctx, kSlotFlipped, size_t(p->batch) * H * W * px + 256, &gf)) return rc;
      if (int rc = plb_conv_bwd(ctx, &q, opt, d_out_grads, d_weights, gf)) return rc;
      return flipField(ctx, gf, d_in_grads, p->batch, H, W, px, two && p->in_flip[0],
                       p->in_flip[two ? 1 : 0] != 0);
    }
  }
  {
    // a dilated input: the gradient of the zero-stuffed tensor,
    // of which the lattice elements are the gradient of the input
    plb_conv_params q;
    DilatedField df;
    if (undilatedInputParams(*p, &q, &df)) {
      const std::string err = validate(*p);
      if (!err.empty()) return fail(PLB_ERR_INVALID_PARAMS, err);
      const size_t px = size_t(p->groups) * p->in_chans_per_group * dtypeBytes(p->output_type);
      void *gd = nullptr;
      if (int rc = scratch(ctx, kSlotDilated, size_t(p->batch) * df.Hd * df.Wd * px + 256, &gd)) return rc;
      if (int rc = plb_conv_bwd(ctx, &q, opt, d_out_grads, d_weights, gd)) return rc;
      return dilateField(ctx, gd, d_in_grads, p->batch, df, px, true);
    }
  }
  ConvShape s;
  if (int rc = igemmConvShape(*p, &s)) return rc;
  if (p->batch == 0 || p->groups == 0 || p->in_chans_per_group == 0 || s.H == 0 || s.W == 0)
    return PLB_OK;
  if (s.zero_fill_in)  // truncated input positions receive no gradient
    PLB_CUDA(cudaMemsetAsync(d_in_grads, 0,
                             size_t(p->batch) * s.H * s.W * p->groups * p->in_chans_per_group *
                                 dtypeBytes(p->output_type),
                             ctx->stream));
  if (s.OHc <= 0 || s.OWc <= 0 || s.He <= 0 || s.We <= 0) {
    if (!s.zero_fill_in)
      PLB_CUDA(cudaMemsetAsync(d_in_grads, 0,
                               size_t(p->batch) * s.H * s.W * p->groups * p->in_chans_per_group *
                                   dtypeBytes(p->output_type),
                               ctx->stream));
    return PLB_OK;
  }
  if (s.KH <= 0 || s.KW <= 0) {
    if (!s.zero_fill_in)
      PLB_CUDA(cudaMemsetAsync(d_in_grads, 0,
                               size_t(p->batch) * s.H * s.W * p->groups * p->in_chans_per_group *
                                   dtypeBytes(p->output_type),
                               ctx->stream));
    return PLB_OK;
  }
  // the caller's operands, the groups apart
  const PassOperands separate{p->input_type, d_out_grads, d_weights, p->out_chans_per_group, p->out_chans_per_group,
                              p->in_chans_per_group};
  // in one launch, without scratch, where that is quicker, or where scratch cannot be had
  auto inPlace = [&](bool slower_too, int *rc) {
    IgemmProblem r[kPatchMaxPhases];
    RowsTiling rows;
    const int groups = groupsTogether(p->groups, p->in_chans_per_group, p->out_chans_per_group, p->input_type);
    const int n = bwdOnPatches(ctx->sm_count, *p, opt, ctx->plan_flags, s, separate, d_in_grads, groups, slower_too, r, &rows);
    if (n > 0) *rc = rows.blocks ? launchRows(ctx, *r, rows) : launchPatch(ctx, r, n, p->input_type, groups > 1);
    return n > 0;
  };
  int done = PLB_OK;
  if (inPlace(false, &done)) return done;
  ctx->scratch_refused = false;
  const int rc = convBwdGeneral(ctx, p, opt, s, separate, d_out_grads, d_weights, d_in_grads);
  if (rc == PLB_OK || !ctx->scratch_refused) return rc;
  const std::string why = plb_last_error();
  return inPlace(true, &done) ? done : fail(rc, why);
}

int plb_conv_fwd_host(plb_context *ctx, const plb_conv_params *p, const plb_conv_options *opt,
                      const void *h_in, const void *h_weights, const float *h_bias, void *h_out) {
  if (int rc = plb_conv_fwd_host_async(ctx, p, opt, h_in, h_weights, h_bias, h_out)) return rc;
  return plb_synchronize(ctx);
}

int plb_conv_fwd_host_async(plb_context *ctx, const plb_conv_params *p,
                            const plb_conv_options *opt, const void *h_in, const void *h_weights,
                            const float *h_bias, void *h_out) {
  if (int rc = activate(ctx)) return rc;
  if (!p) return fail(PLB_ERR_INVALID_PARAMS, "null params");
  const std::string err = validate(*p);
  if (!err.empty()) return fail(PLB_ERR_INVALID_PARAMS, err);
  const size_t es = dtypeBytes(p->input_type), os = dtypeBytes(p->output_type);
  size_t in_px = 1, taps = 1, out_px = 1;
  for (unsigned d = 0; d != p->num_field_dims; ++d) {
    in_px *= p->field[d];
    taps *= p->kernel[d];
    out_px *= size_t(outputSize(*p, d));
  }
  const size_t in_bytes = size_t(p->batch) * in_px * p->groups * p->in_chans_per_group * es;
  const size_t w_bytes = size_t(p->groups) * taps * p->in_chans_per_group * p->out_chans_per_group * es;
  const size_t out_bytes = size_t(p->batch) * out_px * p->groups * p->out_chans_per_group * os;
  const size_t bias_bytes = size_t(p->groups) * p->out_chans_per_group * sizeof(float);
  void *di = nullptr, *dw = nullptr, *dout = nullptr, *dbias = nullptr;
  if (int rc = scratch(ctx, kSlotHostIn, in_bytes + 16, &di)) return rc;
  if (int rc = scratch(ctx, kSlotHostWeights, w_bytes + 16, &dw)) return rc;
  if (int rc = scratch(ctx, kSlotHostOut, out_bytes + 16, &dout)) return rc;
  if (h_bias) {
    if (int rc = scratch(ctx, kSlotHostBias, bias_bytes + 16, &dbias)) return rc;
    if (int rc = plb_memcpy_h2d(ctx, dbias, h_bias, bias_bytes)) return rc;
  }
  if (int rc = plb_memcpy_h2d(ctx, di, h_in, in_bytes)) return rc;
  if (int rc = plb_memcpy_h2d(ctx, dw, h_weights, w_bytes)) return rc;
  if (int rc = plb_conv_fwd(ctx, p, opt, di, dw, static_cast<const float *>(dbias), dout)) return rc;
  // enqueued only: the caller synchronises (plb_synchronize) before reading h_out
  if (out_bytes)
    PLB_CUDA(cudaMemcpyAsync(h_out, dout, out_bytes, cudaMemcpyDeviceToHost, ctx->stream));
  return PLB_OK;
}

}  // extern "C"
