// Forward convolution for layers whose input has too few channels for a TMA
// row (the ResNet stem: 3 channels, 7x7, stride 2).  NHWC pixels of 6 bytes
// cannot be addressed by TMA (16-byte granularity), and a 3-channel reduction
// would waste the tensor core's K dimension.  The layer is rewritten as an
// equivalent stride-1 convolution with the horizontal taps folded into K:
//
//  1. space-to-depth: stride s and the padding are absorbed into a rearranged
//     input X2[n][h2][w2][(ph, pw, c)] with C2 = s*s*Cp channels (Cp = channels
//     padded so that a pixel is a multiple of 16 bytes), zero where the
//     original is padding.  The s-strided KHxKW filter becomes a stride-1
//     K2h x K2w filter over X2 (K2 = ceil(K / s)).
//  2. the K2w horizontal taps of one output pixel are K2w consecutive pixels
//     of X2, i.e. one contiguous run of K2w*C2 elements (<= 64): the activation
//     tensor map describes overlapping windows (pixel stride C2 elements,
//     window 64 elements), so each K step is one ordinary 128-byte row per
//     output pixel and the implicit-GEMM kernel runs unchanged with K2h taps.
//
// This is the role the reference gives to its expandDims / outChanFlattenDims
// input transforms for small channel counts (lib/poplin/ConvPlan.cpp:1100-1224,
// lib/poplin/Convolution.cpp:665-978).
#include <cuda_fp16.h>

#include <algorithm>

#include "conv_geometry.h"
#include "runtime.h"
#include "small_channel.h"
#include "sm100_prims.cuh"
#include "stem.h"

namespace plb {

// W2[a][co][(b*s*s + ph*s + pw)*Cp + c] = W[a*s + ph][b*s + pw][co][c], rows padded to 64:
// element i of the folded weights.
__device__ __forceinline__ __half foldedWeight(const __half *__restrict__ w, const S2dShape &g,
                                               unsigned co_total, unsigned i) {
  const unsigned k = i & 63u;
  const unsigned r = i >> 6;
  const unsigned a = r / co_total, co = r - a * co_total;
  const unsigned b = k / unsigned(g.C2);
  if (b >= unsigned(g.K2w)) return __float2half(0.f);
  const unsigned c2 = k - b * g.C2;
  const unsigned sub = c2 / unsigned(g.Cp), c = c2 - sub * g.Cp;
  const unsigned ph = sub / unsigned(g.s), pw = sub - ph * g.s;
  const unsigned kh = a * g.s + ph, kw = b * g.s + pw;
  if (c < unsigned(g.C) && kh < unsigned(g.KH) && kw < unsigned(g.KW))
    return w[((size_t(kh) * g.KW + kw) * co_total + co) * g.C + c];
  return __float2half(0.f);
}

// Block `block` (128 threads) of the blocks that fold the weights; the first of them
// clears the 128 bytes after X2, which only ever meet zero weights but must be finite.
__device__ __forceinline__ void foldWeightsAndTail(const S2dShape &g, unsigned block, __half *x2,
                                                   const __half *__restrict__ w, __half *__restrict__ w2, int co_total) {
  const unsigned total = unsigned(g.K2h) * unsigned(co_total) * 64u, i = block * 128u + threadIdx.x;
  if (i < total) w2[i] = foldedWeight(w, g, unsigned(co_total), i);
  if (block == 0 && threadIdx.x < 8)
    reinterpret_cast<uint4 *>(x2 + size_t(g.N) * g.H2 * g.W2 * g.C2)[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
}

// X2[n][h2][w2][(ph*s + pw)*Cp + c] = X[n][h2*s + ph - padH][w2*s + pw - padW][c],
// zero outside the input and for channels C..Cp-1.  One thread per 16-byte vector of
// X2, its up to eight elements loaded independently of one another: they are
// neighbours of what the neighbouring threads load, so L1 serves most of them, and
// with nothing staged or shared between threads every block has all its loads in
// flight at once (staging rows in shared memory behind two barriers took 9.4 us for
// 98 images of 60x161x1, now 3.0).  Blocks past the first `row_blocks` fold the
// weights and clear the tail of X2.
// kCp: Cp where it is one of the usual ones (divisions by constants), else 0.
template <int kS, int kCp>
__global__ void __launch_bounds__(128)
s2dInputKernel(const __half *__restrict__ x, __half *__restrict__ x2, S2dShape g, FastDiv fd_row, FastDiv fd_h2,
               unsigned row_blocks, const __half *__restrict__ w, __half *__restrict__ w2, int co_total) {
  const unsigned vecs = kCp ? unsigned(kS * kS * kCp / 8) : unsigned(g.C2) / 8;  // per pixel of X2
  pdl_launch_dependents();
  pdl_wait();
  if (blockIdx.x >= row_blocks) {
    foldWeightsAndTail(g, blockIdx.x - row_blocks, x2, w, w2, co_total);
    return;
  }
  // the block's first vector in 64 bits, the rest relative to its row in 32
  const unsigned per_row = unsigned(g.W2) * vecs;
  const unsigned long long base = blockIdx.x * 128ull, row0 = base / per_row;
  const unsigned rel = unsigned(base - row0 * per_row) + threadIdx.x, down = fast_div(rel, fd_row);
  const unsigned row = unsigned(row0) + down;
  if (row >= unsigned(g.N) * unsigned(g.H2)) return;
  const unsigned at = rel - down * per_row, pix = at / vecs, v = at - pix * vecs;
  const unsigned n = fast_div(row, fd_h2);
  const int h0 = int(row - n * unsigned(g.H2)) * kS - g.padH, w0 = int(pix) * kS - g.padW;
  __align__(16) uint16_t vals[8];
  const uint16_t *img = reinterpret_cast<const uint16_t *>(x) + size_t(n) * g.H * g.W * g.C;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int cp = kCp ? kCp : g.Cp;
    const int c2 = int(v) * 8 + j, sub = kS == 1 ? 0 : c2 / cp, c = c2 - sub * cp;
    const int ih = h0 + sub / kS, iw = w0 + sub % kS;
    const bool in = c < g.C && unsigned(ih) < unsigned(g.H) && unsigned(iw) < unsigned(g.W);
    vals[j] = in ? img[((long long)ih * g.W + iw) * g.C + c] : uint16_t(0);
  }
  *reinterpret_cast<uint4 *>(x2 + (base + threadIdx.x) * 8) = *reinterpret_cast<const uint4 *>(vals);
}

// The same rearrangement for the common stem shape (3 channels, stride 2, so
// Cp = 4 and one X2 pixel is two 16-byte vectors, one per vertical phase):
// a vector is [X(ih, iw) c0..2, 0, X(ih, iw+1) c0..2, 0], i.e. six consecutive
// halves of one input row.  One block per (n, h2) row of X2, one thread per
// pixel of it (both vectors), so a warp reads one contiguous span of each of
// the two input rows (four aligned 32-bit loads per thread and row,
// overlapping its neighbours' in L1) and writes 1024 contiguous bytes.  No
// shared memory; the only division is one 32-bit one per thread.  The blocks
// past the last row fold the weights and clear the 128 bytes after X2 (they
// only ever meet zero weights, but must be finite), so the layer's
// preparation is one launch.
__global__ void __launch_bounds__(128)
s2dStem3Kernel(const uint32_t *__restrict__ x32, uint4 *__restrict__ x2, S2dShape g,
               const __half *__restrict__ w, __half *__restrict__ w2, int co_total) {
  // the convolution that follows may set itself up meanwhile; it waits for this
  // grid to finish before it reads
  pdl_launch_dependents();
  pdl_wait();  // (the input, or X2 of an earlier call, may belong to the previous kernel)
  const unsigned rows = unsigned(g.N) * unsigned(g.H2);
  if (blockIdx.x >= rows) {
    foldWeightsAndTail(g, blockIdx.x - rows, reinterpret_cast<__half *>(x2), w, w2, co_total);
    return;
  }
  const int row_words = g.W * 3 / 2;  // W * 3 is even: rows start on a 32-bit word
  // last rows first: the convolution starts with the first images, which are
  // then the ones most recently written and still in L2
  const unsigned row = rows - 1 - blockIdx.x;
  const unsigned n = row / unsigned(g.H2);
  const int h2 = int(row - n * unsigned(g.H2));
  uint4 *dst = x2 + (size_t(row) * g.W2 << 1);
  for (int w2 = threadIdx.x; w2 < g.W2; w2 += blockDim.x) {
    const int iw = 2 * w2 - g.padW;
    const bool cols = iw + 1 >= 0 && iw < g.W;
    const int h0 = iw * 3;               // first half wanted, relative to the row (may be negative)
    const int odd = h0 & 1;
    const int w0 = (h0 - odd) >> 1;      // first 32-bit word (exact; arithmetic shift)
    const bool left = iw >= 0, right = iw + 1 < g.W;
    uint4 out[2];
#pragma unroll
    for (int ph = 0; ph < 2; ++ph) {
      const int ih = 2 * h2 + ph - g.padH;
      out[ph] = make_uint4(0u, 0u, 0u, 0u);
      if (cols && ih >= 0 && ih < g.H) {
        const uint32_t *row = x32 + (size_t(n) * g.H + ih) * row_words;
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) w[k] = (w0 + k >= 0 && w0 + k < row_words) ? row[w0 + k] : 0u;
        // halves h0 .. h0 + 5 of the 8 loaded
        uint32_t a, b, c;  // (h0,h1) (h2,h3) (h4,h5)
        if (odd) {
          a = __funnelshift_r(w[0], w[1], 16);
          b = __funnelshift_r(w[1], w[2], 16);
          c = __funnelshift_r(w[2], w[3], 16);
        } else {
          a = w[0];
          b = w[1];
          c = w[2];
        }
        // pixel iw: h0 h1 h2; pixel iw + 1: h3 h4 h5
        out[ph].x = left ? a : 0u;
        out[ph].y = left ? (b & 0xffffu) : 0u;
        out[ph].z = right ? ((b >> 16) | (c << 16)) : 0u;
        out[ph].w = right ? (c >> 16) : 0u;
      }
    }
    dst[size_t(w2) << 1] = out[0];
    dst[(size_t(w2) << 1) + 1] = out[1];
  }
}


// The shape of the rearranged layer; PLB_ERR_UNSUPPORTED (with a message) when it
// does not fit this path.
int smallChannelShape(const plb_conv_params &p, S2dShape *out) {
  if (p.num_field_dims != 2 || p.groups != 1 || !is16BitFloat(p.input_type))
    return fail(PLB_ERR_UNSUPPORTED,
                "input channel count must be a multiple of 8 (half) / 16 (quarter) unless the "
                "layer is a 2-D, ungrouped half convolution");
  for (unsigned d = 0; d != 2; ++d)
    if (p.in_trunc_lo[d] || p.in_trunc_hi[d] || p.in_dilation[d] != 1 || p.in_flip[d] ||
        p.k_trunc_lo[d] || p.k_trunc_hi[d] || p.k_pad_lo[d] || p.k_pad_hi[d] || p.k_flip[d] ||
        p.k_dilation[d] != 1 || p.out_trunc_lo[d] || p.out_trunc_hi[d] || p.out_pad_lo[d] ||
        p.out_pad_hi[d])
      return fail(PLB_ERR_UNSUPPORTED,
                  "small-channel convolutions support padding and stride only");
  if (p.stride[0] != p.stride[1] || p.stride[0] > 2)
    return fail(PLB_ERR_UNSUPPORTED, "small-channel convolutions need equal strides of 1 or 2");
  S2dShape g{};
  g.N = int(p.batch);
  g.H = int(p.field[0]);
  g.W = int(p.field[1]);
  g.C = int(p.in_chans_per_group);
  g.s = int(p.stride[0]);
  g.padH = int(p.in_pad_lo[0]);
  g.padW = int(p.in_pad_lo[1]);
  g.KH = int(p.kernel[0]);
  g.KW = int(p.kernel[1]);
  g.OH = int(outputSize(p, 0));
  g.OW = int(outputSize(p, 1));
  // pixel of X2 must be a multiple of 16 bytes = 8 halves
  g.Cp = g.C;
  while ((g.s * g.s * g.Cp) % 8 != 0) ++g.Cp;
  g.C2 = g.s * g.s * g.Cp;
  g.K2h = (g.KH + g.s - 1) / g.s;
  g.K2w = (g.KW + g.s - 1) / g.s;
  if (g.K2w * g.C2 > 64)
    return fail(PLB_ERR_UNSUPPORTED,
                "small-channel convolution: folded filter row of " +
                    std::to_string(g.K2w * g.C2) + " elements exceeds one 128-byte K step");
  g.H2 = g.OH + g.K2h - 1;
  g.W2 = g.OW + g.K2w - 1;
  if (uint64_t(g.N) * g.H2 >= uint64_t(1) << 31 || uint64_t(g.N) * g.H2 * g.W2 * (g.C2 / 8) >= uint64_t(1) << 37)
    return fail(PLB_ERR_UNSUPPORTED, "small-channel convolution: too many rows");
  *out = g;
  return PLB_OK;
}

// Elements of X2, the window of the last pixel included: it may run past the
// K2w*C2 elements that carry weights (64 elements, cleared).
size_t smallChannelElems(const S2dShape &g) { return size_t(g.N) * g.H2 * g.W2 * g.C2 + 64; }

// Writes X2, and with `w2` the folded weights ([K2h][co][64]).
int smallChannelPrepare(plb_context *ctx, const S2dShape &g, const void *d_in, __half *x2, const void *d_weights,
                        __half *w2, int co) {
  const size_t w2_elems = w2 ? size_t(g.K2h) * co * 64 : 0;
  // (at least one block past the rows: it clears the tail of X2)
  const unsigned wblocks = unsigned(std::max<size_t>(1, (w2_elems + 127) / 128));
  const __half *w = static_cast<const __half *>(d_weights);
  const int w_co = w2 ? co : 0;
  if (g.C == 3 && g.s == 2 && g.Cp == 4 && (g.W * g.C) % 2 == 0 && (reinterpret_cast<uintptr_t>(d_in) & 3) == 0)
    return launchPdl(ctx, s2dStem3Kernel, dim3(unsigned(g.N) * unsigned(g.H2) + wblocks), dim3(128), 0,
                     static_cast<const uint32_t *>(d_in), reinterpret_cast<uint4 *>(x2), g, w, w2, w_co);
  const size_t vecs = size_t(g.N) * g.H2 * g.W2 * (g.C2 / 8);
  const unsigned blocks = unsigned((vecs + 127) / 128);
  auto launch = [&](auto kernel) {
    return launchPdl(ctx, kernel, dim3(blocks + wblocks), dim3(128), 0, static_cast<const __half *>(d_in), x2, g,
                     make_fastdiv(unsigned(g.W2) * unsigned(g.C2 / 8)), make_fastdiv(unsigned(g.H2)), blocks, w, w2, w_co);
  };
  if (g.s == 1) return g.Cp == 8 ? launch(s2dInputKernel<1, 8>) : launch(s2dInputKernel<1, 0>);
  switch (g.Cp) {
    case 2: return launch(s2dInputKernel<2, 2>);
    case 4: return launch(s2dInputKernel<2, 4>);
    default: return launch(s2dInputKernel<2, 0>);
  }
}

// Whether the stem kernel runs the forward pass.
bool stemLayer(int sm_count, int plan_flags, const plb_conv_params &p, const plb_conv_options *opt, const void *d_out, bool slower_too, S2dShape *g) {
  return smallChannelShape(p, g) == PLB_OK && plan_flags == 0 && (!opt || (opt->plan_flags == 0 && opt->tile_n == 0)) &&
         stemSuits(sm_count, *g, int(p.out_chans_per_group), p.output_type == PLB_FLOAT, d_out, slower_too);
}

int convFwdSmallChannels(plb_context *ctx, const plb_conv_params &p, const plb_conv_options *opt,
                         const void *d_in, const void *d_weights, const float *d_bias,
                         void *d_out, plb_plan *plan_only) {
  S2dShape g{};
  if (int rc = smallChannelShape(p, &g)) return rc;
  const int co = int(p.out_chans_per_group);
  const size_t x2_elems = smallChannelElems(g);
  const size_t w2_elems = size_t(g.K2h) * co * 64;

  IgemmProblem q;
  q.bf16 = p.input_type == PLB_BFLOAT16;
  q.act_dims[0] = 64;
  q.act_dims[1] = uint64_t(g.OW);
  q.act_dims[2] = uint64_t(g.H2);
  q.act_dims[3] = uint64_t(g.N);
  q.act_strides[0] = uint64_t(g.C2) * 2;
  q.act_strides[1] = uint64_t(g.W2) * g.C2 * 2;
  q.act_strides[2] = uint64_t(g.H2) * g.W2 * g.C2 * 2;
  q.wgt_dims[0] = 64;
  q.wgt_dims[1] = uint64_t(co);
  q.wgt_dims[2] = uint64_t(g.K2h);
  q.wgt_strides[0] = 128;
  q.wgt_strides[1] = uint64_t(co) * 128;
  q.out_w = g.OW;
  q.out_h = g.OH;
  q.out_n = g.N;
  q.n_total = co;
  q.k_per_tap = g.K2w * g.C2;  // (the rest of a window meets zero weights)
  q.taps_h = g.K2h;
  q.taps_w = 1;
  q.ldc = co;
  q.bias = d_bias;
  q.out_f32 = p.output_type == PLB_FLOAT;
  q.force_tile_n = opt ? opt->tile_n : 0;
  q.plan_flags = opt ? opt->plan_flags : 0;
  // The K loop here is short (K2h steps), below the planner's general threshold
  // for CTA pairs, but with 64 output channels the instruction is bound by its
  // activation operand, which a pair splits between two SMs: measured 197 ->
  // 191 us on the 7x7 stride-2 stem of 256 images.  Taken when there are many tiles.
  const int sms = ctx ? ctx->sm_count : 148;
  if ((q.plan_flags & PLB_PLAN_NO_CTA_PAIR) == 0 &&
      uint64_t(g.OW) * g.OH * g.N >= uint64_t(128) * 8 * sms)
    q.plan_flags |= PLB_PLAN_FORCE_CTA_PAIR;
  plb_plan plan{};
  if (int rc = planIgemm(q, sms, &plan)) return rc;
  plan.kernel = 2;
  plan.workspace_bytes = (x2_elems + w2_elems) * 2;
  if (plan_only) {
    *plan_only = plan;
    return PLB_OK;
  }
  void *ws = nullptr;
  if (int rc = scratch(ctx, kSlotOperands, plan.workspace_bytes + 256, &ws)) return rc;
  __half *x2 = static_cast<__half *>(ws);
  __half *w2 = x2 + ((x2_elems + 127) & ~size_t(127));
  if (int rc = smallChannelPrepare(ctx, g, d_in, x2, d_weights, w2, co)) return rc;
  q.act = x2;
  q.wgt = w2;
  q.out = d_out;
  return launchIgemm(ctx, q, plan);
}

}  // namespace plb
