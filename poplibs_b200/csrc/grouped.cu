// Convolutions with many narrow channel groups.
//
// A group of 8 channels fills an eighth of a 128-byte operand row, and the copy
// engine takes a row at a time (measured: 4 clocks and more per 16-byte row, which
// made a 3x3 layer of 32 groups of 8 channels spend 115 us on 26 MB).  So
// neighbouring groups are contracted together as one dense block: their channels
// lie side by side in memory already, and the weights become a block-diagonal
// filter in scratch.  The tensor core multiplies the zeros off the diagonal, work
// that is free where the copies are the bound.
//
// Zero times an infinity or a NaN is a NaN, though, and in a dense block it would
// reach the other groups' outputs, which do not depend on that element.  The
// implicit-GEMM kernel therefore notes whether any of its sums is not finite, and
// a second kernel, which otherwise leaves at once, computes every output that is
// not finite again from its own group alone.  With finite sums the result is the
// separate groups': adding products that are zero changes no sum.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <algorithm>

#include "grouped.h"
#include "sm100_prims.cuh"

namespace plb {

namespace {

// [G][taps][rows][cols] -> [G/S][taps][S*rows][S*cols], zero off the diagonal.
template <typename T>
__global__ void __launch_bounds__(256)
blockDiagonalKernel(const T *__restrict__ src, T *__restrict__ dst, uint32_t S, uint32_t taps, uint32_t rows,
                    uint32_t cols, size_t total, int *nonfinite) {
  pdl_launch_dependents();
  pdl_wait();  // the weights may come from the previous kernel in the stream
  if (blockIdx.x == 0 && threadIdx.x == 0) *nonfinite = 0;
  const uint32_t width = S * cols, height = S * rows;
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x) {
    const size_t row = i / width;
    const uint32_t col = uint32_t(i - row * width);
    const size_t tile = row / height;
    const uint32_t r = uint32_t(row - tile * height), gr = r / rows, gc = col / cols;
    const size_t sg = tile / taps;
    const uint32_t tap = uint32_t(tile - sg * taps);
    dst[i] = gr == gc ? src[(((sg * S + gr) * taps + tap) * rows + (r - gr * rows)) * cols + (col - gc * cols)] : T(0);
  }
}

struct RepairArgs {
  const uint8_t *act, *wgt;
  uint64_t act_dims[4], act_strides[3], act_group_stride, wgt_strides[2];
  int b_mn, k, taps_h, taps_w, pad_h, pad_w, dil_h, dil_w, stride_h, stride_w, flip_h, flip_w, in_dil_h, in_dil_w;
  int tap_first_h, tap_step_h, tap_pitch_h, tap_first_w, tap_step_w, taps_stored;
  int groups, n_total, out_w, out_h, out_n;
  void *out;
  long long ldc, out_stride_h, out_stride_n, out_group_stride;
  const float *bias;
  float alpha;
  int out_is_f32, type, fmt_a, fmt_b;
};

__device__ float operandValue(const uint8_t *p, int type, int fmt) {
  switch (type) {
    case PLB_FLOAT: return *reinterpret_cast<const float *>(p);
    case PLB_BFLOAT16: return __bfloat162float(*reinterpret_cast<const __nv_bfloat16 *>(p));
    case PLB_HALF: return __half2float(*reinterpret_cast<const __half *>(p));
    default: return __half2float(__half(__nv_cvt_fp8_to_halfraw(*p, fmt == PLB_F152 ? __NV_E5M2 : __NV_E4M3)));
  }
}

// Every output that is not finite, from its own group's operands.
__global__ void __launch_bounds__(128) repairKernel(const RepairArgs a, const int *__restrict__ nonfinite) {
  pdl_launch_dependents();
  pdl_wait();
  if (*nonfinite == 0) return;
  const size_t es = a.type == PLB_FLOAT ? 4 : a.type == PLB_QUARTER ? 1 : 2;
  const size_t total = size_t(a.groups) * a.n_total * a.out_w * a.out_h * a.out_n;
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x) {
    size_t r = i;
    const int c = int(r % a.n_total);
    r /= a.n_total;
    const int g = int(r % a.groups);
    r /= a.groups;
    const int ow = int(r % a.out_w);
    r /= a.out_w;
    const int oh = int(r % a.out_h), on = int(r / a.out_h);
    const long long off = on * a.out_stride_n + oh * a.out_stride_h + ow * a.ldc + g * a.out_group_stride + c;
    const float old = a.out_is_f32 ? static_cast<const float *>(a.out)[off]
                                   : __half2float(static_cast<const __half *>(a.out)[off]);
    if (isfinite(old)) continue;
    float sum = 0.f;
    for (int t = 0; t < a.taps_h * a.taps_w; ++t) {
      const int th = t / a.taps_w, tw = t - th * a.taps_w;
      const long long ih = (long long)oh * a.stride_h + th * a.dil_h - a.pad_h;
      const long long iw = (long long)ow * a.stride_w + tw * a.dil_w - a.pad_w;
      if (ih < 0 || iw < 0 || ih % a.in_dil_h != 0 || iw % a.in_dil_w != 0) continue;
      const long long xh = ih / a.in_dil_h, xw = iw / a.in_dil_w;
      if (xh >= (long long)a.act_dims[2] || xw >= (long long)a.act_dims[1]) continue;
      const uint8_t *x = a.act + on * a.act_strides[2] + xh * a.act_strides[1] + xw * a.act_strides[0] +
                         g * a.act_group_stride;
      const int tile = ((a.flip_h ? a.taps_h - 1 - th : th) * a.tap_step_h + a.tap_first_h) * a.tap_pitch_h +
                       (a.flip_w ? a.taps_w - 1 - tw : tw) * a.tap_step_w + a.tap_first_w + g * a.taps_stored;
      const uint8_t *w = a.wgt + tile * a.wgt_strides[1];
      for (int k = 0; k < a.k; ++k) {
        const uint8_t *wk = a.b_mn ? w + k * a.wgt_strides[0] + c * es : w + c * a.wgt_strides[0] + k * es;
        sum += operandValue(x + k * es, a.type, a.fmt_a) * operandValue(wk, a.type, a.fmt_b);
      }
    }
    sum *= a.alpha;
    if (a.bias) sum += a.bias[g * a.n_total + c];
    if (a.out_is_f32)
      static_cast<float *>(a.out)[off] = sum;
    else
      static_cast<__half *>(a.out)[off] = __float2half_rn(sum);
  }
}

}  // namespace

// Chosen by operand rows: `bytes` per channel as they reach the tensor core, the
// cost the 128-byte operand rows loaded per pixel, times the 64-column output
// blocks where a block exceeds one.  Only divisors of the group count: a block that
// ran past a pixel's last group would read the next pixel's channels.
uint32_t groupsTogether(uint32_t groups, uint32_t ci, uint32_t co, int type) {
  const uint32_t bytes = type == PLB_FLOAT ? 6 : uint32_t(dtypeBytes(type));
  uint32_t best = 1;
  double best_cost = 0;
  for (uint32_t s = 1; s <= groups; ++s) {
    if (s > 1 && (uint64_t(s) * ci * bytes > 384 || uint64_t(s) * co > 128)) break;
    if (groups % s != 0) continue;
    const bool repacked = type != PLB_FLOAT && (uint64_t(s) * ci * bytes) % 16 != 0;
    const double cost = double(groups / s) * double((uint64_t(s) * ci * bytes + 127) / 128) *
                        std::max(1.0, double(s) * co / 64.0) * (repacked ? 1.5 : 1.0);
    if (s == 1 || cost < best_cost) {
      best = s;
      best_cost = cost;
    }
  }
  return best;
}

int *nonfiniteFlag(plb_context *ctx) { return reinterpret_cast<int *>(ctx->d_ticket) + 16; }

int blockDiagonalWeights(plb_context *ctx, int type, const void *src, uint32_t groups, uint32_t S, uint32_t taps,
                         uint32_t rows, uint32_t cols, const void **out) {
  const size_t es = dtypeBytes(type), total = size_t(groups) * taps * rows * cols * S;
  void *ws = nullptr;
  if (int rc = scratch(ctx, kSlotBlockDiagonal, total * es + 256, &ws)) return rc;
  *out = ws;
  const dim3 grid(unsigned(std::max<size_t>(1, std::min<size_t>((total + 255) / 256, size_t(ctx->sm_count) * 8))));
  auto launch = [&](auto t) {
    using T = decltype(t);
    return launchPdl(ctx, blockDiagonalKernel<T>, grid, dim3(256), 0, static_cast<const T *>(src), static_cast<T *>(ws),
                     S, taps, rows, cols, total, nonfiniteFlag(ctx));
  };
  return es == 1 ? launch(uint8_t()) : es == 2 ? launch(uint16_t()) : launch(uint32_t());
}

int repairNonFinite(plb_context *ctx, const IgemmProblem &p, int type, int in_dil_h, int in_dil_w) {
  RepairArgs a{};
  a.act = static_cast<const uint8_t *>(p.act);
  a.wgt = static_cast<const uint8_t *>(p.wgt);
  std::copy(p.act_dims, p.act_dims + 4, a.act_dims);
  std::copy(p.act_strides, p.act_strides + 3, a.act_strides);
  std::copy(p.wgt_strides, p.wgt_strides + 2, a.wgt_strides);
  a.act_group_stride = p.act_group_stride;
  a.b_mn = p.b_mn;
  a.k = p.k_per_tap;
  a.taps_h = p.taps_h;
  a.taps_w = p.taps_w;
  a.pad_h = p.pad_h;
  a.pad_w = p.pad_w;
  a.dil_h = p.dil_h;
  a.dil_w = p.dil_w;
  a.stride_h = p.stride_h;
  a.stride_w = p.stride_w;
  a.flip_h = p.flip_h;
  a.flip_w = p.flip_w;
  a.in_dil_h = in_dil_h;
  a.in_dil_w = in_dil_w;
  a.tap_first_h = p.tap_first_h;
  a.tap_step_h = p.tap_step_h;
  a.tap_pitch_h = p.tap_pitch_h ? p.tap_pitch_h : p.taps_w;
  a.tap_first_w = p.tap_first_w;
  a.tap_step_w = p.tap_step_w;
  a.taps_stored = p.taps_stored ? p.taps_stored : p.taps_h * p.taps_w;
  a.groups = p.groups;
  a.n_total = p.n_total;
  a.out_w = p.out_w;
  a.out_h = p.out_h;
  a.out_n = p.out_n;
  a.out = p.out;
  a.ldc = p.ldc;
  a.out_stride_h = p.out_stride_h;
  a.out_stride_n = p.out_stride_n;
  a.out_group_stride = p.out_group_stride;
  a.bias = p.bias;
  a.alpha = p.alpha;
  a.out_is_f32 = p.out_f32 ? 1 : 0;
  a.type = type;
  a.fmt_a = p.fmt_a;
  a.fmt_b = p.fmt_b;
  // Shared memory that is not used: its blocks start early and wait, and next to the contraction's CTAs, whose
  // registers leave room for one of them, and many to an SM they keep the next contraction's out
  // (1x1, 16 groups of 4 -> 32, 53 images of 7 x 9 8.4 us without, 7.5 with; 322 passes of layers of narrow groups
  // 0.985 of their time in all, 0.995 with 12 KB, 0.987 with 48).
  constexpr size_t kApart = 24 * 1024;
  return launchPdl(ctx, repairKernel, dim3(unsigned(ctx->sm_count)), dim3(128), kApart, a, (const int *)nonfiniteFlag(ctx));
}

}  // namespace plb
