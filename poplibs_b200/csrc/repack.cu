// Operands brought into a form the tensor maps can describe: rows whose pitch (or
// address) is not a multiple of 16 bytes are copied with the pitch rounded up and
// the gap zeroed; float operands are split into their bfloat16 pieces on the way.
//
//   float x = x_hi + x_lo + O(2^-17 |x|),  x_hi = bf16(x),  x_lo = bf16(x - x_hi)
//   x * w ~= x_hi*w_hi + x_lo*w_hi + x_hi*w_lo           (error O(2^-16 |x w|))
//
// (poplar::FLOAT inputs, which the reference accepts next to half and quarter,
// lib/poplin/ConvValidation.cpp:11-70.)  bfloat16 keeps float's exponent range, so
// no scaling is needed.  The three terms lie one after the other along the
// reduction dimension: x as (hi, lo, hi), w as (hi, hi, lo); what runs is the
// ordinary kernel on a reduction three times as long, fp32 accumulation as always.
#include <cuda_bf16.h>

#include <algorithm>

#include "runtime.h"
#include "sm100_prims.cuh"

namespace plb {

namespace {

struct RepackArgs {
  const uint8_t *src;
  uint8_t *dst;
  unsigned long long rows, src_pitch;  // src_pitch in bytes
  uint32_t cols;                       // elements of a row
  uint32_t vecs;                       // 16-byte vectors of a destination row
  uint32_t units;                      // steps per row: vecs, or groups of elements (kSplitCols)
  uint32_t group;                      // elements a thread splits at a time (kSplitCols), 8 or 2
  int aligned;                         // kSplitCols: pairs start at multiples of 8 bytes
  FastDiv fd_units;
  uint32_t elem_bytes;
  int mode;                            // RepackMode
  int weights;                         // pieces (hi, hi, lo) instead of (hi, lo, hi)
  unsigned long long mid;              // rows per plane (kSplitPlanes)
  uint32_t parts, sub_w, sub_h, full_w, full_h, step_w, step_h;  // Repack::lattice (sub_w 0: all rows)
};

constexpr int kRepackThreads = 256;
// Steps of a thread: one in operands that fill the device no more than twice, where the
// length of a block counts (160 x 1472 and 1472 x 1120 floats with the product 16.5 ->
// 15.9 us); else as many loads as help: four vectors of a copy (37845 rows of 396 halves
// with the product 26.8 -> 25.6 us), two steps of a split (four: 68.6 -> 70.4 us with
// the product at 4032 x 5312 floats), but twice as many pairs, which are short.
constexpr int kFewSteps = 1, kSplitSteps = 2, kCopySteps = 4;
__host__ __device__ constexpr int pairSteps(int steps) { return 2 * steps; }

// The first `valid` bytes from any address, zero beyond, out of the up to five aligned
// words that hold them.
__device__ __forceinline__ uint4 gatherBytes(const uint8_t *src, int valid) {
  const uint32_t off = uint32_t(reinterpret_cast<uintptr_t>(src)) & 3, bytes = uint32_t(min(valid, 16));
  const uint32_t *at = reinterpret_cast<const uint32_t *>(src - off);
  uint32_t w[5], o[4];
#pragma unroll
  for (int j = 0; j < 5; ++j) w[j] = 4 * j < off + bytes ? at[j] : 0u;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    o[j] = __funnelshift_r(w[j], w[j + 1], off * 8);
    const int n = int(bytes) - 4 * j;
    if (n < 4) o[j] = n <= 0 ? 0u : o[j] & ((1u << (8 * n)) - 1);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// Piece 0..2 of a float.  An infinity or NaN stays in the first piece alone: in
// the other two it would meet the zero low piece of the other operand and make a
// NaN of a product that is an infinity.
__device__ __forceinline__ uint16_t floatPiece(float x, int piece, int weights) {
  const __nv_bfloat16 hi = __float2bfloat16_rn(x);
  if (piece == 0) return __bfloat16_as_ushort(hi);
  if (!isfinite(x)) return 0;
  const bool low = weights ? piece == 2 : piece == 1;
  return __bfloat16_as_ushort(low ? __float2bfloat16_rn(x - __bfloat162float(hi)) : hi);
}

// The pieces of two floats, packed.
struct Pieces {
  uint32_t piece[3];
};
__device__ __forceinline__ Pieces splitPair(float x, float y, int weights) {
  const __nv_bfloat162 hi = __floats2bfloat162_rn(x, y);
  const float2 back = __bfloat1622float2(hi);
  const __nv_bfloat162 lo = __floats2bfloat162_rn(x - back.x, y - back.y);
  const uint32_t finite = (isfinite(x) ? 0xffffu : 0u) | (isfinite(y) ? 0xffff0000u : 0u);
  const uint32_t h = *reinterpret_cast<const uint32_t *>(&hi);
  const uint32_t h2 = h & finite, l = *reinterpret_cast<const uint32_t *>(&lo) & finite;
  return Pieces{{h, weights ? h2 : l, weights ? l : h2}};
}

// The source row of a destination row.
__device__ __forceinline__ unsigned long long sourceRow(const RepackArgs &a, unsigned long long row) {
  if (a.sub_w == 0) return row;
  // row = (image, h, w, part) of the sub-lattice
  const uint32_t per_w = uint32_t(row / a.parts), part = uint32_t(row - (unsigned long long)per_w * a.parts);
  const uint32_t rows = per_w / a.sub_w, w = per_w - rows * a.sub_w, n = rows / a.sub_h, h = rows - n * a.sub_h;
  return (((unsigned long long)n * a.full_h + h * a.step_h) * a.full_w + w * a.step_w) * a.parts + part;
}

// Both splits below: a thread loads neighbouring floats once and stores their three
// pieces; steps beyond the columns zero the row's padding, and all of a thread's steps
// load before any of them stores.  Destination vectors gathered one by one instead load
// and convert each float three times, with the lanes' loads 32 bytes apart.

// kSplitCols, eight floats at a time (16-byte aligned rows of a multiple of 8):
// 6689 rows of 1104 floats 27 -> 11 us.
template <int kPer>
__device__ __forceinline__ void splitEights(const RepackArgs &a, unsigned long long row0, uint32_t rest) {
  const uint32_t in_row = a.cols / 8;
  __align__(16) float f[kPer][8];
  uint4 *dst[kPer];
  bool pad[kPer];
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const uint32_t i = rest + uint32_t(u) * kRepackThreads + threadIdx.x;
    const uint32_t down = fast_div(i, a.fd_units);
    const uint32_t v = i - down * a.units;
    const unsigned long long row = row0 + down;
    dst[u] = nullptr;
    if (row >= a.rows) continue;
    pad[u] = v >= in_row;
    dst[u] = reinterpret_cast<uint4 *>(a.dst) + row * a.vecs + (pad[u] ? 2 * in_row : 0) + v;
    if (pad[u]) continue;
    const float4 *x = reinterpret_cast<const float4 *>(a.src + sourceRow(a, row) * a.src_pitch) + 2 * v;
    *reinterpret_cast<float4 *>(&f[u][0]) = x[0];
    *reinterpret_cast<float4 *>(&f[u][4]) = x[1];
  }
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    if (dst[u] == nullptr) continue;
    if (pad[u]) {
      *dst[u] = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    Pieces o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = splitPair(f[u][2 * j], f[u][2 * j + 1], a.weights);
#pragma unroll
    for (int k = 0; k < 3; ++k)
      dst[u][k * in_row] = make_uint4(o[0].piece[k], o[1].piece[k], o[2].piece[k], o[3].piece[k]);
  }
}

// kSplitCols, two floats at a time.  Every store is 4 bytes and aligned, which in a row
// of odd length the second pieces are one element earlier.  kAligned: rows of even length
// at multiples of 8 bytes.  6689 rows of 1102 and of 1103 floats 45 -> 17 and
// 21 us.
template <bool kAligned, int kPer>
__device__ __forceinline__ void splitPairs(const RepackArgs &a, unsigned long long row0, uint32_t rest) {
  const uint32_t odd = kAligned ? 0 : a.cols & 1, pitch = a.vecs * 8;
  float f[kPer][3];
  uint16_t *dst[kPer];
  uint32_t col[kPer];
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const uint32_t i = rest + uint32_t(u) * kRepackThreads + threadIdx.x;
    const uint32_t down = fast_div(i, a.fd_units);
    const uint32_t c = 2 * (i - down * a.units);
    const unsigned long long row = row0 + down;
    dst[u] = nullptr;
    if (row >= a.rows) continue;
    dst[u] = reinterpret_cast<uint16_t *>(a.dst) + row * pitch + c;
    col[u] = c;
    if (c >= a.cols) continue;
    const float *x = reinterpret_cast<const float *>(a.src + sourceRow(a, row) * a.src_pitch) + c;
    if constexpr (kAligned) {
      const float2 t = *reinterpret_cast<const float2 *>(x);
      f[u][0] = t.x;
      f[u][1] = t.y;
    } else {
      f[u][0] = x[0];
      f[u][1] = c + 1 < a.cols ? x[1] : 0.f;
      f[u][2] = odd && c ? x[-1] : 0.f;
    }
  }
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    if (dst[u] == nullptr) continue;
    const uint32_t c = col[u];
    uint32_t *const third = reinterpret_cast<uint32_t *>(dst[u] + 2 * a.cols);
    if (c >= a.cols) {  // the padding, from its first even element on
      *third = 0u;
      continue;
    }
    const Pieces o = splitPair(f[u][0], f[u][1], a.weights);
    *third = o.piece[2];  // (an odd row's last: its element and the first of the padding)
    if (!odd) {
      *reinterpret_cast<uint32_t *>(dst[u]) = o.piece[0];
      *reinterpret_cast<uint32_t *>(dst[u] + a.cols) = o.piece[1];
      continue;
    }
    const Pieces q = splitPair(f[u][2], f[u][0], a.weights);  // the pair one element earlier
    if (c + 1 < a.cols)
      *reinterpret_cast<uint32_t *>(dst[u]) = o.piece[0];
    else
      *dst[u] = uint16_t(o.piece[0]);
    if (c)
      *reinterpret_cast<uint32_t *>(dst[u] + a.cols - 1) = q.piece[1];
    else
      dst[u][a.cols] = uint16_t(o.piece[1]);
  }
}

// A step of kRepackCopy (one 16-byte destination vector) or kSplitPlanes (three).
// Rows start anywhere, so a vector is gathered from the aligned words that hold it;
// neighbouring threads read neighbouring bytes, and the overlap of their loads is
// caught by L1.  Bound by those loads: five words beat 8 halves or 16 bytes (quarter
// operands of 331 x 145 x 2588 8.5 -> 8.2 us with the product, half of 20000 x 33 x 40
// 9.7 -> 9.0); one 4-byte destination word per step, or two 16-byte loads shifted into
// place, were no faster.
__device__ __forceinline__ void vectorStep(const RepackArgs &a, unsigned long long row, uint32_t v) {
  const uint8_t *src = a.src + sourceRow(a, row) * a.src_pitch;
  if (a.mode == kRepackCopy) {
    const int valid = int(a.cols * a.elem_bytes) - int(v) * 16;
    uint4 o = make_uint4(0u, 0u, 0u, 0u);
    if (valid > 0) {
      src += size_t(v) * 16;
      const uintptr_t at = reinterpret_cast<uintptr_t>(src);
      if ((at & 15) == 0 && valid >= 16)
        o = *reinterpret_cast<const uint4 *>(src);
      else
        o = gatherBytes(src, valid);
    }
    *reinterpret_cast<uint4 *>(a.dst + (row * a.vecs + v) * 16) = o;
    return;
  }
  const float *x = reinterpret_cast<const float *>(src) + v * 8;
  __align__(16) uint16_t o[3][8];
  __align__(16) float f[8];
  if (v * 8 + 8 <= a.cols && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
    *reinterpret_cast<float4 *>(&f[0]) = *reinterpret_cast<const float4 *>(x);
    *reinterpret_cast<float4 *>(&f[4]) = *reinterpret_cast<const float4 *>(x + 4);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = v * 8 + j < a.cols ? x[j] : 0.f;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int k = 0; k < 3; ++k) o[k][j] = floatPiece(f[j], k, a.weights);
  const unsigned long long outer = a.mid < a.rows ? row / a.mid : 0, plane0 = outer * 2 * a.mid + row;
#pragma unroll
  for (int k = 0; k < 3; ++k)
    *reinterpret_cast<uint4 *>(a.dst + ((plane0 + k * a.mid) * a.vecs + v) * 16) =
        *reinterpret_cast<const uint4 *>(o[k]);
}

// Both operands of a call go in one launch.  kCols: one of them is kSplitCols (an
// instance of its own, since it takes more registers).
template <bool kCols, int kPer>
__global__ void __launch_bounds__(kRepackThreads)
repackKernel(const RepackArgs first, const RepackArgs second, unsigned first_blocks) {
  pdl_launch_dependents();
  pdl_wait();  // operands may come from the previous kernel in the stream
  const bool is_first = blockIdx.x < first_blocks;
  const RepackArgs &a = is_first ? first : second;
  const unsigned block = is_first ? blockIdx.x : blockIdx.x - first_blocks;
  const bool cols = kCols && a.mode == kRepackSplitCols;
  // the block's first step in 64 bits, the rest relative to its row in 32
  const uint32_t per_thread = cols && a.group < 8 ? pairSteps(kPer) : kPer;
  const unsigned long long base = (unsigned long long)block * (kRepackThreads * per_thread);
  const unsigned long long row0 = base / a.units;
  const uint32_t rest = uint32_t(base - row0 * a.units);
  if (cols) {
    if (a.group == 8)
      splitEights<kPer>(a, row0, rest);
    else if (a.aligned)
      splitPairs<true, pairSteps(kPer)>(a, row0, rest);
    else
      splitPairs<false, pairSteps(kPer)>(a, row0, rest);
    return;
  }
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const uint32_t i = rest + uint32_t(u) * kRepackThreads + threadIdx.x;
    const uint32_t down = fast_div(i, a.fd_units);
    const uint32_t v = i - down * a.units;
    const unsigned long long row = row0 + down;
    if (row >= a.rows) return;
    vectorStep(a, row, v);
  }
}

}  // namespace

size_t repackBytes(const Repack &r) {
  const size_t rows = r.mode == kRepackSplitPlanes ? 3 * size_t(r.rows) : size_t(r.rows);
  return rows * r.dst_pitch * (r.mode == kRepackCopy ? r.elem_bytes : 2);
}

int repack(plb_context *ctx, const Repack *jobs, int n) {
  RepackArgs args[2] = {};
  unsigned blocks[2] = {0, 0};
  int used = 0;
  uint64_t steps = 0;
  for (int i = 0; i < n; ++i) {
    const Repack &r = jobs[i];
    if (r.rows == 0 || r.cols == 0) continue;
    RepackArgs &a = args[used];
    a.src = static_cast<const uint8_t *>(r.src);
    a.dst = static_cast<uint8_t *>(r.dst);
    a.rows = r.rows;
    a.src_pitch = r.src_pitch * r.elem_bytes;
    a.cols = r.cols;
    a.vecs = uint32_t(size_t(r.dst_pitch) * (r.mode == kRepackCopy ? r.elem_bytes : 2) / 16);
    a.elem_bytes = r.elem_bytes;
    a.mode = r.mode;
    a.weights = r.weights ? 1 : 0;
    a.mid = r.mid ? r.mid : r.rows;
    a.units = a.vecs;
    if (r.mode == kRepackSplitCols) {
      const auto starts_at = [&](unsigned bytes) {
        return reinterpret_cast<uintptr_t>(r.src) % bytes == 0 && a.src_pitch % bytes == 0;
      };
      a.group = r.cols % 8 == 0 && starts_at(16) ? 8 : 2;
      a.aligned = r.cols % 2 == 0 && starts_at(8);
      a.units = (r.dst_pitch - 2 * r.cols) / a.group;  // columns and padding
    }
    a.fd_units = make_fastdiv(a.units);
    a.parts = r.lattice.parts;
    a.sub_w = r.lattice.sub_w;
    a.sub_h = r.lattice.sub_h;
    a.full_w = r.lattice.full_w;
    a.full_h = r.lattice.full_h;
    a.step_w = r.lattice.step_w;
    a.step_h = r.lattice.step_h;
    steps += r.rows * a.units;
    ++used;
  }
  if (used == 0) return PLB_OK;
  const bool cols = args[0].mode == kRepackSplitCols || (used > 1 && args[1].mode == kRepackSplitCols);
  const bool copy = args[0].mode == kRepackCopy;  // (the operands of a call have one type)
  const int per = steps <= uint64_t(2 * 2048) * uint64_t(ctx->sm_count) ? kFewSteps : copy ? kCopySteps : kSplitSteps;
  for (int i = 0; i < used; ++i) {
    const RepackArgs &a = args[i];
    const uint64_t block = kRepackThreads * (a.mode == kRepackSplitCols && a.group < 8 ? pairSteps(per) : per);
    const uint64_t b = (a.rows * a.units + block - 1) / block;
    if (b + blocks[0] > 0x7fffffffull || uint64_t(a.units) + block > 0x7fffffffull)
      return fail(PLB_ERR_UNSUPPORTED, "operand too large to be repacked");
    blocks[i] = unsigned(b);
  }
  auto kernel = per == kFewSteps     ? (cols ? repackKernel<true, kFewSteps> : repackKernel<false, kFewSteps>)
                : per == kSplitSteps ? (cols ? repackKernel<true, kSplitSteps> : repackKernel<false, kSplitSteps>)
                                     : repackKernel<false, kCopySteps>;
  return launchPdl(ctx, kernel, dim3(blocks[0] + blocks[1]), dim3(kRepackThreads), 0, args[0], args[1], blocks[0]);
}

}  // namespace plb
