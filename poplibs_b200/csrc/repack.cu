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
  FastDiv fd_vecs;
  uint32_t elem_bytes;
  int mode;                            // RepackMode
  int weights;                         // pieces (hi, hi, lo) instead of (hi, lo, hi)
  unsigned long long mid;              // rows per plane (kSplitPlanes)
  uint32_t parts, sub_w, sub_h, full_w, full_h, step_w, step_h;  // Repack::lattice (sub_w 0: all rows)
};

constexpr int kRepackThreads = 256;
constexpr int kRepackPerThread = 2;

// `bytes` (a multiple of G) bytes from an address aligned to G, zero beyond `valid`
template <typename G>
__device__ __forceinline__ uint4 gatherBytes(const uint8_t *src, int valid) {
  constexpr int n = 16 / int(sizeof(G));
  __align__(16) G g[n];
#pragma unroll
  for (int j = 0; j < n; ++j) g[j] = int(j * sizeof(G)) < valid ? reinterpret_cast<const G *>(src)[j] : G(0);
  return *reinterpret_cast<const uint4 *>(g);
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

// One 16-byte destination vector per step (three in kSplitPlanes).  Rows start
// anywhere, so a vector is gathered with the widest loads its source address
// allows; neighbouring threads read neighbouring bytes, and the overlap of their
// narrow loads is caught by L1.  Bound by those loads (4.5 TB/s at 2 bytes per
// lane), which beats what a byte per thread with two divisions reached 10 to 20
// times over.  Both operands of a call go in one launch.
__global__ void __launch_bounds__(kRepackThreads)
repackKernel(const RepackArgs first, const RepackArgs second, unsigned first_blocks) {
  pdl_launch_dependents();
  pdl_wait();  // operands may come from the previous kernel in the stream
  const bool is_first = blockIdx.x < first_blocks;
  const RepackArgs &a = is_first ? first : second;
  const unsigned block = is_first ? blockIdx.x : blockIdx.x - first_blocks;
  // the block's first vector in 64 bits, the rest relative to its row in 32
  const unsigned long long base = (unsigned long long)block * (kRepackThreads * kRepackPerThread);
  const unsigned long long row0 = base / a.vecs;
  const uint32_t rest = uint32_t(base - row0 * a.vecs);
#pragma unroll
  for (int u = 0; u < kRepackPerThread; ++u) {
    const uint32_t i = rest + uint32_t(u) * kRepackThreads + threadIdx.x;
    const uint32_t down = fast_div(i, a.fd_vecs);
    const uint32_t v = i - down * a.vecs;
    const unsigned long long row = row0 + down;
    if (row >= a.rows) return;
    unsigned long long src_row = row;
    if (a.sub_w != 0) {
      // row = (image, h, w, part) of the sub-lattice
      const uint32_t per_w = uint32_t(row / a.parts), part = uint32_t(row - (unsigned long long)per_w * a.parts);
      const uint32_t rows = per_w / a.sub_w, w = per_w - rows * a.sub_w, n = rows / a.sub_h, h = rows - n * a.sub_h;
      src_row = (((unsigned long long)n * a.full_h + h * a.step_h) * a.full_w + w * a.step_w) * a.parts + part;
    }
    const uint8_t *src = a.src + src_row * a.src_pitch;
    if (a.mode == kRepackCopy) {
      const int valid = int(a.cols * a.elem_bytes) - int(v) * 16;
      uint4 o = make_uint4(0u, 0u, 0u, 0u);
      if (valid > 0) {
        src += size_t(v) * 16;
        const uintptr_t at = reinterpret_cast<uintptr_t>(src);
        if ((at & 15) == 0 && valid >= 16)
          o = *reinterpret_cast<const uint4 *>(src);
        else if ((at & 3) == 0 && (valid & 3) == 0)
          o = gatherBytes<uint32_t>(src, valid);
        else if ((at & 1) == 0 && (valid & 1) == 0)
          o = gatherBytes<uint16_t>(src, valid);
        else
          o = gatherBytes<uint8_t>(src, valid);
      }
      *reinterpret_cast<uint4 *>(a.dst + (row * a.vecs + v) * 16) = o;
      continue;
    }
    const float *x = reinterpret_cast<const float *>(src);
    __align__(16) uint16_t o[3][8];
    if (a.mode == kRepackSplitCols && a.cols % 8 == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
      // the eight elements are neighbours and of one piece (or beyond the last)
      const uint32_t piece = v * 8 / a.cols, col = v * 8 - piece * a.cols;
      const float4 f0 = *reinterpret_cast<const float4 *>(x + col), f1 = *reinterpret_cast<const float4 *>(x + col + 4);
      const float f[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) o[0][j] = piece < 3 ? floatPiece(f[j], int(piece), a.weights) : uint16_t(0);
      *reinterpret_cast<uint4 *>(a.dst + (row * a.vecs + v) * 16) = *reinterpret_cast<const uint4 *>(o[0]);
    } else if (a.mode == kRepackSplitCols) {
      // (piece, column) of the eight elements
      uint32_t piece = v * 8 / a.cols, col = v * 8 - piece * a.cols;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        o[0][j] = piece < 3 ? floatPiece(x[col], int(piece), a.weights) : uint16_t(0);
        if (++col == a.cols) {
          col = 0;
          ++piece;
        }
      }
      *reinterpret_cast<uint4 *>(a.dst + (row * a.vecs + v) * 16) = *reinterpret_cast<const uint4 *>(o[0]);
    } else {
      float f[8];
      if (v * 8 + 8 <= a.cols && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        const float4 f0 = *reinterpret_cast<const float4 *>(x + v * 8), f1 = *reinterpret_cast<const float4 *>(x + v * 8 + 4);
        f[0] = f0.x;
        f[1] = f0.y;
        f[2] = f0.z;
        f[3] = f0.w;
        f[4] = f1.x;
        f[5] = f1.y;
        f[6] = f1.z;
        f[7] = f1.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = v * 8 + j < a.cols ? x[v * 8 + j] : 0.f;
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
    a.fd_vecs = make_fastdiv(a.vecs);
    a.elem_bytes = r.elem_bytes;
    a.mode = r.mode;
    a.weights = r.weights ? 1 : 0;
    a.mid = r.mid ? r.mid : r.rows;
    a.parts = r.lattice.parts;
    a.sub_w = r.lattice.sub_w;
    a.sub_h = r.lattice.sub_h;
    a.full_w = r.lattice.full_w;
    a.full_h = r.lattice.full_h;
    a.step_w = r.lattice.step_w;
    a.step_h = r.lattice.step_h;
    const uint64_t per_block = kRepackThreads * kRepackPerThread;
    const uint64_t b = (r.rows * a.vecs + per_block - 1) / per_block;
    if (b + blocks[0] > 0x7fffffffull || uint64_t(a.vecs) + per_block > 0x7fffffffull)
      return fail(PLB_ERR_UNSUPPORTED, "operand too large to be repacked");
    blocks[used++] = unsigned(b);
  }
  if (used == 0) return PLB_OK;
  return launchPdl(ctx, repackKernel, dim3(blocks[0] + blocks[1]), dim3(kRepackThreads), 0, args[0], args[1],
                   blocks[0]);
}

}  // namespace plb
