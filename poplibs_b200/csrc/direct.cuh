// Matrix product kernel for small products:  D = alpha * A * B (+ beta * C).
//
// The implicit-GEMM kernel (igemm_sm100.cuh) needs rows at multiples of 16 bytes.
// Ragged rows, float operands and transposed quarter ones reach it through a copy, a
// launch more, which on a small product takes longer than the contraction, as does the
// set-up of tensor memory, tensor maps and a pipeline.  Here every thread loads what its
// block needs from the operands where they lie, eight elements at a time, from any
// address, converts them on the way to shared memory (float to two bfloat16 pieces,
// quarter to half) and the warps multiply with mma.sync.  The warps share out the K range
// besides the tile, so that a short product is one or two round trips to memory.  Bound by
// the latency of those and by the launch; the rate of mma.sync (a fraction of tcgen05's)
// and the work of a load from any address matter once there is more to do than that,
// which is where the dispatch (direct.cu) draws the line.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "direct.h"
#include "sm100_prims.cuh"

namespace plb {

constexpr int kDirectTeam = 256, kDirectTeams = 2;  // threads of a team, most teams
constexpr int kDirectStages = 4;                    // of operands that are copied as they are

struct DirectArgs {
  const uint8_t *a, *b;
  long long a_pitch, b_pitch, a_group, b_group;  // bytes
  int m, n, k, n_tiles, groups;
  FastDiv fd_groups, fd_n;
  int fmt_a, fmt_b;        // plb_quarter_format
  void *out;
  const void *addend;
  long long ldc, out_group, addend_ld, addend_group;  // elements
  int out_vec;             // four output columns are one aligned store
  float alpha, beta;
  int out_f32;
};

// Tile of a block: BM rows x BN columns.  A team of kM x kN x kK warps covers the tile
// and, kK ways, a K step of kStep elements; the teams of a block (one or two) take
// alternate steps, each at its own pace.
template <int kBM, int kBN, int kWarpsM, int kWarpsN, int kWarpsK, int kKStep>
struct DirectShape {
  static constexpr int BM = kBM, BN = kBN, M = kWarpsM, N = kWarpsN, K = kWarpsK, kStep = kKStep;
  static_assert(kWarpsM * kWarpsN * kWarpsK * 32 == kDirectTeam, "eight warps");
  static constexpr int kPitch = kBN + 8;  // floats of a row of sums
  // per team: 16-bit tiles of both operands (float: in two pieces) per stage, or the
  // warps' sums
  static constexpr int kTiles = (kBM + kBN) * kKStep * 2, kSums = kWarpsK * kBM * kPitch * 4;
  template <int kType, bool kVec> static constexpr int kStages = kType == PLB_HALF && kVec ? kDirectStages : 2;
  template <int kType, bool kVec> static constexpr int kStageBytes = kStages<kType, kVec> * kTiles * (kType == PLB_FLOAT ? 2 : 1);
  template <int kType, bool kVec>
  static constexpr int kSmem = kStageBytes<kType, kVec> > kSums ? kStageBytes<kType, kVec> : kSums;
};

// ---- eight elements of an operand -----------------------------------------------
// Loaded raw, so that all loads of a step are in flight before the first is looked at.
// load: all eight exist (kVec: at a multiple of a whole load); loadSome: the first `n`,
// the rest zero.  A load from any address reads the aligned 16-byte vectors (quarter:
// words) that hold the elements, which lie in the same allocation.
template <int kType, bool kVec> struct DirectUnit;

// 16-bit elements: two aligned vectors, shifted into place.  (Five aligned words are fewer
// instructions, but their lanes lie 16 bytes apart: 2.5 times the passes through L1.)
template <bool kVec> struct DirectUnit<PLB_HALF, kVec> {
  static constexpr int kBytes = 2, kPlanes = 1, kWords = kVec ? 4 : 8;
  uint32_t w[kWords];
  uint32_t off;
  __device__ __forceinline__ void put(int at, const uint4 &v) {
    w[at] = v.x;
    w[at + 1] = v.y;
    w[at + 2] = v.z;
    w[at + 3] = v.w;
  }
  __device__ __forceinline__ void load(const uint8_t *p) {
    if constexpr (kVec) {
      put(0, *reinterpret_cast<const uint4 *>(p));
    } else {
      off = uint32_t(reinterpret_cast<uintptr_t>(p)) & 15;
      const uint4 *x = reinterpret_cast<const uint4 *>(p - off);
      put(0, x[0]);
      put(4, off ? x[1] : make_uint4(0u, 0u, 0u, 0u));
    }
  }
  __device__ __forceinline__ void loadSome(const uint8_t *p, int n) {
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    if constexpr (kVec) {
      put(0, n > 0 ? *reinterpret_cast<const uint4 *>(p) : zero);
      keep(n);
    } else {
      off = uint32_t(reinterpret_cast<uintptr_t>(p)) & 15;
      const uint4 *x = reinterpret_cast<const uint4 *>(p - off);
      put(0, n > 0 ? x[0] : zero);
      put(4, n > 0 && int(off) + 2 * min(n, 8) > 16 ? x[1] : zero);
      place();
      keep(n);
      off = 0u;
    }
  }
  // the first n elements, the rest zero
  __device__ __forceinline__ void keep(int n) {
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = n >= 2 * j + 2 ? w[j] : n == 2 * j + 1 ? w[j] & 0xffffu : 0u;
  }
  // the elements to the front
  __device__ __forceinline__ void place() {
    const bool two = (off & 8) != 0, one = (off & 4) != 0;
#pragma unroll
    for (int j = 0; j < 6; ++j) w[j] = two ? w[j + 2] : w[j];
#pragma unroll
    for (int j = 0; j < 5; ++j) w[j] = one ? w[j + 1] : w[j];
    const uint32_t shift = (off & 2) * 8;
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = __funnelshift_r(w[j], w[j + 1], shift);
  }
  __device__ __forceinline__ void store(uint32_t dst, uint32_t, int, int &) {
    if constexpr (!kVec) place();
    st_shared_v4(dst, w[0], w[1], w[2], w[3]);
  }
};

// Eight quarters as halves, which hold every one of them exactly.
template <bool kVec> struct DirectUnit<PLB_QUARTER, kVec> {
  static constexpr int kBytes = 1, kPlanes = 1;
  uint32_t w[3];
  uint32_t shift;
  __device__ __forceinline__ void load(const uint8_t *p) {
    if constexpr (kVec) {
      const uint2 v = *reinterpret_cast<const uint2 *>(p);
      w[0] = v.x;
      w[1] = v.y;
      w[2] = shift = 0u;
    } else {
      const uint32_t off = uint32_t(reinterpret_cast<uintptr_t>(p)) & 3;
      const uint32_t *x = reinterpret_cast<const uint32_t *>(p - off);
      shift = off * 8;
      w[0] = x[0];
      w[1] = x[1];
      w[2] = off ? x[2] : 0u;
    }
  }
  __device__ __forceinline__ void loadSome(const uint8_t *p, int n) {
    const uint32_t off = uint32_t(reinterpret_cast<uintptr_t>(p)) & 3;
    const uint32_t *x = reinterpret_cast<const uint32_t *>(p - off);
    const int bytes = n > 0 ? int(off) + min(n, 8) : 0;
#pragma unroll
    for (int j = 0; j < 3; ++j) w[j] = 4 * j < bytes ? x[j] : 0u;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint32_t v = __funnelshift_r(w[j], w[j + 1], off * 8);
      const int rest = n - 4 * j;
      w[j] = rest >= 4 ? v : rest <= 0 ? 0u : v & ((1u << (8 * rest)) - 1);
    }
    w[2] = shift = 0u;
  }
  __device__ __forceinline__ void store(uint32_t dst, uint32_t, int fmt, int &) {
    const __nv_fp8_interpretation_t f = fmt == PLB_F152 ? __NV_E5M2 : __NV_E4M3;
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t v = kVec ? w[j / 2] : __funnelshift_r(w[j / 2], w[j / 2 + 1], shift);
      const __half2_raw r = __nv_cvt_fp8x2_to_halfraw2(__nv_fp8x2_storage_t(v >> (j % 2 * 16)), f);
      o[j] = uint32_t(r.x) | uint32_t(r.y) << 16;
    }
    st_shared_v4(dst, o[0], o[1], o[2], o[3]);
  }
};

// Floats as x_hi + x_lo, x_hi = bf16(x), x_lo = bf16(x - x_hi) (0 where x is not finite,
// which sets `odd`).
template <bool kVec> struct DirectUnit<PLB_FLOAT, kVec> {
  static constexpr int kBytes = 4, kPlanes = 2, kWords = kVec ? 8 : 12;
  float f[kWords];
  uint32_t off;
  __device__ __forceinline__ void load(const uint8_t *p) {
    off = kVec ? 0u : uint32_t(reinterpret_cast<uintptr_t>(p)) & 15;
    const float4 *v = reinterpret_cast<const float4 *>(p - off);
    *reinterpret_cast<float4 *>(&f[0]) = v[0];
    *reinterpret_cast<float4 *>(&f[4]) = v[1];
    if constexpr (!kVec) *reinterpret_cast<float4 *>(&f[8]) = off ? v[2] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __device__ __forceinline__ void loadSome(const uint8_t *p, int n) {
    off = kVec ? 0u : uint32_t(reinterpret_cast<uintptr_t>(p)) & 15;
    const float4 *v = reinterpret_cast<const float4 *>(p - off);
    const int bytes = n > 0 ? int(off) + 4 * min(n, 8) : 0;
#pragma unroll
    for (int j = 0; j < kWords / 4; ++j)
      *reinterpret_cast<float4 *>(&f[4 * j]) = 16 * j < bytes ? v[j] : make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (!kVec) place();
    off = 0u;
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = j < n ? f[j] : 0.f;
  }
  // the elements to the front
  __device__ __forceinline__ void place() {
    const bool two = (off & 8) != 0, one = (off & 4) != 0;
#pragma unroll
    for (int j = 0; j < 10; ++j) f[j] = two ? f[j + 2] : f[j];
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = one ? f[j + 1] : f[j];
  }
  __device__ __forceinline__ void store(uint32_t dst, uint32_t plane, int, int &odd) {
    if constexpr (!kVec) place();
    uint32_t hi[4], lo[4];
    __nv_bfloat162 most;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
      hi[j] = *reinterpret_cast<const uint32_t *>(&h);
      const __nv_bfloat162 l = __floats2bfloat162_rn(f[2 * j] - __uint_as_float(hi[j] << 16),
                                                     f[2 * j + 1] - __uint_as_float(hi[j] & 0xffff0000u));
      lo[j] = *reinterpret_cast<const uint32_t *>(&l);
      most = j == 0 ? l : __hmax2_nan(most, l);
    }
    if (!__hbeq2(most, most)) {  // (the low piece of what is not finite is a NaN)
      odd = 1;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        lo[j] &= (isfinite(f[2 * j]) ? 0xffffu : 0u) | (isfinite(f[2 * j + 1]) ? 0xffff0000u : 0u);
    }
    st_shared_v4(dst, hi[0], hi[1], hi[2], hi[3]);
    st_shared_v4(dst + plane, lo[0], lo[1], lo[2], lo[3]);
  }
};

// 16 bytes straight to shared memory, the first `bytes` of them read, the rest zero.
__device__ __forceinline__ void copyAsync(uint32_t dst, const uint8_t *src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// ---- shared-memory tiles -----------------------------------------------------------
// Rows of kChunks 16-byte chunks; the chunk number is XORed so that eight rows' chunks of
// one column lie in different banks.
template <int kChunks> __device__ __forceinline__ uint32_t directAt(uint32_t row, uint32_t chunk) {
  constexpr int kShift = kChunks >= 8 ? 0 : kChunks == 4 ? 1 : kChunks == 2 ? 2 : 3;
  constexpr uint32_t kMask = kChunks >= 8 ? 7 : kChunks - 1;
  return (row * kChunks + (chunk ^ ((row >> kShift) & kMask))) * 16;
}

template <bool kTrans> __device__ __forceinline__ void loadMatrices(uint32_t at, uint32_t (&r)[4]) {
  if constexpr (kTrans)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}

template <bool kBf16>
__device__ __forceinline__ void multiply(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (kBf16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The finite ones of two bfloat16s, zero for the others.
__device__ __forceinline__ uint32_t finitePair(uint32_t v) {
  return v & (((v & 0x7f80u) == 0x7f80u ? 0u : 0xffffu) | ((v & 0x7f800000u) == 0x7f800000u ? 0u : 0xffff0000u));
}

// A team's sums: warp (wm, wn, wk) adds its TM x TN part over its share of the step.
// kAMn / kBMn: the tile lies [k][m] / [k][n], else [m][k] / [n][k].  Float operands as
// a_hi*b_hi + a_lo*b_hi + a_hi*b_lo; with `odd` (an infinity or NaN in the block's
// operands) it stays in the first product alone: the others would multiply it with a
// zero piece.
template <int kType, class S, bool kAMn, bool kBMn>
struct DirectTile {
  static constexpr int kStep = S::kStep, TM = S::BM / S::M, TN = S::BN / S::N, KW = kStep / S::K;
  static constexpr int kPlanes = kType == PLB_FLOAT ? 2 : 1;
  static constexpr uint32_t kABytes = S::BM * kStep * 2, kBBytes = S::BN * kStep * 2;
  static constexpr uint32_t kBuffer = kPlanes * (kABytes + kBBytes);
  static constexpr int kAChunks = (kAMn ? S::BM : kStep) / 8, kBChunks = (kBMn ? S::BN : kStep) / 8;
  static_assert(TM % 16 == 0 && TN % 16 == 0 && KW % 16 == 0, "whole instructions");
  float acc[TM / 16][TN / 8][4];

  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < TM / 16; ++i)
#pragma unroll
      for (int j = 0; j < TN / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
  }
  __device__ __forceinline__ void step(uint32_t a_tile, uint32_t b_tile, bool odd) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x % kDirectTeam / 32;
    const uint32_t wm = warp % S::M, wn = warp / S::M % S::N, wk = warp / (S::M * S::N);
#pragma unroll
    for (int kk = 0; kk < KW; kk += 16) {
      const uint32_t k = wk * KW + kk;
      uint32_t a[kPlanes][TM / 16][4], b[kPlanes][TN / 16][4];
#pragma unroll
      for (int p = 0; p < kPlanes; ++p) {
#pragma unroll
        for (int i = 0; i < TM / 16; ++i) {
          const uint32_t m = wm * TM + i * 16;
          const uint32_t at = kAMn ? directAt<kAChunks>(k + (lane & 7) + (lane >> 4) * 8, m / 8 + ((lane >> 3) & 1))
                                   : directAt<kAChunks>(m + (lane & 15), k / 8 + (lane >> 4));
          loadMatrices<kAMn>(a_tile + p * kABytes + at, a[p][i]);
        }
#pragma unroll
        for (int j = 0; j < TN / 16; ++j) {
          const uint32_t n = wn * TN + j * 16;
          const uint32_t at = kBMn ? directAt<kBChunks>(k + (lane & 15), n / 8 + (lane >> 4))
                                   : directAt<kBChunks>(n + (lane & 7) + (lane >> 4) * 8, k / 8 + ((lane >> 3) & 1));
          loadMatrices<kBMn>(b_tile + p * kBBytes + at, b[p][j]);
        }
      }
      constexpr bool kBf16 = kType == PLB_FLOAT;
#pragma unroll
      for (int i = 0; i < TM / 16; ++i)
#pragma unroll
        for (int j = 0; j < TN / 8; ++j)
          multiply<kBf16>(acc[i][j], a[0][i], b[0][j / 2][j % 2 * 2], b[0][j / 2][j % 2 * 2 + 1]);
      if constexpr (kPlanes == 2) {
        if (odd) {
#pragma unroll
          for (int i = 0; i < TM / 16; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) a[0][i][e] = finitePair(a[0][i][e]);
#pragma unroll
          for (int j = 0; j < TN / 16; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) b[0][j][e] = finitePair(b[0][j][e]);
        }
#pragma unroll
        for (int i = 0; i < TM / 16; ++i)
#pragma unroll
          for (int j = 0; j < TN / 8; ++j) {
            multiply<kBf16>(acc[i][j], a[1][i], b[0][j / 2][j % 2 * 2], b[0][j / 2][j % 2 * 2 + 1]);
            multiply<kBf16>(acc[i][j], a[0][i], b[1][j / 2][j % 2 * 2], b[1][j / 2][j % 2 * 2 + 1]);
          }
      }
    }
  }
  // -> rows of S::kPitch floats, one set per share of K
  __device__ __forceinline__ void leave(float *sums) const {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x % kDirectTeam / 32;
    const uint32_t wm = warp % S::M, wn = warp / S::M % S::N, wk = warp / (S::M * S::N);
    float *mine = sums + wk * (S::BM * S::kPitch) + (wm * TM + lane / 4) * S::kPitch + wn * TN + lane % 4 * 2;
#pragma unroll
    for (int i = 0; i < TM / 16; ++i)
#pragma unroll
      for (int j = 0; j < TN / 8; ++j) {
        float *at = mine + i * 16 * S::kPitch + j * 8;
        *reinterpret_cast<float2 *>(at) = make_float2(acc[i][j][0], acc[i][j][1]);
        *reinterpret_cast<float2 *>(at + 8 * S::kPitch) = make_float2(acc[i][j][2], acc[i][j][3]);
      }
  }
};

// kVec: rows of both operands start at multiples of a whole load.
template <int kType, class S, bool kAMn, bool kBMn, bool kVec>
__global__ void __launch_bounds__(kDirectTeam * kDirectTeams)
directKernel(const __grid_constant__ DirectArgs g) {
  using Unit = DirectUnit<kType, kVec>;
  using Tile = DirectTile<kType, S, kAMn, kBMn>;
  constexpr int kStep = Tile::kStep, es = Unit::kBytes;
  extern __shared__ __align__(16) uint8_t direct_smem[];
  __shared__ int odd_flag;
  pdl_launch_dependents();
  const int tid = int(threadIdx.x) % kDirectTeam, team = int(threadIdx.x) / kDirectTeam, teams = int(blockDim.x) / kDirectTeam;
  const uint32_t smem = smem_u32(direct_smem) + team * S::template kSmem<kType, kVec>;
  const uint32_t by_group = fast_div(blockIdx.x, g.fd_groups);
  const int group = int(blockIdx.x - by_group * g.groups);
  const uint32_t mt = fast_div(by_group, g.fd_n);
  const int m0 = int(mt) * S::BM, n0 = int(by_group - mt * g.n_tiles) * S::BN;

  // An operand's tile is rows of units: rows of m (or n) and units of k, or the other way
  // round.  Thread t takes unit t % units of rows t / units, + step, ...
  constexpr int kAUnits = (kAMn ? S::BM : kStep) / 8, kARows = kAMn ? kStep : S::BM, kAStep = kDirectTeam / kAUnits;
  constexpr int kBUnits = (kBMn ? S::BN : kStep) / 8, kBRows = kBMn ? kStep : S::BN, kBStep = kDirectTeam / kBUnits;
  constexpr int NA = (kARows + kAStep - 1) / kAStep, NB = (kBRows + kBStep - 1) / kBStep;
  constexpr bool kAWhole = kARows % kAStep == 0, kBWhole = kBRows % kBStep == 0;
  const int a_row = tid / kAUnits, a_col = tid % kAUnits * 8, b_row = tid / kBUnits, b_col = tid % kBUnits * 8;
  const uint8_t *pa = g.a + group * g.a_group + (kAMn ? a_row * g.a_pitch + (m0 + a_col) * es : (m0 + a_row) * g.a_pitch + a_col * es);
  const uint8_t *pb = g.b + group * g.b_group + (kBMn ? b_row * g.b_pitch + (n0 + b_col) * es : (n0 + b_row) * g.b_pitch + b_col * es);
  // (a team's first step, and from one of its steps to the next)
  const long long a_step = kAMn ? kStep * g.a_pitch : kStep * es, b_step = kBMn ? kStep * g.b_pitch : kStep * es;
  pa += team * a_step;
  pb += team * b_step;
  const long long a_down = kAStep * g.a_pitch, b_down = kBStep * g.b_pitch;

  Tile t;
  t.clear();
  if constexpr (kType == PLB_FLOAT) {
    if (threadIdx.x == 0) odd_flag = 0;
    __syncthreads();
  }
  pdl_wait();  // operands may come from the previous kernel in the stream
  const int steps = (g.k + kStep - 1) / kStep, mine = (steps - team + teams - 1) / teams;
  const auto barrier = [&] { asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(kDirectTeam) : "memory"); };
  if constexpr (kVec && kType == PLB_HALF) {
    // Nothing to convert: copies go straight to shared memory, several steps ahead.
    constexpr int kStages = S::template kStages<kType, kVec>;
    auto copy = [&](int i) {
      const uint32_t buffer = smem + (i % kStages) * Tile::kBuffer;
      const int k0 = (i * teams + team) * kStep;
      const int a_left = kAMn ? g.m - m0 - a_col : g.k - k0 - a_col, a_rows = kAMn ? g.k - k0 : g.m - m0;
      const int b_left = kBMn ? g.n - n0 - b_col : g.k - k0 - b_col, b_rows = kBMn ? g.k - k0 : g.n - n0;
#pragma unroll
      for (int j = 0; j < NA; ++j) {
        const int row = a_row + j * kAStep, n = row < a_rows ? min(max(a_left, 0), 8) : 0;
        if (kAWhole || row < kARows) copyAsync(buffer + directAt<Tile::kAChunks>(row, a_col / 8), n ? pa + j * a_down : g.a, 2 * n);
      }
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const int row = b_row + j * kBStep, n = row < b_rows ? min(max(b_left, 0), 8) : 0;
        if (kBWhole || row < kBRows)
          copyAsync(buffer + Tile::kABytes + directAt<Tile::kBChunks>(row, b_col / 8), n ? pb + j * b_down : g.b, 2 * n);
      }
      pa += teams * a_step;
      pb += teams * b_step;
    };
#pragma unroll 1
    for (int i = 1 - kStages; i < mine; ++i) {
      const int ahead = i + kStages - 1;
      if (i >= 0) {
        // (all but the newest kStages - 2 groups: step i's)
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        barrier();  // everyone's copies of step i are there, and step i - 1 has been read
      }
      if (ahead < mine) copy(ahead);
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (i >= 0) {
        const uint32_t buffer = smem + (i % kStages) * Tile::kBuffer;
        t.step(buffer, buffer + Tile::kABytes, false);
      }
    }
    barrier();
  } else {
    const bool inside = m0 + S::BM <= g.m && n0 + S::BN <= g.n;
    Unit ua[NA], ub[NB];
    auto load = [&](int k0) {
      if (inside && k0 + kStep <= g.k) {
#pragma unroll
        for (int i = 0; i < NA; ++i)
          if (kAWhole || a_row + i * kAStep < kARows) ua[i].load(pa + i * a_down);
#pragma unroll
        for (int i = 0; i < NB; ++i)
          if (kBWhole || b_row + i * kBStep < kBRows) ub[i].load(pb + i * b_down);
      } else {
        // (at the edges only what exists is read)
        const int a_left = kAMn ? g.m - m0 - a_col : g.k - k0 - a_col, a_rows = kAMn ? g.k - k0 : g.m - m0;
        const int b_left = kBMn ? g.n - n0 - b_col : g.k - k0 - b_col, b_rows = kBMn ? g.k - k0 : g.n - n0;
#pragma unroll
        for (int i = 0; i < NA; ++i) {
          const int n = a_row + i * kAStep < min(kARows, a_rows) ? a_left : 0;
          if (n >= 8)
            ua[i].load(pa + i * a_down);
          else
            ua[i].loadSome(pa + i * a_down, n);
        }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          const int n = b_row + i * kBStep < min(kBRows, b_rows) ? b_left : 0;
          if (n >= 8)
            ub[i].load(pb + i * b_down);
          else
            ub[i].loadSome(pb + i * b_down, n);
        }
      }
      pa += teams * a_step;
      pb += teams * b_step;
    };
    auto store = [&](uint32_t buffer) {
      int odd = 0;
#pragma unroll
      for (int i = 0; i < NA; ++i)
        if (kAWhole || a_row + i * kAStep < kARows)
          ua[i].store(buffer + directAt<Tile::kAChunks>(a_row + i * kAStep, a_col / 8), Tile::kABytes, g.fmt_a, odd);
      const uint32_t b = buffer + Tile::kPlanes * Tile::kABytes;
#pragma unroll
      for (int i = 0; i < NB; ++i)
        if (kBWhole || b_row + i * kBStep < kBRows)
          ub[i].store(b + directAt<Tile::kBChunks>(b_row + i * kBStep, b_col / 8), Tile::kBBytes, g.fmt_b, odd);
      if (kType == PLB_FLOAT && odd) *static_cast<volatile int *>(&odd_flag) = 1;
    };
    // a step's loads are in flight while the team's previous one is multiplied
#pragma unroll 1
    for (int i = 0; i <= mine; ++i) {
      if (i < mine) load((i * teams + team) * kStep);
      if (i > 0) {
        const uint32_t buffer = smem + ((i - 1) & 1) * Tile::kBuffer;
        t.step(buffer, buffer + Tile::kPlanes * Tile::kABytes, kType == PLB_FLOAT && *static_cast<volatile int *>(&odd_flag) != 0);
      }
      if (i < mine) store(smem + (i & 1) * Tile::kBuffer);
      barrier();
    }
  }

  // the warps' shares of K, added in order, then scale / add / cast
  float *const sums = reinterpret_cast<float *>(direct_smem);
  constexpr int kTeamFloats = S::template kSmem<kType, kVec> / 4, kSet = S::BM * S::kPitch;
  t.leave(sums + team * kTeamFloats);
  __syncthreads();
  const long long out0 = group * g.out_group, addend0 = group * g.addend_group;
  if (g.out_vec) {
#pragma unroll 1
    for (int i = int(threadIdx.x); i < S::BM * S::BN / 4; i += int(blockDim.x)) {
      const int r = i / (S::BN / 4), c = i % (S::BN / 4) * 4, row = m0 + r, col = n0 + c;
      if (row >= g.m || col >= g.n) continue;  // (n is a multiple of 4)
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int e = 0; e < teams; ++e)
#pragma unroll
        for (int k = 0; k < S::K; ++k) {
          const float4 u = *reinterpret_cast<const float4 *>(sums + e * kTeamFloats + k * kSet + r * S::kPitch + c);
          v.x += u.x;
          v.y += u.y;
          v.z += u.z;
          v.w += u.w;
        }
      v.x *= g.alpha;
      v.y *= g.alpha;
      v.z *= g.alpha;
      v.w *= g.alpha;
      if (g.addend) {
        const long long at = addend0 + row * g.addend_ld + col;
        auto add = [&](int j) {
          return g.beta * (g.out_f32 ? static_cast<const float *>(g.addend)[at + j]
                                     : __half2float(static_cast<const __half *>(g.addend)[at + j]));
        };
        v.x += add(0);
        v.y += add(1);
        v.z += add(2);
        v.w += add(3);
      }
      const long long at = out0 + row * g.ldc + col;
      if (g.out_f32) {
        *reinterpret_cast<float4 *>(static_cast<float *>(g.out) + at) = v;
      } else {
        const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
        *reinterpret_cast<uint2 *>(static_cast<__half *>(g.out) + at) =
            make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
      }
    }
  } else {
    // neighbouring threads, neighbouring columns
#pragma unroll 1
    for (int i = int(threadIdx.x); i < S::BM * S::BN; i += int(blockDim.x)) {
      const int r = i / S::BN, c = i % S::BN, row = m0 + r, col = n0 + c;
      if (row >= g.m || col >= g.n) continue;
      float v = 0.f;
      for (int e = 0; e < teams; ++e)
#pragma unroll
        for (int k = 0; k < S::K; ++k) v += sums[e * kTeamFloats + k * kSet + r * S::kPitch + c];
      v *= g.alpha;
      if (g.addend) {
        const long long at = addend0 + row * g.addend_ld + col;
        v += g.beta * (g.out_f32 ? static_cast<const float *>(g.addend)[at]
                                 : __half2float(static_cast<const __half *>(g.addend)[at]));
      }
      const long long at = out0 + row * g.ldc + col;
      if (g.out_f32)
        static_cast<float *>(g.out)[at] = v;
      else
        static_cast<__half *>(g.out)[at] = __float2half_rn(v);
    }
  }
}

// The shapes, by what a block covers.
using DirectFew = DirectShape<16, 32, 1, 1, 8, 256>;    // a handful of rows
using DirectSmall = DirectShape<32, 32, 1, 1, 8, 128>;  // few tiles: K over the warps
using DirectMid = DirectShape<32, 64, 1, 2, 4, 128>;
using DirectWide = DirectShape<64, 64, 2, 2, 2, 64>;

enum DirectKind : int { kDirectFew, kDirectSmall, kDirectMid, kDirectWide };

// Floats from any address hold three vectors for each unit in registers.  In blocks of 32 x 64
// they take 2.4 times as long as floats in whole loads, longer than in the others (112 x 685 x 2151
// 26.7 us, on the general route 17.9; 127 sampled products 0.72 of the time without that shape).
constexpr bool directHas(DirectKind kind, int type, bool whole) {
  return type != PLB_FLOAT || whole || kind != kDirectMid;
}

struct DirectVariant {
  DirectKind kind;
  bool a_mn, b_mn, vec;
  unsigned blocks, teams;
};
int launchDirectHalf(plb_context *ctx, const DirectVariant &v, const DirectArgs &g);
int launchDirectFloat(plb_context *ctx, const DirectVariant &v, const DirectArgs &g);
int launchDirectQuarter(plb_context *ctx, const DirectVariant &v, const DirectArgs &g);

}  // namespace plb
