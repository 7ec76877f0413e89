// Per-channel sums over, and element-wise maps with per-channel operands of,
// device-layout activations [rows][chans] (NHWC: the channels of a pixel are
// contiguous): what batch normalisation and the bias of a convolution are made
// of.
//
// Every operation here moves each element once or twice and does a handful of
// flops on it, so it is bound by memory as long as enough 16-byte accesses are
// in flight and nothing is recomputed per element.  Both forms therefore view
// the tensor as SUPER-ROWS: the fewest rows whose elements are a whole number of
// 16-byte vectors (1 row if the channel count is a multiple of the vector, up to
// 8 if it is odd).  A vector's place inside its super-row fixes which channels it
// holds, so a thread that keeps one place and walks the super-rows keeps its
// per-channel operands (or sums) in registers, loads whole vectors at any channel
// count, and never divides.  Only the last, partial super-row is done element by
// element.  A tensor whose base is not 16-byte aligned takes vectors of one element.
#pragma once

#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>

#include "runtime.h"
#include "sm100_prims.cuh"

namespace plb {

template <typename T> __device__ __forceinline__ float toFloat(T v);
template <> __device__ __forceinline__ float toFloat<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float toFloat<float>(float v) { return v; }
template <typename T> __device__ __forceinline__ T fromFloat(float v);
template <> __device__ __forceinline__ __half fromFloat<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ float fromFloat<float>(float v) { return v; }

// A vector of V elements as it is loaded and stored.
template <typename T, int V> struct ChanVec {
  using Raw = uint4;
  static_assert(V * sizeof(T) == 16, "a vector is 16 bytes, or one element");
  static __device__ __forceinline__ void unpack(const Raw &v, float (&f)[V]) {
    if constexpr (sizeof(T) == 2) {
      const __half2 *h = reinterpret_cast<const __half2 *>(&v);
#pragma unroll
      for (int j = 0; j < V / 2; ++j) {
        const float2 t = __half22float2(h[j]);
        f[2 * j] = t.x;
        f[2 * j + 1] = t.y;
      }
    } else {
      f[0] = __uint_as_float(v.x);
      f[1] = __uint_as_float(v.y);
      f[2] = __uint_as_float(v.z);
      f[3] = __uint_as_float(v.w);
    }
  }
  static __device__ __forceinline__ Raw pack(const float (&f)[V]) {
    Raw v;
    if constexpr (sizeof(T) == 2) {
      __half2 *h = reinterpret_cast<__half2 *>(&v);
#pragma unroll
      for (int j = 0; j < V / 2; ++j) h[j] = __floats2half2_rn(f[2 * j], f[2 * j + 1]);
    } else {
      v = make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
    }
    return v;
  }
};
template <typename T> struct ChanVec<T, 1> {
  using Raw = T;
  static __device__ __forceinline__ void unpack(const Raw &v, float (&f)[1]) { f[0] = toFloat(v); }
  static __device__ __forceinline__ Raw pack(const float (&f)[1]) { return fromFloat<T>(f[0]); }
};

// Two neighbouring elements in one load.
template <typename T> struct ChanPair;
template <> struct ChanPair<__half> {
  using Type = __half2;
  static __device__ __forceinline__ void unpack(Type v, float (&f)[2]) {
    const float2 t = __half22float2(v);
    f[0] = t.x;
    f[1] = t.y;
  }
};
template <> struct ChanPair<float> {
  using Type = float2;
  static __device__ __forceinline__ void unpack(Type v, float (&f)[2]) {
    f[0] = v.x;
    f[1] = v.y;
  }
};

// How [rows][chans] is walked.  A block is vec_lanes x row_lanes threads: thread
// (vx, ry) owns vector `blockIdx.x * vec_lanes + vx` of the super-rows ry,
// ry + stride, ... of its slab blockIdx.y.
struct ChanWalk {
  uint32_t chans;
  uint32_t fold;             // rows per super-row
  uint32_t vecs;             // vectors per super-row
  uint32_t vec_lanes_log2;   // <= 5
  uint32_t slabs;            // gridDim.y
  unsigned long long full;   // whole super-rows
  unsigned long long total;  // elements of the tensor
};

// `per_sm`: blocks of `threads` threads wanted per SM once there is work for them.
// `most_slabs`: a cap on the slabs besides that (0: none).
inline ChanWalk chanWalk(const plb_context *ctx, uint64_t rows, uint32_t chans, uint32_t V, uint32_t threads,
                         uint32_t per_sm, uint32_t rows_each, uint64_t most_slabs, dim3 *grid) {
  ChanWalk w{};
  w.chans = chans;
  uint32_t g = chans, t = V;  // gcd
  while (t) {
    const uint32_t u = g % t;
    g = t;
    t = u;
  }
  w.fold = V / g;
  w.vecs = chans / g;  // = fold * chans / V
  w.full = rows / w.fold;
  w.total = rows * chans;
  // vectors side by side in a block: at least 64 bytes of a row, as many as leave
  // the fewest threads without a vector
  while (w.vec_lanes_log2 < 2 && (1u << w.vec_lanes_log2) < w.vecs) ++w.vec_lanes_log2;
  for (uint32_t l = w.vec_lanes_log2 + 1; l <= 5; ++l)
    if (((w.vecs + (1u << l) - 1) >> l << l) <= ((w.vecs + (1u << w.vec_lanes_log2) - 1) >> w.vec_lanes_log2 << w.vec_lanes_log2))
      w.vec_lanes_log2 = l;
  const uint32_t lanes = 1u << w.vec_lanes_log2, row_lanes = threads >> w.vec_lanes_log2;
  const uint32_t cols = (w.vecs + lanes - 1) / lanes;
  // rows_each super-rows per thread while that leaves SMs idle, then a grid that is
  // resident at once and walks
  const uint64_t slab = uint64_t(row_lanes) * rows_each, want = std::max<uint64_t>(1, (w.full + slab - 1) / slab);
  uint64_t cap = std::max<uint64_t>(1, uint64_t(ctx->sm_count) * per_sm / cols);
  if (most_slabs) cap = std::min(cap, most_slabs);
  w.slabs = uint32_t(std::min<uint64_t>(std::min(want, cap), 65535));
  *grid = dim3(cols, w.slabs);
  return w;
}

// ---- sums ------------------------------------------------------------------------

// What is added up per channel (two sums at once).
enum ChanSums : int {
  kSumXAndXX = 0,     // sum x, sum x^2
  kSumCentredXX = 1,  // -, sum (x - centre[c])^2     (centre in the activations' type)
  kSumXYAndY = 2,     // sum x * y, sum y             (whitened activations x gradients)
  kSumX = 3,          // sum x, -
};

// What becomes of the sums: a = scale * first sum, b = scale * second sum.  Any
// pointer may be null; *_half says which of the two types it points to.
struct ChanFinish {
  float scale;
  void *a, *b;
  float *a_f32, *b_f32;  // the same in fp32
  int a_half, b_half;
  // 1 / sqrt((b - a^2 + eps) * scale_var), a rounded to its type first
  void *inv_std;
  float eps, scale_var;
  // bias[c] += a
  void *bias;
  int bias_half;
  int totals_fit;  // (set by chanSums) the last block can hold all column totals in shared memory
};

__device__ __forceinline__ void storeChan(void *p, int is_half, uint32_t c, float v) {
  if (is_half)
    static_cast<__half *>(p)[c] = __float2half_rn(v);
  else
    static_cast<float *>(p)[c] = v;
}

template <typename T>
__device__ __forceinline__ void finishChan(const ChanFinish &fin, uint32_t c, float sa, float sb) {
  const float va = __fmul_rn(sa, fin.scale), vb = __fmul_rn(sb, fin.scale);
  if (fin.a) storeChan(fin.a, fin.a_half, c, va);
  if (fin.b) storeChan(fin.b, fin.b_half, c, vb);
  if (fin.a_f32) fin.a_f32[c] = va;
  if (fin.b_f32) fin.b_f32[c] = vb;
  if (fin.inv_std) {
    // plb_norm_inv_std_dev's arithmetic on the values as stored: the mean
    // rounded to its type, the power in fp32
    const float mean = toFloat(fromFloat<T>(va));
    float var = vb - mean * mean;
    if (var < 0.f) var = 0.f;
    var = (var + fin.eps) * fin.scale_var;
    storeChan(fin.inv_std, fin.a_half, c, 1.0f / sqrtf(var));
  }
  if (fin.bias) {
    const float old = fin.bias_half ? __half2float(static_cast<const __half *>(fin.bias)[c])
                                    : static_cast<const float *>(fin.bias)[c];
    storeChan(fin.bias, fin.bias_half, c, old + va);
  }
}

// What one element adds to the two sums; m is the centre.
template <typename T, int kMode>
__device__ __forceinline__ void addElement(float &a, float &b, float x, float y, float m) {
  if constexpr (kMode == kSumXAndXX) {
    a += x;
    b += x * x;
  } else if constexpr (kMode == kSumCentredXX) {
    // the deviation is formed in the activations' type, as the reference's
    // "acts - cast(mean)" map does (lib/poplin/Norms.cpp:216-219)
    const float d = toFloat(fromFloat<T>(x - m));
    b += d * d;
  } else if constexpr (kMode == kSumXYAndY) {
    a += x * y;
    b += y;
  } else {
    a += x;
  }
}

// The sums of the threads of a warp that hold the same vector (thread numbers that
// differ in bits `lanes` and up): in each step a thread hands half of its columns to
// its partner and takes the partner's sums of the other half, so that V columns cost
// V - 1 shuffles instead of V per step (two sums of 8 columns in 8 lanes: 12
// instead of 32, which at 32 warps a block are 0.3 us).
template <int V, bool kHasA, bool kHasB, int D>
__device__ __forceinline__ void foldWarp(float *a, float *b, uint32_t lanes, uint32_t &first, uint32_t &held,
                                         bool &writes) {
  if constexpr (D > 0) {
    if (uint32_t(D) < lanes) return;
    const bool upper = (threadIdx.x & D) != 0;
    constexpr int kStep = D == 16 ? 0 : D == 8 ? 1 : D == 4 ? 2 : D == 2 ? 3 : 4;
    constexpr int n = (V >> kStep) < 1 ? 1 : V >> kStep;  // columns held so far
    if constexpr (n > 1) {
#pragma unroll
      for (int j = 0; j < n / 2; ++j) {
        if constexpr (kHasA) {
          const float give = upper ? a[j] : a[j + n / 2], keep = upper ? a[j + n / 2] : a[j];
          a[j] = keep + __shfl_xor_sync(0xffffffffu, give, D);
        }
        if constexpr (kHasB) {
          const float give = upper ? b[j] : b[j + n / 2], keep = upper ? b[j + n / 2] : b[j];
          b[j] = keep + __shfl_xor_sync(0xffffffffu, give, D);
        }
      }
      first += upper ? n / 2 : 0;
      held = n / 2;
    } else {
      if constexpr (kHasA) a[0] += __shfl_xor_sync(0xffffffffu, a[0], D);
      if constexpr (kHasB) b[0] += __shfl_xor_sync(0xffffffffu, b[0], D);
      writes = writes && !upper;
    }
    foldWarp<V, kHasA, kHasB, D / 2>(a, b, lanes, first, held, writes);
  }
}

// One launch: every block leaves the sums of its slab as one row of the partial
// matrices [slabs * fold][chans], and the block that finishes last adds the rows.
// Rows are added in a fixed order, whichever block that is, so the result does
// not depend on timing.  One block per SM: few rows for the last block to add, and
// the 64 KB its threads have in flight (16 bytes x 4096 / kThreads loads each) are
// 9.7 MB over the device, above the 5 MB that 6.5 TB/s times the memory latency asks
// for.  Small tensors are bound by latency: a launch, four trips to L2 or memory
// (data, partial rows out, ticket, partial rows in) and what the warps of a block
// execute one after the other, so there are few warps (512 threads; the last block
// goes on with as few as its rows need) and few slabs.  Sums of 64 x 16 halves
// take 4.1 us, of 12544 x 36 5.8, of 100352 x 64 6.8 (with 1024 threads throughout 5.7, 6.7
// and 7.7); of 200704 x 128 (51 MB) 10.8; of 200704 x 256 (103 MB) 20.5 (5.0 TB/s;
// a read-only stream gets 5.6 here).
template <typename T, int kMode, int V, int kThreads>
__global__ void __launch_bounds__(kThreads, 1)
chanSumsKernel(const T *__restrict__ x, const T *__restrict__ y, const T *__restrict__ centre, const ChanWalk w,
               float *__restrict__ partial_a, float *__restrict__ partial_b, unsigned *__restrict__ ticket,
               const ChanFinish fin) {
  using Vec = ChanVec<T, V>;
  using Raw = typename Vec::Raw;
  constexpr bool kHasA = kMode != kSumCentredXX, kHasB = kMode != kSumX, kHasY = kMode == kSumXYAndY;
  constexpr int kLoads = 4096 / kThreads, kUnroll = kHasY ? kLoads / 2 : kLoads, kWarps = kThreads / 32;
  constexpr int kQuads = kThreads + kThreads / 2;  // float4s of the last block's table
  extern __shared__ float4 chan_smem[];
  float *red = reinterpret_cast<float *>(chan_smem);
  __shared__ unsigned last;
  pdl_launch_dependents();
  const uint32_t lanes = 1u << w.vec_lanes_log2, row_lanes = kThreads >> w.vec_lanes_log2;
  const uint32_t vx = threadIdx.x & (lanes - 1), ry = threadIdx.x >> w.vec_lanes_log2;
  const uint32_t vec = blockIdx.x * lanes + vx;
  const bool mine = vec < w.vecs;
  const size_t pitch = size_t(w.vecs) * V;
  float a[V], b[V];
  [[maybe_unused]] float m[V];
#pragma unroll
  for (int j = 0; j < V; ++j) a[j] = b[j] = 0.f;
  pdl_wait();  // inputs may come from the previous kernel in the stream
  if constexpr (kMode == kSumCentredXX) {
    if (mine)
#pragma unroll
      for (int j = 0; j < V; ++j) m[j] = toFloat(centre[(vec * V + j) % w.chans]);
  }
  auto add = [&](const float (&xv)[V], const float (&yv)[V], int j) {
    addElement<T, kMode>(a[j], b[j], xv[j], kHasY ? yv[j] : 0.f, kMode == kSumCentredXX ? m[j] : 0.f);
  };
  if (mine) {
    const size_t step = size_t(gridDim.y) * row_lanes;
    const T *px = x + size_t(vec) * V;
    const T *py = kHasY ? y + size_t(vec) * V : nullptr;
    for (size_t r = size_t(blockIdx.y) * row_lanes + ry; r < w.full; r += kUnroll * step) {
      Raw rx[kUnroll];
      [[maybe_unused]] Raw rv[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const size_t row = r + u * step;
        if (row < w.full) {
          rx[u] = *reinterpret_cast<const Raw *>(px + row * pitch);
          if constexpr (kHasY) rv[u] = *reinterpret_cast<const Raw *>(py + row * pitch);
        }
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        if (r + u * step < w.full) {
          float xv[V], yv[V];
          Vec::unpack(rx[u], xv);
          if constexpr (kHasY) Vec::unpack(rv[u], yv);
#pragma unroll
          for (int j = 0; j < V; ++j) add(xv, yv, j);
        }
      }
    }
    // the rows that do not fill a super-row
    if (w.fold > 1 && blockIdx.y == 0 && ry == 0) {
      const size_t base = w.full * pitch + size_t(vec) * V;
      float xv[V], yv[V];
#pragma unroll
      for (int j = 0; j < V; ++j)
        if (base + j < w.total) {
          xv[j] = toFloat(x[base + j]);
          if constexpr (kHasY) yv[j] = toFloat(y[base + j]);
          add(xv, yv, j);
        }
    }
  }
  // Threads of a warp that share a vector first, then the warps: `per` neighbouring
  // threads share the 32 warps' values of a column (both sums' columns at once; a
  // row pitch of cols + 1 words keeps them in different banks).  Every tree is
  // fixed, so the result does not depend on timing.
  const uint32_t warp = threadIdx.x >> 5, cols = lanes * V;
  const uint32_t block_col0 = blockIdx.x * cols;
  {
    constexpr uint32_t kSums = (kHasA ? 1 : 0) + (kHasB ? 1 : 0);
    float *rb = red + (kHasA ? kWarps * (cols + 1) : 0);
    uint32_t first = 0, held = V;  // the columns of the vector this thread ends up with
    bool writes = true;
    foldWarp<V, kHasA, kHasB, 16>(a, b, lanes, first, held, writes);
    if (writes)
#pragma unroll
      for (int j = 0; j < V; ++j)
        if (j < held) {
          if constexpr (kHasA) red[warp * (cols + 1) + vx * V + first + j] = a[j];
          if constexpr (kHasB) rb[warp * (cols + 1) + vx * V + first + j] = b[j];
        }
    __syncthreads();
    const uint32_t items = kSums * cols, per = min(uint32_t(kWarps), kThreads / items);  // powers of two
    const uint32_t item = threadIdx.x / per, part = threadIdx.x & (per - 1), rows = kWarps / per;
    float t = 0.f;
    const bool second = kHasA && item >= cols;
    const uint32_t col = second ? item - cols : item;
    if (item < items) {
      const float *r = (second ? rb : red) + part * rows * (cols + 1) + col;
#pragma unroll 4
      for (uint32_t k = 0; k < rows; ++k) t += r[k * (cols + 1)];
    }
    for (uint32_t d = per >> 1; d >= 1; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
    if (part == 0 && item < items && block_col0 + col < pitch)
      (second || !kHasA ? partial_b : partial_a)[size_t(blockIdx.y) * pitch + block_col0 + col] = t;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    // one thread's release publishes the block's stores (the barrier above orders
    // them before it), its acquire the other blocks' to this one
    unsigned before;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(ticket) : "memory");
    last = before == gridDim.x * gridDim.y - 1;
    if (last) *ticket = 0u;  // for the next launch in the stream
  }
  __syncthreads();
  if (!last) return;
  if constexpr (V > 1) {
    if (fin.totals_fit) {
      // The slabs' rows of `pitch` columns: four columns per thread, the rows shared
      // out between the threads of a column so that all are in flight at once, their
      // sums added through shared memory, then the rows of a super-row.
      // As few warps as that takes with eight rows and a few columns each.
      const uint32_t quads = uint32_t(pitch / 4);
      uint32_t t_log2 = 8;
      while ((1u << t_log2) < kThreads && ((8u << t_log2) < gridDim.y * quads || (1u << t_log2) < max(w.chans, 2 * quads))) ++t_log2;
      const uint32_t threads = 1u << t_log2;
      if (threadIdx.x >= threads) return;
      auto barrier = [&] { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); };
      uint32_t ql_log2 = 1;
      while (ql_log2 < 8 && (1u << ql_log2) < quads) ++ql_log2;
      const uint32_t ql = 1u << ql_log2, part_lanes = threads >> ql_log2;
      const uint32_t cl = threadIdx.x & (ql - 1), pl = threadIdx.x >> ql_log2;
      // (rows of ql + 1: neighbouring threads' reads below fall into different banks)
      float4 *sums_a = chan_smem, *sums_b = sums_a + kQuads;
      float *total_a = red + 8 * kQuads, *total_b = total_a + pitch;
      auto take = [](float4 &s, const float4 &v) {
        s.x += v.x;
        s.y += v.y;
        s.z += v.z;
        s.w += v.w;
      };
      for (uint32_t q0 = 0; q0 < quads; q0 += ql) {
        float4 sa = make_float4(0.f, 0.f, 0.f, 0.f), sb = sa;
        if (q0 + cl < quads) {
          const size_t at = size_t(q0 + cl) * 4;
#pragma unroll 4
          for (uint32_t k = pl; k < gridDim.y; k += part_lanes) {
            if constexpr (kHasA) take(sa, __ldcg(reinterpret_cast<const float4 *>(partial_a + k * pitch + at)));
            if constexpr (kHasB) take(sb, __ldcg(reinterpret_cast<const float4 *>(partial_b + k * pitch + at)));
          }
        }
        if (kHasA) sums_a[pl * (ql + 1) + cl] = sa;
        if (kHasB) sums_b[pl * (ql + 1) + cl] = sb;
        barrier();
        // columns of both sums over the threads, `per` neighbouring threads to a column
        const uint32_t cols4 = 4 * ql, items_log2 = ql_log2 + (kHasA && kHasB ? 3 : 2), items = 1u << items_log2;
        const uint32_t per_log2 = items_log2 >= t_log2 ? 0u : min(5u, t_log2 - max(items_log2, ql_log2));
        const uint32_t per = 1u << per_log2;
        for (uint32_t i0 = 0; i0 < items; i0 += threads >> per_log2) {
          const uint32_t item = i0 + (threadIdx.x >> per_log2), part = threadIdx.x & (per - 1);
          const bool second = kHasA && item >= cols4;
          const uint32_t col = second ? item - cols4 : item;
          float t = 0.f;
          if (item < items) {
            const float *src = reinterpret_cast<const float *>(second || !kHasA ? sums_b : sums_a);
#pragma unroll 4
            for (uint32_t k = part; k < part_lanes; k += per) t += src[k * (cols4 + 4) + col];
          }
          for (uint32_t d = per >> 1; d >= 1; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
          if (part == 0 && item < items && q0 * 4 + col < pitch) (second || !kHasA ? total_b : total_a)[q0 * 4 + col] = t;
        }
        barrier();
      }
      for (uint32_t c = threadIdx.x; c < w.chans; c += threads) {
        float ta = 0.f, tb = 0.f;
        for (uint32_t r = 0; r < w.fold; ++r) {
          if constexpr (kHasA) ta += total_a[r * w.chans + c];
          if constexpr (kHasB) tb += total_b[r * w.chans + c];
        }
        finishChan<T>(fin, c, ta, tb);
      }
      return;
    }
  }
  // any channel count: [slabs * fold][chans], a channel per thread
  const uint32_t parts = gridDim.y * w.fold;
  for (uint32_t c = threadIdx.x; c < w.chans; c += kThreads) {
    float sa = 0.f, sb = 0.f;
#pragma unroll 8
    for (uint32_t k = 0; k < parts; ++k) {
      if constexpr (kHasA) sa += __ldcg(partial_a + size_t(k) * w.chans + c);
      if constexpr (kHasB) sb += __ldcg(partial_b + size_t(k) * w.chans + c);
    }
    finishChan<T>(fin, c, sa, sb);
  }
}

// Few rows, in two launches: a block covers 64 channels and a slab of rows (a thread two
// neighbouring channels of every eighth row), then a warp per channel adds the slabs,
// lane l slabs l, l + 32, ... in order, the lanes by a fixed tree.  kPairs: the two
// channels are one load (an even count, aligned to it).
constexpr int kColChans = 64, kColRows = 8, kColSlabs = 128;
template <typename T, int kMode, bool kPairs>
__global__ void __launch_bounds__(32 * kColRows)
chanColumnsKernel(const T *__restrict__ x, const T *__restrict__ y, const T *__restrict__ centre, size_t rows,
                  uint32_t chans, float *__restrict__ partial_a, float *__restrict__ partial_b) {
  using Pair = typename ChanPair<T>::Type;
  constexpr bool kHasY = kMode == kSumXYAndY;
  __shared__ float sums[2][kColRows][kColChans];
  pdl_launch_dependents();
  pdl_wait();  // inputs may come from the previous kernel in the stream
  const uint32_t c0 = blockIdx.x * kColChans + 2 * threadIdx.x;
  float a[2] = {0.f, 0.f}, b[2] = {0.f, 0.f}, m[2] = {0.f, 0.f};
  if constexpr (kMode == kSumCentredXX)
    for (int j = 0; j < 2; ++j)
      if (c0 + j < chans) m[j] = toFloat(centre[c0 + j]);
  auto load = [&](const T *t, size_t r, float (&f)[2]) {
    if constexpr (kPairs) {
      ChanPair<T>::unpack(*reinterpret_cast<const Pair *>(t + r * chans + c0), f);
    } else {
      f[0] = toFloat(t[r * chans + c0]);
      f[1] = c0 + 1 < chans ? toFloat(t[r * chans + c0 + 1]) : 0.f;
    }
  };
  if (c0 < chans) {
#pragma unroll 8
    for (size_t r = blockIdx.y * size_t(kColRows) + threadIdx.y; r < rows; r += size_t(gridDim.y) * kColRows) {
      float xv[2], yv[2] = {0.f, 0.f};
      load(x, r, xv);
      if constexpr (kHasY) load(y, r, yv);
#pragma unroll
      for (int j = 0; j < 2; ++j) addElement<T, kMode>(a[j], b[j], xv[j], yv[j], m[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    sums[0][threadIdx.y][2 * threadIdx.x + j] = a[j];
    sums[1][threadIdx.y][2 * threadIdx.x + j] = b[j];
  }
  __syncthreads();
  const uint32_t t = threadIdx.y * 32 + threadIdx.x, which = t / kColChans, col = t % kColChans;
  const uint32_t c = blockIdx.x * kColChans + col;
  if (which < 2 && c < chans) {
    float total = sums[which][0][col];
#pragma unroll
    for (int l = 1; l < kColRows; ++l) total += sums[which][l][col];
    (which ? partial_b : partial_a)[size_t(blockIdx.y) * chans + c] = total;
  }
}
template <typename T>
__global__ void __launch_bounds__(256)
chanFinishKernel(const float *__restrict__ partial_a, const float *__restrict__ partial_b, uint32_t slabs,
                 uint32_t chans, const ChanFinish fin) {
  pdl_launch_dependents();
  pdl_wait();  // the slabs' sums come from the previous kernel in the stream
  const uint32_t c = blockIdx.x * 8 + threadIdx.y;
  if (c >= chans) return;  // (whole warps leave together)
  float a = 0.f, b = 0.f;
  for (uint32_t k = threadIdx.x; k < slabs; k += 32) {
    a += partial_a[size_t(k) * chans + c];
    b += partial_b[size_t(k) * chans + c];
  }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, d);
    b += __shfl_xor_sync(0xffffffffu, b, d);
  }
  if (threadIdx.x == 0) finishChan<T>(fin, c, a, b);
}

// A power of two of values, neighbours first: the large sums are few.
template <int N>
__device__ __forceinline__ float pairwise(float (&v)[N]) {
#pragma unroll
  for (int d = 1; d < N; d *= 2)
#pragma unroll
    for (int k = 0; k + d < N; k += 2 * d) v[k] += v[k + d];
  return v[0];
}

// The same in one launch, where rows are whole vectors: the blocks of a cluster of up to eight have the
// slabs, and the first reads the others' sums from their shared memory, in their order.  Bound by latency: the
// launch, one or two batches of loads, the two meetings of the cluster.
constexpr int kClusterThreads = 512, kClusterBlocks = 8;
template <typename T, int kMode, int V>
__global__ void __launch_bounds__(kClusterThreads, 1)
chanClusterKernel(const T *__restrict__ x, const T *__restrict__ y, const T *__restrict__ centre, uint32_t rows,
                  uint32_t chans, const ChanFinish fin) {
  using Vec = ChanVec<T, V>;
  using Raw = typename Vec::Raw;
  constexpr bool kHasA = kMode != kSumCentredXX, kHasB = kMode != kSumX, kHasY = kMode == kSumXYAndY;
  constexpr uint32_t kLanes = kColChans / V, kRowLanes = kClusterThreads / kLanes, kWarps = kClusterThreads / 32;
  constexpr int kUnroll = kHasY ? 4 : 8;
  __shared__ float red[2][kWarps][kColChans + 1];
  __shared__ float sums[2][kColChans];
  pdl_launch_dependents();
  const uint32_t vx = threadIdx.x % kLanes, ry = threadIdx.x / kLanes, warp = threadIdx.x / 32;
  const uint32_t c0 = blockIdx.x * kColChans + vx * V;
  const bool mine = c0 < chans;
  float a[V], b[V], m[V];
#pragma unroll
  for (int j = 0; j < V; ++j) a[j] = b[j] = m[j] = 0.f;
  pdl_wait();  // inputs may come from the previous kernel in the stream
  if (mine) {
    if constexpr (kMode == kSumCentredXX)
#pragma unroll
      for (int j = 0; j < V; ++j) m[j] = toFloat(centre[c0 + j]);
    const uint32_t step = gridDim.y * kRowLanes;
    for (uint32_t r = blockIdx.y * kRowLanes + ry; r < rows; r += kUnroll * step) {
      Raw rx[kUnroll];
      [[maybe_unused]] Raw rv[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u)
        if (r + u * step < rows) {
          rx[u] = *reinterpret_cast<const Raw *>(x + size_t(r + u * step) * chans + c0);
          if constexpr (kHasY) rv[u] = *reinterpret_cast<const Raw *>(y + size_t(r + u * step) * chans + c0);
        }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u)
        if (r + u * step < rows) {
          float xv[V], yv[V];
          Vec::unpack(rx[u], xv);
          if constexpr (kHasY) Vec::unpack(rv[u], yv);
#pragma unroll
          for (int j = 0; j < V; ++j) addElement<T, kMode>(a[j], b[j], xv[j], kHasY ? yv[j] : 0.f, m[j]);
        }
    }
  }
  uint32_t first = 0, held = V;  // the columns of the vector this thread ends up with
  bool writes = true;
  foldWarp<V, kHasA, kHasB, 16>(a, b, kLanes, first, held, writes);
  if (writes)
#pragma unroll
    for (int j = 0; j < V; ++j)
      if (j < held) {
        if constexpr (kHasA) red[0][warp][vx * V + first + j] = a[j];
        if constexpr (kHasB) red[1][warp][vx * V + first + j] = b[j];
      }
  __syncthreads();
  const uint32_t which = threadIdx.x / kColChans, col = threadIdx.x % kColChans, c = blockIdx.x * kColChans + col;
  if (which < 2 && (which == 0 ? kHasA : kHasB)) {
    float part[kWarps];
#pragma unroll
    for (uint32_t k = 0; k < kWarps; ++k) part[k] = red[which][k][col];
    sums[which][col] = pairwise(part);
  }
  if (gridDim.y > 1)
    cluster_sync_all();
  else
    __syncthreads();
  if (blockIdx.y == 0 && which == 0 && c < chans) {
    float ta[kClusterBlocks], tb[kClusterBlocks];
#pragma unroll
    for (uint32_t k = 0; k < kClusterBlocks; ++k) {
      auto read = [&](const float *p) {
        float v;
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(map_to_cta(smem_u32(p), k)) : "memory");
        return v;
      };
      ta[k] = kHasA && k < gridDim.y ? read(&sums[0][col]) : 0.f;
      tb[k] = kHasB && k < gridDim.y ? read(&sums[1][col]) : 0.f;
    }
    finishChan<T>(fin, c, pairwise(ta), pairwise(tb));
  }
  if (gridDim.y > 1) cluster_sync_all();  // (no block leaves before its sums have been read)
}
template <typename T, int kMode, int V>
int launchChanCluster(plb_context *ctx, uint64_t rows, uint32_t chans, const T *x, const T *y, const T *centre, const ChanFinish &fin) {
  constexpr uint32_t kRowLanes = kClusterThreads / (kColChans / V);
  // four rows a thread and more, as long as there are blocks for them
  uint32_t blocks = 1;
  while (blocks < kClusterBlocks && uint64_t(blocks) * kRowLanes * 4 < rows) blocks *= 2;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = blocks;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((chans + kColChans - 1) / kColChans, blocks);
  cfg.blockDim = dim3(kClusterThreads);
  cfg.stream = ctx->stream;
  cfg.attrs = attr;
  cfg.numAttrs = (ctx->plan_flags & PLB_PLAN_NO_PDL) ? 1 : 2;
  PLB_CUDA(cudaLaunchKernelEx(&cfg, chanClusterKernel<T, kMode, V>, x, y, centre, uint32_t(rows), chans, fin));
  PLB_CUDA(cudaGetLastError());
  ctx->launches++;
  return PLB_OK;
}

template <typename T, int kMode>
int launchChanColumns(plb_context *ctx, uint64_t rows, uint32_t chans, const T *x, const T *y, const T *centre,
                      const ChanFinish &fin) {
  const uint32_t cols = (chans + kColChans - 1) / kColChans;
  // four rows per thread and more, four slabs per lane of the second kernel at most
  const uint64_t want = std::max<uint64_t>(1, (rows + 4 * kColRows - 1) / (4 * kColRows));
  const uint32_t slabs = uint32_t(std::min<uint64_t>(want, kColSlabs));
  void *ws = nullptr;
  if (int rc = scratch(ctx, kSlotChannelSums, size_t(2) * slabs * chans * sizeof(float), &ws)) return rc;
  float *pa = static_cast<float *>(ws), *pb = pa + size_t(slabs) * chans;
  const uintptr_t at = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y);
  const bool pairs = chans % 2 == 0 && at % (2 * sizeof(T)) == 0;
  if (int rc = launchPdl(ctx, pairs ? chanColumnsKernel<T, kMode, true> : chanColumnsKernel<T, kMode, false>,
                         dim3(cols, slabs), dim3(32, kColRows), 0, x, y, centre, size_t(rows), chans, pa, pb))
    return rc;
  return launchPdl(ctx, chanFinishKernel<T>, dim3((chans + 7) / 8), dim3(32, 8), 0, (const float *)pa, (const float *)pb,
                   slabs, chans, fin);
}

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <typename T, int kMode, int V, int kThreads>
int launchChanSums(plb_context *ctx, uint64_t rows, uint32_t chans, uint64_t most_slabs, const T *x, const T *y,
                   const T *centre, ChanFinish fin) {
  constexpr size_t kMost = 160 * 1024;
  // four loads at once take a thread hardly longer than one, and a quarter of the
  // slabs leave the last block fewer rows (4 images of 14x14, 256 channels: 6.3 -> 5.5 us)
  constexpr uint32_t kRowsEach = 4;
  dim3 grid;
  const ChanWalk w = chanWalk(ctx, rows, chans, V, kThreads, 1, kRowsEach, most_slabs, &grid);
  const size_t pitch = size_t(w.vecs) * V, cols = size_t(V) << w.vec_lanes_log2;
  void *ws = nullptr;
  if (int rc = scratch(ctx, kSlotChannelSums, size_t(2) * w.slabs * pitch * sizeof(float) + 16, &ws)) return rc;
  float *pa = static_cast<float *>(ws), *pb = pa + (size_t(w.slabs) * pitch + 3) / 4 * 4;
  const size_t finish = 8 * (kThreads + kThreads / 2) * sizeof(float) + 2 * pitch * sizeof(float);
  fin.totals_fit = V > 1 && finish <= kMost ? 1 : 0;
  const size_t smem = std::max(2 * (kThreads / 32) * (cols + 1) * sizeof(float), fin.totals_fit ? finish : size_t(0));
  static std::atomic<bool> configured[64] = {};  // (contexts may live on several threads)
  std::atomic<bool> &done = configured[ctx->device & 63];
  if (!done) {
    PLB_CUDA(cudaFuncSetAttribute(chanSumsKernel<T, kMode, V, kThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(kMost)));
    done = true;
  }
  return launchPdl(ctx, chanSumsKernel<T, kMode, V, kThreads>, grid, dim3(kThreads), smem, x, y, centre, w, pa, pb,
                   ctx->d_ticket, fin);
}

// The forms that leave partial sums in scratch memory.  `vec`: in loads of 16 bytes.
template <typename T, int kMode>
int chanSumsScratch(plb_context *ctx, const T *x, const T *y, const T *centre, uint64_t rows, uint32_t chans, bool vec,
                    const ChanFinish &fin) {
  constexpr int kVec = 16 / sizeof(T);
  // Slabs: one per SM, but each slab's row of sums is work for the last block.  Up
  // to 128 columns that is nothing; wider rows take fewer slabs, down to one per four
  // SMs, unless a slab has 256 KB to read and more (25088 x 256 halves: 9.4 us with 148
  // slabs, 8.9 with 74).
  const uint64_t bytes = rows * chans * sizeof(T);
  const uint64_t most_slabs =
      std::max<uint64_t>({uint64_t(ctx->sm_count) / 4, uint64_t(ctx->sm_count) * 128 / std::max(chans, 1u), bytes / (256 * 1024)});
  // The others up to 8192, and more that are no whole vectors: two short launches over narrow columns,
  // where a block's wide row of sums would be most of the work and the last block's finish most of
  // the time (324 x 253 halves 7.8 -> 3.6 us, 1058 x 351 floats 7.7 -> 4.2, 8281 x 64 halves 5.7 -> 5.5; 16641
  // x 64 5.7 against 6.9; 16641 x 255 halves 10.8 -> 7.5).
  if (rows <= (vec && chans % kVec == 0 ? 8192u : 24576u) && bytes <= (uint64_t(16) << 20))
    return launchChanColumns<T, kMode>(ctx, rows, chans, x, y, centre, fin);
  if (!vec) return launchChanSums<T, kMode, 1, 512>(ctx, rows, chans, most_slabs, x, y, centre, fin);
  // Twice the warps keep the loads of a long slab going while a part of them adds (64
  // images of 56x56, 256 channels, 103 MB: 20.4 us, with 512 threads 22.0); elsewhere they only
  // add to what every warp executes once (32 images of 56x56, 64 channels: 7.1 us, 6.8).
  if (bytes >= (uint64_t(64) << 20))
    return launchChanSums<T, kMode, kVec, 1024>(ctx, rows, chans, most_slabs, x, y, centre, fin);
  return launchChanSums<T, kMode, kVec, 512>(ctx, rows, chans, most_slabs, x, y, centre, fin);
}

template <typename T, int kMode>
int chanSums(plb_context *ctx, const T *x, const T *y, const T *centre, uint64_t rows, uint32_t chans,
             const ChanFinish &fin) {
  constexpr int kVec = 16 / sizeof(T);
  // (a super-row's columns are counted in 32 bits)
  const bool vec = aligned16(x) && (y == nullptr || aligned16(y)) && uint64_t(chans) * kVec <= 0xffffffffull;
  const uint64_t bytes = rows * chans * sizeof(T);
  // Few rows: one launch of clusters over narrow columns (halves, with the two launches below before:
  // 64 x 64 3.2 -> 2.2 us, 784 x 1024 5.3 -> 3.4, 4096 x 64 4.5 -> 3.4, 4096 x 256 7.0 -> 3.6, 8192 x 512 7.9 -> 4.6;
  // floats alike).  Eight blocks have all the rows of 64 columns.  Up to 64 columns the other forms
  // are quicker from 8192 rows on (two sums 5.0 against 5.3), up to 16 from 4096 (5000 x 8, two sums 3.6
  // against 4.1), up to 128 from 12544 (6.1 against 7.1), up to 768, where slabs leave wide rows of sums
  // (8192 x 768 halves 8.5 against 4.7), from 16384 (floats 10.0 against 11.1).  Wider
  // rows have more clusters than the SMs hold at once, which is worth it where single blocks have
  // a column (256 x 16384 halves 4.5, the two launches 8.2) or sums of moderate size come in few waves (1024 x 2048
  // halves 3.4, 6.8; 4096 x 1024 6.2, slabs 7.8), not beyond (1024 x 16384 floats 45 against 19, 2048 x 4096
  // halves 14.4 against 11.2, 4096 x 8192 28 against 22).
  const bool whole = vec && chans % kVec == 0;
  const bool clusters = chans <= 768 ? rows <= (chans <= 16 ? 4095u : chans <= 64 ? 6144u : chans <= 128 ? 8192u : 12544u)
                                     : rows <= 4 * (kClusterThreads / (kColChans / kVec)) || bytes < (uint64_t(6) << 20) ||
                                           (rows > 2560 && bytes <= (uint64_t(24) << 20));
  if (whole && clusters) return launchChanCluster<T, kMode, kVec>(ctx, rows, chans, x, y, centre, fin);
  ctx->scratch_refused = false;
  const int rc = chanSumsScratch<T, kMode>(ctx, x, y, centre, rows, chans, vec, fin);
  // (in a stream capture scratch cannot grow: few rows do without it, however long that takes)
  return rc != PLB_OK && ctx->scratch_refused && whole && rows <= 12544
             ? launchChanCluster<T, kMode, kVec>(ctx, rows, chans, x, y, centre, fin) : rc;
}

// ---- maps ------------------------------------------------------------------------

enum ChanMap : int {
  kWhiten = 0,      // (x - p[c]) * q[c]
  kScaleShift = 1,  // x * p[c] + q[c]
  kScale = 2,       // x * p[c]
  kStatsGrad = 3,   // (y + x * p[c] + q[c]) * r[c]     x = whitened, y = gradient
  kNormalise = 4,   // w = (x - p[c]) * q[c] rounded to T (stored in out2 if given), w * r[c] + s[c]
  kAddChan = 5,     // x + p[c]
};

template <typename T>
struct ChanMapArgs {
  const T *x, *y;
  const T *p, *q, *r, *s;    // per channel
  const float *pf, *qf;      // the same in fp32 (instead of p, q)
  T *out, *out2;             // out may be x
  int whole;                 // (set by chanMap) a vector's operands are whole vectors of p, q, r, s too
};

constexpr int kChanMapThreads = 256;

// kRows: super-rows a thread has in flight.
template <typename T, int kMode, int V, int kRows>
__global__ void __launch_bounds__(kChanMapThreads)
chanMapKernel(const ChanMapArgs<T> g, const ChanWalk w) {
  using Vec = ChanVec<T, V>;
  using Raw = typename Vec::Raw;
  constexpr bool kHasY = kMode == kStatsGrad;
  constexpr int kUnroll = kRows;
  pdl_launch_dependents();
  const uint32_t lanes = 1u << w.vec_lanes_log2, row_lanes = kChanMapThreads >> w.vec_lanes_log2;
  const uint32_t vx = threadIdx.x & (lanes - 1), ry = threadIdx.x >> w.vec_lanes_log2;
  const uint32_t vec = blockIdx.x * lanes + vx;
  pdl_wait();  // inputs may come from the previous kernel in the stream
  if (vec >= w.vecs) return;
  const size_t pitch = size_t(w.vecs) * V, step = size_t(gridDim.y) * row_lanes;
  size_t row0 = size_t(blockIdx.y) * row_lanes + ry;
  Raw rx[kUnroll];
  [[maybe_unused]] Raw rv[kUnroll];
  auto fetch = [&]() {
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const size_t row = row0 + u * step;
      if (row < w.full) {
        rx[u] = *reinterpret_cast<const Raw *>(g.x + row * pitch + size_t(vec) * V);
        if constexpr (kHasY) rv[u] = *reinterpret_cast<const Raw *>(g.y + row * pitch + size_t(vec) * V);
      }
    }
  };
  fetch();  // (ahead of the operands, so that both are in flight)
  float p[V], q[V], r[V], s[V];
  constexpr bool kHasQ = kMode != kScale && kMode != kAddChan, kHasR = kMode == kStatsGrad || kMode == kNormalise;
  if (g.whole) {
    auto load = [&](const T *src, float (&f)[V]) { Vec::unpack(*reinterpret_cast<const Raw *>(src + size_t(vec) * V), f); };
    if (kMode == kStatsGrad && g.pf) {
#pragma unroll
      for (int j = 0; j < V; ++j) {
        p[j] = g.pf[size_t(vec) * V + j];
        q[j] = g.qf[size_t(vec) * V + j];
      }
    } else {
      load(g.p, p);
      if constexpr (kHasQ) load(g.q, q);
    }
    if constexpr (kHasR) load(g.r, r);
    if constexpr (kMode == kNormalise) load(g.s, s);
  } else {
    uint32_t c = uint32_t(size_t(vec) * V % w.chans);
#pragma unroll
    for (int j = 0; j < V; ++j) {
      p[j] = g.pf ? g.pf[c] : toFloat(g.p[c]);
      if constexpr (kHasQ) q[j] = g.qf ? g.qf[c] : toFloat(g.q[c]);
      if constexpr (kHasR) r[j] = toFloat(g.r[c]);
      if constexpr (kMode == kNormalise) s[j] = toFloat(g.s[c]);
      if (++c == w.chans) c = 0;
    }
  }
  auto map = [&](float x, float y, int j, float &white) -> float {
    if constexpr (kMode == kWhiten) {
      return (x - p[j]) * q[j];
    } else if constexpr (kMode == kScaleShift) {
      return x * p[j] + q[j];
    } else if constexpr (kMode == kScale) {
      return x * p[j];
    } else if constexpr (kMode == kStatsGrad) {
      return (y + x * p[j] + q[j]) * r[j];
    } else if constexpr (kMode == kNormalise) {
      // rounded before it is scaled: the bits of kWhiten followed by kScaleShift
      white = toFloat(fromFloat<T>((x - p[j]) * q[j]));
      return white * r[j] + s[j];
    } else {
      return x + p[j];
    }
  };
  for (; row0 < w.full; row0 += kUnroll * step, fetch()) {
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const size_t row = row0 + u * step;
      if (row < w.full) {
        float xv[V], yv[V], o[V], white[V];
        Vec::unpack(rx[u], xv);
        if constexpr (kHasY) Vec::unpack(rv[u], yv);
#pragma unroll
        for (int j = 0; j < V; ++j) o[j] = map(xv[j], kHasY ? yv[j] : 0.f, j, white[j]);
        if constexpr (kMode == kNormalise)
          if (g.out2) *reinterpret_cast<Raw *>(g.out2 + row * pitch + size_t(vec) * V) = Vec::pack(white);
        *reinterpret_cast<Raw *>(g.out + row * pitch + size_t(vec) * V) = Vec::pack(o);
      }
    }
  }
  // the rows that do not fill a super-row
  if (w.fold > 1 && blockIdx.y == 0 && ry == 0) {
    const size_t base = w.full * pitch + size_t(vec) * V;
#pragma unroll
    for (int j = 0; j < V; ++j)
      if (base + j < w.total) {
        float white = 0.f;
        const float o = map(toFloat(g.x[base + j]), kHasY ? toFloat(g.y[base + j]) : 0.f, j, white);
        if constexpr (kMode == kNormalise)
          if (g.out2) g.out2[base + j] = fromFloat<T>(white);
        g.out[base + j] = fromFloat<T>(o);
      }
  }
}

template <typename T, int kMode>
int chanMap(plb_context *ctx, ChanMapArgs<T> g, uint64_t rows, uint32_t chans) {
  if (rows == 0 || chans == 0) return PLB_OK;
  constexpr uint32_t kVec = 16 / sizeof(T);
  const bool vec = uint64_t(chans) * kVec <= 0xffffffffull && aligned16(g.x) && aligned16(g.out) && (g.y == nullptr || aligned16(g.y)) &&
                   (g.out2 == nullptr || aligned16(g.out2));
  // Blocks that all are resident and walk, but a large tensor takes as many as fit: what
  // counts there is loads in flight (whitening and scaling 100352 x 1024 halves: 57.1 us
  // with 4 blocks per SM, 52.2 with 16; 3136 x 1024: 5.3 with 4, 7.7 with 16).
  const uint32_t per_sm = rows * chans * sizeof(T) >= (uint64_t(32) << 20) ? 16 : 4;
  dim3 grid;
  const ChanWalk w = chanWalk(ctx, rows, chans, vec ? kVec : 1, kChanMapThreads, per_sm, 1, 0, &grid);
  g.whole = vec && w.fold == 1 && aligned16(g.p) && aligned16(g.q) && aligned16(g.r) && aligned16(g.s);
  // Where a thread has one super-row the code for several only has to be fetched
  // (whitening and scaling 4225 x 256 halves: 3.8 us).
  constexpr int kMany = kMode == kStatsGrad ? 2 : 4;
  const bool one = w.full <= uint64_t(grid.y) * (kChanMapThreads >> w.vec_lanes_log2);
  if (!vec) return launchPdl(ctx, chanMapKernel<T, kMode, 1, kMany>, grid, dim3(kChanMapThreads), 0, g, w);
  return launchPdl(ctx, one ? chanMapKernel<T, kMode, int(kVec), 1> : chanMapKernel<T, kMode, int(kVec), kMany>, grid,
                   dim3(kChanMapThreads), 0, g, w);
}

}  // namespace plb
