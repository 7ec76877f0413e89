// Forward convolution of few input channels (a stem: 7x7, stride 2, 3 channels) from the
// image as it is.
//
// Rearranged in global memory (small_channel.cu), such a layer writes and reads its input
// once more, in a launch of its own, and every filter row fetches 128 bytes of overlapping
// windows for each output pixel.  Here a block loads the rows of a strip of output pixels
// once, as superpixels of 16 bytes: the stride's pixels of a row side by side (3 channels,
// stride 2: 6 halves and two zeros).  Output pixel i and horizontal tap t of a filter row
// then meet at superpixel i + t, so consecutive output pixels' operand rows lie 16 bytes
// apart.  That is the unswizzled K-major layout of tcgen05 (core matrices of eight 16-byte
// rows), whose core-matrix stride along K is 16 bytes here: they overlap, nothing is copied
// per tap, and the instruction is as fast as from 128-byte rows (48 cycles of 128 x 64 x 16
// either way).  Filter rows of one parity of the stride share a plane of superpixel rows, P
// apart; a tile is 128 consecutive positions of the strip, the last T-1 of every row not
// stored.
//
// Roles: 7 warps load strips (two in flight), one issues the instructions, two groups
// of 4 warps store alternate tiles.  Loads, results and operands share the SM's path to
// shared memory and L1; a tile of 14 instructions (7x7) takes 1350 cycles of the 670 that the
// instructions alone would, one of 6 (3x3) is bound by its results.  Measured against the rearranged
// form: 3x3, 1 -> 96 on 147 images of 118 x 118 122 -> 96 us, 3x3/2, 4 -> 64 on 11 of 102 x 192 9.1 ->
// 5.4, 7x7/2, 3 -> 64 on 256 of 224 x 224 162 -> 147 to 158 by the device's clock (medians of six).  (Whole lines of results, stored from 16
// x 256-bit reads of tensor memory, two issuers or four accumulators: no gain.)
#include <algorithm>
#include <atomic>
#include <cmath>

#include "sm100_prims.cuh"
#include "stem.h"

namespace plb {
namespace {

constexpr int kStemThreads = 512, kStemMmaWarp = 8, kStemLoaders = 224;

struct StemArgs {
  const uint16_t *x, *w;
  const float *bias;
  __half *out;
  int *status;
  S2dShape g;
  int co, co_pad;         // co_pad: columns of an accumulator
  int taps;               // superpixels of a filter row, even
  int pad_w, shift;       // padding rounded up to the stride; by how much
  int tile_w, rows, pitch;  // a strip: output columns and rows, superpixels of a row
  int parts, h_blocks, units;
  uint32_t plane_bytes, strip_bytes, weight_bytes;
  uint32_t idesc, tmem_cols;
  FastDiv fd_pitch, fd_parts, fd_h_blocks, fd_co, fd_taps;
};

// A sum over the pixels that exist.
template <bool kBf16>
__device__ __noinline__ float stemSum(const StemArgs &a, int n, int oh, int ow, int co) {
  const S2dShape &g = a.g;
  auto value = [](uint16_t v) {
    return kBf16 ? __uint_as_float(uint32_t(v) << 16) : __half2float(__ushort_as_half(v));
  };
  float sum = 0.f;
#pragma unroll 1
  for (int r = 0; r < g.KH; ++r)
#pragma unroll 1
    for (int s = 0; s < g.KW; ++s) {
      const int ih = oh * g.s + r - g.padH, iw = ow * g.s + s - g.padW;
      if (ih < 0 || iw < 0 || ih >= g.H || iw >= g.W) continue;
#pragma unroll 1
      for (int c = 0; c < g.C; ++c)
        sum += value(a.x[(((long long)n * g.H + ih) * g.W + iw) * g.C + c]) * value(a.w[((r * g.KW + s) * a.co + co) * g.C + c]);
    }
  return sum;
}

// K-major operand without swizzle: core matrices of eight 16-byte rows, `lbo` apart along K
// and `sbo` along M or N.
__device__ __forceinline__ uint64_t plainDesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return uint64_t((addr & 0x3ffffu) >> 4) | uint64_t(lbo >> 4) << 16 | uint64_t(sbo >> 4) << 32 | uint64_t(1) << 46;
}

// kWords: 32-bit words of a superpixel, 0 where its elements are loaded one by one.
template <int kWords, bool kBf16>
__global__ void __launch_bounds__(kStemThreads, 1)
stemKernel(const __grid_constant__ StemArgs a) {
  extern __shared__ __align__(128) uint8_t stem_smem[];
  __shared__ __align__(8) uint64_t bars[9];  // strip full, strip free, accumulator full, accumulator free, drain
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  __shared__ __align__(16) float bias[256];
  const S2dShape &g = a.g;
  // (the warp is the same in all lanes, as the compiler sees it)
  const int tid = int(threadIdx.x), warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t weights = smem_u32(stem_smem), strips = weights + a.weight_bytes;
  volatile int *abort_flag = &abort_word;
  auto stripFull = [&](int i) { return smem_u32(bars + i); };
  auto stripFree = [&](int i) { return smem_u32(bars + 2 + i); };
  auto accFull = [&](int i) { return smem_u32(bars + 4 + i); };
  auto accFree = [&](int i) { return smem_u32(bars + 6 + i); };
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(stripFull(i), kStemLoaders);
      mbar_init(stripFree(i), 1);
      mbar_init(accFull(i), 1);
      mbar_init(accFree(i), 128);
    }
    mbar_init(smem_u32(bars + 8), 1);
    abort_word = 0;
    mbar_fence_init();
  }
  if (warp == kStemMmaWarp) {
    tmem_alloc(smem_u32(&tmem_slot), a.tmem_cols);
    tmem_relinquish();
  }
  pdl_wait();  // (all threads: they read the operands, or write over what the last kernel read)
  // weights: [filter row][superpixel][output channel] of 16 bytes
  const int weight_units = g.KH * a.taps * a.co, next_column = (a.co - 1) * g.C;
  for (int i = tid; i < weight_units; i += kStemThreads) {
    const int rt = int(fast_div(uint32_t(i), a.fd_co)), co = i - rt * a.co, r = int(fast_div(uint32_t(rt), a.fd_taps));
    const int s = (rt - r * a.taps) * g.s - a.shift;  // the first pixel's filter column; C elements on, the next one's
    const uint16_t *const p = a.w + ((r * g.KW + s) * a.co + co) * g.C;
    const int first = s >= 0 && s < g.KW ? g.C : 0, last = g.s == 2 && s + 1 >= 0 && s + 1 < g.KW ? 2 * g.C : g.C;
    uint16_t e[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) e[k] = k < g.C ? (k < first ? p[k] : uint16_t(0)) : k < last ? p[k + next_column] : uint16_t(0);
    st_shared_v4(weights + uint32_t(i) * 16, e[0] | uint32_t(e[1]) << 16, e[2] | uint32_t(e[3]) << 16, e[4] | uint32_t(e[5]) << 16,
                 e[6] | uint32_t(e[7]) << 16);
  }
  if (tid < a.co_pad) bias[tid] = a.bias && tid < a.co ? a.bias[tid] : 0.f;
  fence_proxy_async_smem();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  pdl_launch_dependents();  // (tensor memory is allocated: the next kernel cannot take it first)
  const uint32_t tmem = __shfl_sync(0xffffffffu, *static_cast<volatile uint32_t *>(&tmem_slot), 0);
  // strip u: image, first output row and column, and its tiles
  auto stripOf = [&](int u, int &n, int &oh0, int &ow0, int &rows, int &cols) {
    const int v = int(fast_div(uint32_t(u), a.fd_parts));
    n = int(fast_div(uint32_t(v), a.fd_h_blocks));
    oh0 = (v - n * a.h_blocks) * a.rows;
    ow0 = (u - v * a.parts) * a.tile_w;
    rows = min(a.rows, g.OH - oh0);
    cols = min(a.tile_w, g.OW - ow0);
    return ((rows - 1) * a.pitch + cols + 127) >> 7;
  };
  bool ok = true;
  auto failed = [&](int code) {
    atomicCAS(a.status, kStatusOk, code);
    ok = false;
  };

  if (warp > kStemMmaWarp) {
    // ---- loaders
    const int me = tid - (kStemMmaWarp + 1) * 32;
    for (int u = int(blockIdx.x), k = 0; u < a.units; u += int(gridDim.x), ++k) {
      int n, oh0, ow0, rows, cols;
      stripOf(u, n, oh0, ow0, rows, cols);
      const int buf = k & 1;
      if (!mbar_wait(stripFree(buf), uint32_t(k >> 1 & 1) ^ 1u, abort_flag)) {
        failed(kStatusProducerTimeout);
        break;
      }
      const uint32_t strip = strips + uint32_t(buf) * a.strip_bytes;
      const int total = ((rows - 1) * g.s + g.KH) * a.pitch, ih0 = oh0 * g.s - g.padH, px0 = ow0 * g.s - a.pad_w;
      const uint16_t *img = a.x + (long long)n * g.H * g.W * g.C;
#pragma unroll 1
      for (int i0 = me; i0 < total; i0 += 4 * kStemLoaders) {
        uint32_t v[4][4], dst[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int i = i0 + j * kStemLoaders;
          const int y = int(fast_div(uint32_t(i), a.fd_pitch)), at = i - y * a.pitch;
          const int q = g.s == 2 ? y >> 1 : y, plane = y - q * g.s;
          const int ih = ih0 + y, px = px0 + at * g.s;
          // (px is a multiple of the stride: all of a superpixel lies left of the image, or none)
          const int there = i < total && uint32_t(ih) < uint32_t(g.H) && px >= 0 ? min(g.W - px, g.s) * g.C : 0;
          dst[j] = strip + uint32_t(plane) * a.plane_bytes + uint32_t(q * a.pitch + at) * 16;
          const uint16_t *p = img + (ih * g.W + px) * g.C;
          if constexpr (kWords > 0) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              v[j][e] = e < kWords && 2 * e < there ? reinterpret_cast<const uint32_t *>(p)[e] : 0u;
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const uint32_t lo = 2 * e < there ? p[2 * e] : 0u, hi = 2 * e + 1 < there ? p[2 * e + 1] : 0u;
              v[j][e] = lo | hi << 16;
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (i0 + j * kStemLoaders < total) st_shared_v4(dst[j], v[j][0], v[j][1], v[j][2], v[j][3]);
      }
      fence_proxy_async_smem();
      mbar_arrive(stripFull(buf));
    }
  } else if (warp == kStemMmaWarp) {
    // ---- instructions: all lanes walk, for each tile one issues, so that the operands come from
    // uniform registers (with one thread in the whole role 200 sampled layers took 1.04 of their time,
    // 7x7/2, 3 -> 64, 256 images of 224 x 224 153 us, now 147)
    auto wait = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag)); };
    const uint32_t b_step = uint32_t(a.co) * 2;
    const uint64_t b_first = plainDesc(weights, uint32_t(a.co) * 16, 128);
    const uint32_t down = uint32_t(a.pitch), plane1 = g.s == 2 ? a.plane_bytes >> 4 : down;
    const uint32_t both = g.s == 2 ? down : 2 * down;
    int c = 0, k = 0;
    for (int u = int(blockIdx.x); ok && u < a.units; u += int(gridDim.x), ++k) {
      int n, oh0, ow0, rows, cols;
      const int tiles = stripOf(u, n, oh0, ow0, rows, cols), buf = k & 1;
      if (!wait(stripFull(buf), uint32_t(k >> 1 & 1))) {
        failed(kStatusMmaTimeout);
        break;
      }
      tc_fence_after_sync();
      const uint32_t strip = strips + uint32_t(buf) * a.strip_bytes;
      for (int t = 0; t < tiles; ++t, ++c) {
        const int acc = c & 1;
        if (!wait(accFree(acc), uint32_t(c >> 1 & 1) ^ 1u)) {
          failed(kStatusMmaTimeout);
          break;
        }
        tc_fence_after_sync();
        const uint32_t d = tmem + uint32_t(acc * a.co_pad);
        uint64_t b = b_first, ad = plainDesc(strip + uint32_t(t * 128) * 16, 16, 128);
        if (elect_one()) {
          // (unrolled: a loop over single instructions paces them, 7x7 190 us)
          auto filterRow = [&](uint64_t at, bool first) {
            umma_ss<false>(d, at, b, a.idesc, first ? 0u : 1u);
            b += b_step;
#pragma unroll 1
            for (int s = 2; s < a.taps; s += 2) {
              at += 2;
              umma_ss<false>(d, at, b, a.idesc, 1u);
              b += b_step;
            }
          };
          if (a.taps == 4) {
            int r = 0;
            uint32_t acc_on = 0;
#pragma unroll 4
            for (; r + 2 <= g.KH; r += 2, ad += both) {
              umma_ss<false>(d, ad, b, a.idesc, acc_on);
              umma_ss<false>(d, ad + 2, b + b_step, a.idesc, 1u);
              umma_ss<false>(d, ad + plane1, b + 2 * b_step, a.idesc, 1u);
              umma_ss<false>(d, ad + plane1 + 2, b + 3 * b_step, a.idesc, 1u);
              b += 4 * b_step;
              acc_on = 1;
            }
            if (r < g.KH) filterRow(ad, r == 0);
          } else {
            for (int r = 0; r < g.KH; ++r) filterRow(ad + (r >> 1) * both + (r & 1) * plane1, r == 0);
          }
          umma_commit(accFull(acc));
        }
        __syncwarp();
      }
      if (ok && elect_one()) umma_commit(stripFree(buf));
      __syncwarp();
    }
    // the last commits arrive here: not before them may the block end, nor tensor memory go
    // while instructions run (after a failure, too)
    if (elect_one()) umma_commit(smem_u32(bars + 8));
    __syncwarp();
    if (!wait(smem_u32(bars + 8), 0)) failed(kStatusDrainTimeout);
    for (int i = 0; ok && i < 2 && i < k; ++i)
      if (!wait(stripFree((k - 1 - i) & 1), uint32_t((k - 1 - i) >> 1 & 1))) failed(kStatusDrainTimeout);
    __syncwarp();
  } else {
    // ---- results
    const int set = warp >> 2, quarter = warp & 3;
    const uint32_t acc = tmem + uint32_t(set * a.co_pad) + (uint32_t(quarter) << 21);
    int c = 0;
    for (int u = int(blockIdx.x); ok && u < a.units; u += int(gridDim.x)) {
      int n, oh0, ow0, rows, cols;
      const int tiles = stripOf(u, n, oh0, ow0, rows, cols);
      for (int t = 0; t < tiles; ++t, ++c) {
        if ((c & 1) != set) continue;
        const int at = t * 128 + quarter * 32 + lane, row = int(fast_div(uint32_t(at), a.fd_pitch)), col = at - row * a.pitch;
        const bool there = row < rows && col < cols;
        __half *dst = a.out + (((long long)n * g.OH + oh0 + row) * g.OW + ow0 + col) * a.co;
        if (!__all_sync(0xffffffffu, mbar_wait(accFull(set), uint32_t(c >> 1 & 1), abort_flag))) {
          failed(kStatusEpilogueTimeout);
          break;
        }
        tc_fence_after_sync();
        for (int n0 = 0; n0 < a.co; n0 += 32) {
          uint32_t v[32];
          __syncwarp();
          tmem_ld_32x32(acc + uint32_t(n0), v);
          tmem_ld_wait_for(v);
          if (n0 + 32 >= a.co) {
            tc_fence_before_sync();
            mbar_arrive(accFree(set));
          }
          float any = 0.f;
          uint32_t pk[16];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 bb = *reinterpret_cast<const float4 *>(&bias[n0 + 4 * j]);
            const float f0 = __uint_as_float(v[4 * j]), f1 = __uint_as_float(v[4 * j + 1]);
            const float f2 = __uint_as_float(v[4 * j + 2]), f3 = __uint_as_float(v[4 * j + 3]);
            if (n0 + 4 * j < a.co) any += (f0 + f1) * 0.f + (f2 + f3) * 0.f;
            const __half2 lo = __floats2half2_rn(f0 + bb.x, f1 + bb.y), hi = __floats2half2_rn(f2 + bb.z, f3 + bb.w);
            pk[2 * j] = *reinterpret_cast<const uint32_t *>(&lo);
            pk[2 * j + 1] = *reinterpret_cast<const uint32_t *>(&hi);
          }
          if (!there) continue;
          st_global_v8(dst + n0, pk[0], pk[1], pk[2], pk[3], pk[4], pk[5], pk[6], pk[7]);
          if (n0 + 16 < a.co) st_global_v8(dst + n0 + 16, pk[8], pk[9], pk[10], pk[11], pk[12], pk[13], pk[14], pk[15]);
          // (products with padding or with the zero weights beside the filter may have made a
          // NaN of an infinite operand)
          if (any != 0.f) {
#pragma unroll 1
            for (int j = n0; j < min(n0 + 32, a.co); ++j)
              if (!isfinite(__half2float(dst[j])))
                dst[j] = __float2half_rn(stemSum<kBf16>(a, n, oh0 + row, ow0 + col, j) + bias[j]);
          }
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == kStemMmaWarp) tmem_dealloc(tmem, a.tmem_cols);
}

struct StemTiling {
  int taps, pad_w, tile_w, rows, pitch;
  size_t plane_bytes, strip_bytes, weight_bytes;
  float us;
};

// Whether the image is loaded in whole words: rows and superpixels start on them.
bool wholeWords(const S2dShape &g) { return g.s * g.C % 2 == 0 && g.W * g.C % 2 == 0; }

// The strip of the least time, and that time.  Cycles of a strip: its tiles (instructions, or
// results where those take longer) or its loads (a round trip to memory, then so much for each
// superpixel and element), and the lesser of the two once more, as they share the path to shared
// memory.  The weights come first, 512 threads with eight loads each at a time.  Fitted to 571
// sampled layers, median error 4 %, a tenth of them 13 %.  (Without the round trip, strips of
// one tile looked best: 7x7/2, 3 -> 128 channels, 41 images of 86 x 117 18.2 us.)
bool stemTiling(int sms, const S2dShape &g, int co, StemTiling *best) {
  StemTiling t{};
  t.pad_w = (g.padW + g.s - 1) / g.s * g.s;
  t.taps = ((g.KW + t.pad_w - g.padW + g.s - 1) / g.s + 1) / 2 * 2;
  t.weight_bytes = (size_t(g.KH) * t.taps * co * 16 + 127) / 128 * 128;
  const double tile = std::max(g.KH * t.taps / 2 * (58.5 + 0.214 * co), 383 + 12.7 * co);
  const double superpixel = 0.574 + 0.165 * (wholeWords(g) ? g.s * g.C / 2 : g.s * g.C);
  const double first = 1.93 + 0.5 * std::ceil(g.KH * t.taps * co / 512.0);
  bool found = false;
  for (int parts = 1; parts <= 8 && (parts == 1 || g.OW >= 16 * parts); ++parts)
    for (int rows = 1; rows <= std::min(16, g.OH); ++rows) {
      t.tile_w = (g.OW + parts - 1) / parts;
      t.pitch = t.tile_w + t.taps - 1;
      t.rows = rows;
      t.plane_bytes = size_t(rows + (g.KH - 1) / g.s) * t.pitch * 16;
      // (a tile reads past its last row)
      t.strip_bytes = (g.s * t.plane_bytes + (128 + size_t(t.taps)) * 16 + 127) / 128 * 128;
      if (t.weight_bytes + 2 * t.strip_bytes > 200 * 1024) break;
      const double superpixels = ((rows - 1.0) * g.s + g.KH) * t.pitch, loads = superpixels * superpixel;
      const double load = 1226 + 21 * (std::ceil(superpixels / (4 * kStemLoaders)) - 1) + loads;
      const double tiles = tile * (((rows - 1) * t.pitch + t.tile_w + 127) / 128);
      const double unit = std::max(tiles, load) + std::min(tiles, loads);
      const double units = double(g.N) * ((g.OH + rows - 1) / rows) * ((g.OW + t.tile_w - 1) / t.tile_w);
      t.us = float(first + (std::ceil(units / sms) * unit + 0.16 * (load + tile)) / 1900);
      if (!found || t.us < best->us) *best = t;
      found = true;
    }
  return found;
}

// What the rearranged form takes, fitted to 729 layers: two launches, a thread for each 16 bytes
// rearranged (3 channels, stride 2: a block for each row), then the tiles of whole pixel boxes;
// median error 10 %.
float rearrangedTime(int sms, const S2dShape &g, int co) {
  double tiles = 1e30;
  for (int w = 128; w >= 1; w >>= 1)
    for (int h = 128 / w; h >= 1; h >>= 1) {
      const int n = 128 / (w * h);
      tiles = std::min(tiles, double((g.OW + w - 1) / w) * ((g.OH + h - 1) / h) * ((g.N + n - 1) / n));
    }
  const bool by_rows = g.C == 3 && g.s == 2 && g.W % 2 == 0;
  const double rearrange = by_rows ? 3.43 * g.N * g.H2 * ((g.W2 + 127) / 128) / (16.0 * sms)
                                   : 4.56 * g.N * g.H2 * g.W2 * (g.C2 / 8) / (2048.0 * sms);
  const int bn = co <= 64 ? 64 : 128;
  const double waves = std::max(1.0, tiles * ((co + bn - 1) / bn) / sms) + 3.43;
  return float(2.47 + rearrange + waves * (0.358 + 0.054 * g.K2h * bn / 64 + 0.062 * co / 64));
}

}  // namespace

// Layers whose estimated time is at most a microsecond above the rearranged form's, whose second
// launch costs a host that issues it 1.9.  Of 652 sampled layers, 571 take it and run in 0.79 of the
// other's time, 32 of them more than 8 % longer on the device.
// Two kinds of large filters stay rearranged besides: those of one channel, where both strides' pixels then share 16
// bytes, half as many instructions (7x7/2, 64 channels: 92 images of 212 x 56 18.6 against 20.2 us),
// and many short rows with more than 32 output channels, whose strips waste a sixth of their
// positions (514 of 79 x 79 51.0 against 61.0, 1066 of 55 x 55, 96 channels, 62.8 against 70.7).
bool stemSuits(int sm_count, const S2dShape &g, int co, bool out_f32, const void *out, bool slower_too) {
  StemTiling t;
  const bool large = g.KH > 3;
  if (large && (g.C == 1 || (co > 32 && g.OW < 64 && uint64_t(g.N) * g.OH * g.OW > uint64_t(1) << 19))) return false;
  return g.s * g.C <= 8 && co % 16 == 0 && co <= 256 && !out_f32 && reinterpret_cast<uintptr_t>(out) % 32 == 0 &&
         uint64_t(g.H) * g.W * g.C < uint64_t(1) << 29 && uint64_t(g.N) * g.OH * g.OW < uint64_t(1) << 30 &&
         stemTiling(sm_count, g, co, &t) && (slower_too || t.us < rearrangedTime(sm_count, g, co) + 1.0f);
}

int launchStem(plb_context *ctx, const S2dShape &g, int co, bool bf16, const void *x, const void *w, const float *bias,
               void *out) {
  StemTiling t;
  if (!stemTiling(ctx->sm_count, g, co, &t)) return fail(PLB_ERR_UNSUPPORTED, "no tiling of the stem kernel");
  StemArgs a{};
  a.x = static_cast<const uint16_t *>(x);
  a.w = static_cast<const uint16_t *>(w);
  a.bias = bias;
  a.out = static_cast<__half *>(out);
  a.status = ctx->d_status;
  a.g = g;
  a.co = co;
  a.co_pad = (co + 31) / 32 * 32;
  a.taps = t.taps;
  a.pad_w = t.pad_w;
  a.shift = t.pad_w - g.padW;
  a.tile_w = t.tile_w;
  a.rows = t.rows;
  a.pitch = t.pitch;
  a.parts = (g.OW + t.tile_w - 1) / t.tile_w;
  a.h_blocks = (g.OH + t.rows - 1) / t.rows;
  a.units = g.N * a.h_blocks * a.parts;
  a.plane_bytes = uint32_t(t.plane_bytes);
  a.strip_bytes = uint32_t(t.strip_bytes);
  a.weight_bytes = uint32_t(t.weight_bytes);
  a.idesc = make_idesc(128, uint32_t(co), bf16 ? 1u : 0u, bf16 ? 1u : 0u, false, false);
  a.tmem_cols = 64;
  while (a.tmem_cols < uint32_t(2 * a.co_pad)) a.tmem_cols *= 2;
  a.fd_pitch = make_fastdiv(uint32_t(t.pitch));
  a.fd_parts = make_fastdiv(uint32_t(a.parts));
  a.fd_h_blocks = make_fastdiv(uint32_t(a.h_blocks));
  a.fd_co = make_fastdiv(uint32_t(co));
  a.fd_taps = make_fastdiv(uint32_t(t.taps));
  const int words = wholeWords(g) && reinterpret_cast<uintptr_t>(x) % 4 == 0 ? g.s * g.C / 2 : 0;
  auto launch = [&](auto kernel, std::atomic<bool> *configured) {
    std::atomic<bool> &done = configured[ctx->device & 63];
    if (!done) {
      PLB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 210 * 1024));
      done = true;
    }
    return launchPdl(ctx, kernel, dim3(unsigned(std::min(a.units, ctx->sm_count))), dim3(kStemThreads),
                     t.weight_bytes + 2 * t.strip_bytes, a);
  };
  auto pick = [&](auto type) {
    constexpr bool kBf16 = decltype(type)::value;
    static std::atomic<bool> configured[5][64] = {};  // (contexts may live on several threads)
    switch (words) {
      case 1: return launch(stemKernel<1, kBf16>, configured[1]);
      case 2: return launch(stemKernel<2, kBf16>, configured[2]);
      case 3: return launch(stemKernel<3, kBf16>, configured[3]);
      case 4: return launch(stemKernel<4, kBf16>, configured[4]);
      default: return launch(stemKernel<0, kBf16>, configured[0]);
    }
  };
  return bf16 ? pick(std::true_type()) : pick(std::false_type());
}

}  // namespace plb
