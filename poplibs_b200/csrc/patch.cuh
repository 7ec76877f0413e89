// Convolution kernel for narrow channel groups and small ragged layers.
//
//   out[pixel, co] = alpha * sum_{tap, ci} act[pixel + offset(tap), ci] * w[tap, co, ci] (+ bias[co])
//
// A group of 8 channels fills a sixteenth of a 128-byte operand row and of a tcgen05
// instruction's columns: as dense blocks of neighbouring groups such layers multiply 8
// zeros for each weight and need block-diagonal weights and a repair pass besides.  Here a
// block keeps the weights of a few neighbouring groups and the input patch of a tile of
// output pixels in shared memory, each pixel's channels of a group rounded up to chunks of
// eight.  ldmatrix takes a row of eight channels from any pixel, so the operand of a filter
// tap is the patch itself, shifted, and each group is multiplied on its own with mma.sync
// (m16n8k16: 16 pixels x 8 output channels x two chunks), whose quarter of tcgen05's rate
// is more than the useful eighth.  Channel counts and addresses are free: chunks are
// loaded from wherever their elements lie, float operands as two bfloat16 pieces.
// Bound by shared memory: one ldmatrix per instruction with 8 output channels.  Loops outside
// the contraction stay rolled: a training step runs several kernels in turn, and with twice
// this code (80 to 139 KB an instance, now 40 to 50) the instructions came from memory each time.
#pragma once

#include <type_traits>

#include "direct.cuh"
#include "patch.h"

namespace plb {

constexpr int kPatchThreads = 256, kPatchWarps = 8;

struct PatchPhase {
  int out_w, out_h;        // output positions
  int taps_h, taps_w, dil_h, dil_w;
  int row0, col0;          // patch row / column that tap (0, 0) of the tile's first pixel reads
  int tap_first, tap_step_h, tap_step_w;  // tap (r, s) is stored tile first + r * step_h + s * step_w
  int pad_h, pad_w;        // (repair)
  int table, chunks;       // its entries of the chunk table
  long long out;           // elements from PatchArgs::out
};

struct PatchArgs {
  const uint8_t *act, *wgt;
  long long act_n, act_group, wgt_tile, wgt_row;  // bytes
  int act_w, act_h;        // bytes (an image is below 1 GB)
  int in_w, in_h, images, stride_h, stride_w;
  int k, n_total, groups, taps_stored;
  int units;               // chunks of a tap: ceil(k / 8)
  int group_block, n_block, n_blocks;  // groups and output channels of a block
  int tile_w, tile_h, tile_n, tiles_w, tiles_h, tiles;  // output pixels of a tile
  int patch_w, patch_h, patch_pixels, pixel_chunks;  // pixel_chunks: odd, so that ldmatrix is free of conflicts
  int first_h, first_w;    // input row / column of the patch's first pixel, relative to the tile's
  int m, m_chunks, n_parts;                       // pixels of a tile; shares of m and n
  int weight_chunks, weight_row;                  // chunks of a group's weights; 16-byte pieces of a K row (MN-major)
  // shared memory: chunk table, tables of the tile's and of the patch's pixels, weights, patch, results
  int at_pixels, at_patch_pixels, at_weights, weight_bytes, patch_bytes, stage_pitch;  // stage_pitch: elements
  FastDiv fd_units, fd_patch_w, fd_patch_h, fd_tile_w, fd_tile_h, fd_tiles_w, fd_tiles_h, fd_blocks;
  FastDiv fd_group_weights, fd_chunk_weights, fd_weight_cols;  // units of a group's weights, of a chunk, of a K row
  int blocks_per_set, act_vec, wgt_vec, fmt_a, fmt_b;
  void *out;
  long long ldc, out_h, out_n, out_group;         // elements
  int run_vec;             // bytes of an aligned store of a pixel's run of channels
  const float *bias;
  float alpha;
  int out_f32, repair, phases;
  PatchPhase phase[kPatchMaxPhases];
};

template <bool kBf16>
__device__ __forceinline__ void multiplyHalfStep(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  if constexpr (kBf16)
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(b0));
  else
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(b0));
}

template <int kType>
__device__ __forceinline__ float patchValue(const uint8_t *p, int fmt) {
  if constexpr (kType == PLB_FLOAT) return *reinterpret_cast<const float *>(p);
  if constexpr (kType == PLB_HALF) return __half2float(*reinterpret_cast<const __half *>(p));
  return __half2float(__half(__nv_cvt_fp8_to_halfraw(*p, fmt == PLB_F152 ? __NV_E5M2 : __NV_E4M3)));
}

// An output in the stage that is not finite again, as the sum over the products that exist,
// padding left out.
template <int kType, bool kBMn>
__device__ __noinline__ void repairOutput(const PatchArgs &g, const PatchPhase &ph, uint8_t *stage, int at, int group, int image, int oh, int ow, int col) {
  if (isfinite(g.out_f32 ? reinterpret_cast<float *>(stage)[at] : __half2float(reinterpret_cast<__half *>(stage)[at]))) return;
  constexpr int es = DirectUnit<kType, false>::kBytes;
  float sum = 0.f;
#pragma unroll 1
  for (int r = 0; r < ph.taps_h; ++r)
#pragma unroll 1
    for (int s = 0; s < ph.taps_w; ++s) {
      const int ih = oh * g.stride_h + r * ph.dil_h - ph.pad_h, iw = ow * g.stride_w + s * ph.dil_w - ph.pad_w;
      if (ih < 0 || iw < 0 || ih >= g.in_h || iw >= g.in_w) continue;
      const uint8_t *x = g.act + group * g.act_group + image * g.act_n + (long long)ih * g.act_h + (long long)iw * g.act_w;
      const uint8_t *w = g.wgt + (ph.tap_first + r * ph.tap_step_h + s * ph.tap_step_w + group * g.taps_stored) * g.wgt_tile;
#pragma unroll 1
      for (int k = 0; k < g.k; ++k)
        sum += patchValue<kType>(x + k * es, g.fmt_a) *
               patchValue<kType>(kBMn ? w + k * g.wgt_row + col * es : w + col * g.wgt_row + k * es, g.fmt_b);
    }
  const float v = sum * g.alpha + (g.bias ? g.bias[group * g.n_total + col] : 0.f);
  if (g.out_f32)
    reinterpret_cast<float *>(stage)[at] = v;
  else
    reinterpret_cast<__half *>(stage)[at] = __float2half_rn(v);
}

// Two neighbouring outputs, of which `left` exist, to column `col` from `at` in the stage.
static __device__ __noinline__ void stageSome(uint32_t at, int col, int left, float v0, float v1, int f32) {
  if (f32) {
    if (left > 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + 4 * col), "f"(v0) : "memory");
    if (left > 1) asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + 4 * col + 4), "f"(v1) : "memory");
  } else {
    if (left > 0) asm volatile("st.shared.b16 [%0], %1;" ::"r"(at + 2 * col), "h"(__half_as_ushort(__float2half_rn(v0))) : "memory");
    if (left > 1) asm volatile("st.shared.b16 [%0], %1;" ::"r"(at + 2 * col + 2), "h"(__half_as_ushort(__float2half_rn(v1))) : "memory");
  }
}

// NT: blocks of eight output channels of an item, MT: of sixteen pixels.
template <int kType, bool kBMn, int MT, int NT>
__global__ void __launch_bounds__(kPatchThreads, 2)
patchKernel(const __grid_constant__ PatchArgs g) {
  constexpr bool kBf16 = kType == PLB_FLOAT;
  constexpr int kPlanes = kBf16 ? 2 : 1;
  using Unit = DirectUnit<kType, false>;
  constexpr int es = Unit::kBytes;
  extern __shared__ __align__(16) uint8_t patch_smem[];
  __shared__ int odd_flag;
  const uint32_t smem = smem_u32(patch_smem);
  const uint32_t weights = smem + g.at_weights, patch = weights + kPlanes * g.weight_bytes;
  uint8_t *const stage = patch_smem + g.at_weights + kPlanes * (g.weight_bytes + g.patch_bytes);
  const int tid = int(threadIdx.x), lane = tid & 31, warp = tid >> 5;
  // the blocks of a tile side by side: neighbouring groups of the same pixels
  const int set = int(fast_div(blockIdx.x, g.fd_blocks)), which = int(blockIdx.x) - set * g.blocks_per_set;
  const int group0 = which / g.n_blocks * g.group_block, n0 = which % g.n_blocks * g.n_block;
  const int n_here = min(g.n_block, g.n_total - n0), sets = int(gridDim.x) / g.blocks_per_set;
  if (tid == 0) odd_flag = 0;
  // ---- tables, the same for all tiles
  // chunk c of the phases: where the patch holds tap (r, s), channels 8u.., relative to an
  // output pixel's own place (bytes), and the stored tile of weights that meets it
  uint2 *const table = reinterpret_cast<uint2 *>(patch_smem);
  const uint32_t b_chunk = kBMn ? uint32_t(g.weight_row) * 128 : uint32_t((g.n_block + 7) / 8) * 128;
#pragma unroll 1
  for (int p = 0; p < g.phases; ++p) {
    const PatchPhase &ph = g.phase[p];
#pragma unroll 1
    for (int i = tid; i < ph.chunks; i += kPatchThreads) {
      const int tap = int(fast_div(uint32_t(i), g.fd_units)), u = i - tap * g.units, r = tap / ph.taps_w, s = tap - r * ph.taps_w;
      const int at = ((ph.row0 + r * ph.dil_h) * g.patch_w + ph.col0 + s * ph.dil_w) * g.pixel_chunks + u;
      table[ph.table + i] = make_uint2(uint32_t(at) * 16, uint32_t(ph.tap_first + r * ph.tap_step_h + s * ph.tap_step_w) << 16 | uint32_t(u));
    }
  }
  // pixel m of a tile: its place in the patch (bytes), its image, row and column
  uint2 *const pixels = reinterpret_cast<uint2 *>(patch_smem + g.at_pixels);
#pragma unroll 1
  for (int m = tid; m < g.m_chunks * MT * 16; m += kPatchThreads) {
    const int mm = min(m, g.m - 1);
    const int t = int(fast_div(uint32_t(mm), g.fd_tile_w)), im = int(fast_div(uint32_t(t), g.fd_tile_h));
    const int th = t - im * g.tile_h, tw = mm - t * g.tile_w;
    pixels[m] = make_uint2(uint32_t(((im * g.patch_h + th * g.stride_h) * g.patch_w + tw * g.stride_w) * g.pixel_chunks) * 16,
                           uint32_t(im) << 24 | uint32_t(th) << 12 | uint32_t(tw));
  }
  // pixel of the patch: its image, row and column
  uint32_t *const patch_pixels = reinterpret_cast<uint32_t *>(patch_smem + g.at_patch_pixels);
#pragma unroll 1
  for (int i = tid; i < g.patch_pixels; i += kPatchThreads) {
    const int row = int(fast_div(uint32_t(i), g.fd_patch_w)), im = int(fast_div(uint32_t(row), g.fd_patch_h));
    patch_pixels[i] = uint32_t(im) << 24 | uint32_t(row - im * g.patch_h) << 12 | uint32_t(i - row * g.patch_w);
  }
  __syncthreads();
  pdl_wait();  // operands may come from the previous kernel in the stream
  int odd = 0;
  // units first, + step .. of what `source` says, four loads of a thread in flight
  auto loadUnits = [&](int first, int step, int count, int fmt, uint32_t plane, auto &&source) {
#pragma unroll 1
    for (int i0 = first; i0 < count; i0 += 4 * step) {
      Unit u[4];
      uint32_t dst[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint8_t *p = g.act;
        int n = 0;
        dst[j] = 0u;
        if (i0 + j * step < count) dst[j] = source(i0 + j * step, p, n);
        u[j].loadSome(p, n);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (dst[j]) u[j].store(dst[j], plane, fmt, odd);
    }
  };
  // (vec: half units on 16-byte addresses)
  auto load = [&](bool vec, int first, int step, int count, int fmt, uint32_t plane, auto &&source) {
    if constexpr (kType == PLB_HALF) {
      if (vec) {
#pragma unroll 2
        for (int i = first; i < count; i += step) {
          const uint8_t *p = nullptr;
          int n = 0;
          const uint32_t dst = source(i, p, n);
          copyAsync(dst, n > 0 ? p : g.act, n > 0 ? min(n, 8) * 2 : 0);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        return;
      }
    }
    loadUnits(first, step, count, fmt, plane, source);
  };
  // ---- weights, chunks in the order of the table: K-major [group][chunk][column][8],
  // MN-major [group][chunk][8 rows][columns]
  {
    const int inner = kBMn ? 8 * ((g.n_block + 7) / 8) : (g.n_block + 7) / 8 * 8, per_group = g.weight_chunks * inner;
    auto source = [&](int i, const uint8_t *&p, int &n) {
      const int gi = int(fast_div(uint32_t(i), g.fd_group_weights)), rest = i - gi * per_group;
      const int chunk = int(fast_div(uint32_t(rest), g.fd_chunk_weights)), in = rest - chunk * inner;
      const uint32_t what = table[chunk].y;
      const int tile = int(what >> 16), c = int(what & 0xffffu) * 8;
      const uint8_t *w = g.wgt + ((group0 + gi) * g.taps_stored + tile) * g.wgt_tile;
      if constexpr (kBMn) {
        const int row = int(fast_div(uint32_t(in), g.fd_weight_cols)), col = in - row * (inner / 8);
        p = w + (c + row) * g.wgt_row + (n0 + col * 8) * es;
        n = c + row < g.k ? n_here - col * 8 : 0;
        return weights + uint32_t(((gi * g.weight_chunks + chunk) * 8 + row) * g.weight_row + col) * 16;
      } else {
        p = w + (n0 + in) * g.wgt_row + c * es;
        n = in < n_here ? g.k - c : 0;
        return weights + uint32_t(i) * 16;
      }
    };
    load(g.wgt_vec != 0, tid, kPatchThreads, g.group_block * per_group, g.fmt_b, uint32_t(g.weight_bytes), source);
  }

  // ---- tiles of output pixels
  auto tileOrigin = [&](int tile, int &w0, int &h0, int &image0) {
    const int t = int(fast_div(uint32_t(tile), g.fd_tiles_w)), tn = int(fast_div(uint32_t(t), g.fd_tiles_h));
    w0 = (tile - t * g.tiles_w) * g.tile_w;
    h0 = (t - tn * g.tiles_h) * g.tile_h;
    image0 = tn * g.tile_n;
  };
  // a thread loads one chunk of every `pixel_step`th pixel
  const int chunks = g.group_block * g.units, pixel_step = kPatchThreads / chunks;
  const int my_chunk = tid % chunks, my_pixel = tid / chunks < pixel_step ? tid / chunks : g.patch_pixels;
  const int my_group = int(fast_div(uint32_t(my_chunk), g.fd_units)), my_channel = (my_chunk - my_group * g.units) * 8;
  const uint8_t *const my_act = g.act + (group0 + my_group) * g.act_group + my_channel * es;
  const uint32_t my_patch = patch + uint32_t(my_chunk) * 16;
  auto loadPatch = [&](int tile) {
    int w0, h0, image0;
    tileOrigin(tile, w0, h0, image0);
    const int ih0 = h0 * g.stride_h + g.first_h, iw0 = w0 * g.stride_w + g.first_w, images = g.images - image0;
    const uint8_t *base = my_act + image0 * g.act_n + ((long long)ih0 * g.act_h + (long long)iw0 * g.act_w);
    const int rest = g.k - my_channel;
    auto source = [&](int i, const uint8_t *&p, int &n) {
      const uint32_t at = patch_pixels[i];
      const int im = int(at >> 24), ph = int(at >> 12 & 0xfffu), pw = int(at & 0xfffu);
      const bool in = uint32_t(ih0 + ph) < uint32_t(g.in_h) && uint32_t(iw0 + pw) < uint32_t(g.in_w) && im < images;
      p = base + im * g.act_n + (ph * g.act_h + pw * g.act_w);
      n = in ? rest : 0;
      return my_patch + uint32_t(i * g.pixel_chunks) * 16;
    };
    load(g.act_vec != 0, my_pixel, pixel_step, g.patch_pixels, g.fmt_a, uint32_t(g.patch_bytes), source);
  };
  // warps share out (phase, group, part of n), and what is left of them the pixels
  const int combos = g.phases * g.group_block * g.n_parts;
  const int share = combos < kPatchWarps ? kPatchWarps / combos : 1;  // warps to a combination
  // (all columns of an item exist)
  const bool whole_columns = n_here % (8 * NT) == 0;
  // (from one tile before the first: only its patch is asked for)
#pragma unroll 1
  for (int tile = set - sets; tile < g.tiles; tile += sets) {
    int w0 = 0, h0 = 0, image0 = 0;
    if (tile >= 0) {
      if (kBf16 && odd) *static_cast<volatile int *>(&odd_flag) = 1;
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      tileOrigin(tile, w0, h0, image0);
    }
    const bool has_odd = kBf16 && *static_cast<volatile int *>(&odd_flag) != 0;
#pragma unroll 1
    for (int combo = tile < 0 ? combos : share > 1 ? warp % combos : warp; combo < combos; combo += share > 1 ? combos : kPatchWarps) {
      const int t1 = combo / g.n_parts, np = combo - t1 * g.n_parts, p = t1 / g.group_block, gi = t1 - p * g.group_block;
      const PatchPhase &ph = g.phase[p];
      // weights: lanes 0-7 the first chunk of a pair, 8-15 the second; 16-31 the next eight
      // columns, or with one block of columns the next pair
      constexpr bool kTwoPairs = NT == 1;
      const uint32_t b_at = weights + uint32_t(gi * g.weight_chunks + ph.table + (lane >> 3) % (kTwoPairs ? 4 : 2)) * b_chunk +
                            (kBMn ? uint32_t((lane & 7) * g.weight_row + np * NT + (kTwoPairs ? 0 : lane >> 4)) * 16
                                  : uint32_t(np * NT * 8 + (lane & 7) + (kTwoPairs ? 0 : (lane >> 4) * 8)) * 16);
      constexpr uint32_t b_col = kBMn ? 32u : 256u;  // sixteen columns on
      const uint32_t *const entry = reinterpret_cast<const uint32_t *>(table + ph.table);
      const int group = group0 + gi, col0 = np * NT * 8 + (lane & 3) * 2, pairs = ph.chunks / 2;
      const uint32_t a_first = patch + uint32_t(gi * g.units) * 16;
      float bias[NT][2];
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) bias[j][e] = g.bias && col0 + j * 8 + e < n_here ? g.bias[group * g.n_total + n0 + col0 + j * 8 + e] : 0.f;
#pragma unroll 1
      for (int mc = share > 1 ? warp / combos : 0; mc < g.m_chunks; mc += share) {
        if (share > 1 && warp >= share * combos) break;
        uint32_t a_at[MT];
#pragma unroll
        for (int i = 0; i < MT; ++i) a_at[i] = a_first + pixels[(mc * MT + i) * 16 + (lane & 15)].x;
        float acc[MT][NT][4];
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
        uint32_t b[kPlanes][(NT + 1) / 2][4], b_now = b_at;
        auto fetchWeights = [&] {
#pragma unroll
          for (int q = 0; q < kPlanes; ++q)
#pragma unroll
            for (int j = 0; j < (NT + 1) / 2; ++j) loadMatrices<kBMn>(b_now + j * b_col + q * g.weight_bytes, b[q][j]);
        };
        // products of a pair of chunks (or the last one alone) with the weights in registers
        // (second: the second of two pairs)
        auto step = [&](auto whole, auto second, int c) {
          constexpr bool kPair = decltype(whole)::value;
          constexpr int kAt = decltype(second)::value ? 2 : 0;
          const uint32_t a_off = entry[2 * (c + (kPair ? lane >> 4 : 0))];
          uint32_t a[kPlanes][MT][4];
#pragma unroll
          for (int q = 0; q < kPlanes; ++q)
#pragma unroll
            for (int i = 0; i < MT; ++i) loadMatrices<false>(a_at[i] + a_off + q * g.patch_bytes, a[q][i]);
          auto product = [&](int qa, int qb) {
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
              for (int j = 0; j < NT; ++j) {
                const uint32_t b0 = b[qb][j / 2][j % 2 * 2 + kAt], b1 = b[qb][j / 2][j % 2 * 2 + kAt + 1];
                if constexpr (kPair)
                  multiply<kBf16>(acc[i][j], a[qa][i], b0, b1);
                else
                  multiplyHalfStep<kBf16>(acc[i][j], a[qa][i][0], a[qa][i][1], b0);
              }
          };
          product(0, 0);
          if constexpr (kBf16) {
            if (has_odd) {
#pragma unroll
              for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) a[0][i][e] = finitePair(a[0][i][e]);
#pragma unroll
              for (int j = 0; j < (NT + 1) / 2; ++j)
#pragma unroll
                for (int e = kAt; e < (kTwoPairs ? kAt + 2 : 4); ++e) b[0][j][e] = finitePair(b[0][j][e]);
            }
            product(1, 0);
            product(0, 1);
          }
        };
        int c = 0;
        if constexpr (kTwoPairs) {
#pragma unroll 2
          for (int i = 0; i < pairs / 2; ++i, c += 4, b_now += 4 * b_chunk) {
            fetchWeights();
            step(std::true_type(), std::false_type(), c);
            step(std::true_type(), std::true_type(), c + 2);
          }
          if (c < ph.chunks) {
            fetchWeights();
            if (pairs & 1) {
              step(std::true_type(), std::false_type(), c);
              if (ph.chunks & 1) step(std::false_type(), std::true_type(), c + 2);
            } else {
              step(std::false_type(), std::false_type(), c);
            }
          }
        } else {
#pragma unroll 2
          for (int i = 0; i < pairs; ++i, c += 2, b_now += 2 * b_chunk) {
            fetchWeights();
            step(std::true_type(), std::false_type(), c);
          }
          if (c < ph.chunks) {
            fetchWeights();
            step(std::false_type(), std::false_type(), c);
          }
        }
        // (with `repair`, products with padding may have made a NaN of an infinite weight)
        float any = 0.f;
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) any += acc[i][j][e] * 0.f;
        // scale, bias, cast -> the stage: [phase][pixel][group][column]
        const int rows = g.m - mc * MT * 16 - (lane >> 2);
        const int at0 = (p * g.m + mc * MT * 16 + (lane >> 2)) * g.stage_pitch + gi * n_here + col0;
        const uint32_t at_stage = smem_u32(stage) + uint32_t(at0) * (g.out_f32 ? 4 : 2);
        const uint32_t stage_down = uint32_t(8 * g.stage_pitch) * (g.out_f32 ? 4 : 2);
        const bool whole = whole_columns && (mc + 1) * MT * 16 <= g.m;
#pragma unroll
        for (int h = 0; h < 2 * MT; ++h)
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            const float v0 = acc[h / 2][j][h % 2 * 2] * g.alpha + bias[j][0], v1 = acc[h / 2][j][h % 2 * 2 + 1] * g.alpha + bias[j][1];
            const uint32_t s = at_stage + h * stage_down;
            if (!whole) {
              if (h * 8 < rows) stageSome(s, j * 8, n_here - col0 - j * 8, v0, v1, g.out_f32);
            } else if (g.out_f32) {
              asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(s + j * 32), "f"(v0), "f"(v1) : "memory");
            } else {
              const __half2 two = __floats2half2_rn(v0, v1);
              asm volatile("st.shared.b32 [%0], %1;" ::"r"(s + j * 16), "r"(*reinterpret_cast<const uint32_t *>(&two)) : "memory");
            }
          }
        if (g.repair && any != 0.f) {
#pragma unroll 1
          for (int i = 0; i < MT * NT * 4; ++i) {
            const int row = i / (2 * NT) * 8, m = mc * MT * 16 + (lane >> 2) + row, col = col0 + i / 2 % NT * 8 + i % 2;
            if (m >= g.m || col >= n_here) continue;
            const uint32_t at = pixels[m].y;
            const int image = image0 + int(at >> 24), oh = h0 + int(at >> 12 & 0xfffu), ow = w0 + int(at & 0xfffu);
            if (oh >= ph.out_h || ow >= ph.out_w || image >= g.images) continue;
            repairOutput<kType, kBMn>(g, ph, stage, (p * g.m + m) * g.stage_pitch + gi * n_here + col, group, image, oh, ow, n0 + col);
          }
        }
      }
    }
    if (tile >= 0) __syncthreads();
    // the next tile's patch is on its way while this tile's results leave
    if (tile + sets < g.tiles)
      loadPatch(tile + sets);
    else
      // (earlier, the next kernel's blocks take the room that blocks of this one free, and come
      // to lie several on one SM: a step of five calls 42.8 -> 38.0 us)
      pdl_launch_dependents();
    if (tile < 0) continue;
    const int os = g.out_f32 ? 4 : 2;
    const int pieces = g.group_block * n_here * os / g.run_vec;
    // a thread stores one piece of every `m_step`th pixel's run, or with more pieces than
    // threads, several
    const int m_step = max(1, kPatchThreads / pieces);
#pragma unroll 1
    for (int piece = pieces > kPatchThreads ? tid : tid % pieces; piece < pieces; piece += kPatchThreads) {
      const int m_first = pieces > kPatchThreads ? 0 : tid / pieces;
      if (m_first >= m_step) break;
#pragma unroll 1
      for (int p = 0; p < g.phases; ++p) {
        const PatchPhase &ph = g.phase[p];
        uint8_t *const base = static_cast<uint8_t *>(g.out) +
                              (ph.out + image0 * g.out_n + h0 * g.out_h + w0 * g.ldc + group0 * g.out_group + n0) * os + piece * g.run_vec;
        const int most_h = ph.out_h - h0, most_w = ph.out_w - w0, images = g.images - image0;
        const uint8_t *src = stage + (p * g.m + m_first) * g.stage_pitch * os + piece * g.run_vec;
#pragma unroll 1
        for (int m = m_first; m < g.m; m += m_step, src += m_step * g.stage_pitch * os) {
          const uint32_t at = pixels[m].y;
          const int im = int(at >> 24), th = int(at >> 12 & 0xfffu), tw = int(at & 0xfffu);
          if (th >= most_h || tw >= most_w || im >= images) continue;
          uint8_t *dst = base + (im * g.out_n + th * g.out_h + tw * g.ldc) * os;
          int width = g.run_vec;
          asm volatile("" : "+r"(width));  // (one loop, not one for each width)
          switch (width) {
            case 16: *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(src); break;
            case 8: *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(src); break;
            case 4: *reinterpret_cast<uint32_t *>(dst) = *reinterpret_cast<const uint32_t *>(src); break;
            default: *reinterpret_cast<uint16_t *>(dst) = *reinterpret_cast<const uint16_t *>(src); break;
          }
        }
      }
    }
  }
}

struct PatchVariant {
  bool b_mn;
  int mt, nt;
  unsigned grid;
  size_t smem;
};
int launchPatchHalf(plb_context *ctx, const PatchVariant &v, const PatchArgs &g);
int launchPatchFloat(plb_context *ctx, const PatchVariant &v, const PatchArgs &g);
int launchPatchQuarter(plb_context *ctx, const PatchVariant &v, const PatchArgs &g);

}  // namespace plb
