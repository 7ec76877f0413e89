// Convolution kernel for channel groups of 8 or 16, filters of 3x3 and 5x5 with unit strides.
//
//   out[pixel, co] = alpha * sum_{r, s, ci} act[pixel + (r, s) - pad, ci] * w[r, s, co, ci] (+ bias[co])
//
// As a dense block of 64 channels such a layer multiplies 8 or 4 times what it has to,
// and needs block-diagonal weights and a repair pass in launches of their own
// (grouped.cu).  Here a block takes 64 channels of a tile of output pixels, and a warp a whole
// group of them.  Its weights, 9 to 25 taps of 8 x 8 or 16 x 16, stay in its registers as
// operands of mma.sync, and it walks down the input rows: a row's operands, read once by ldmatrix
// for each horizontal tap (two taps of 8 channels to an instruction), are multiplied for
// all the output rows that they belong to, whose sums lie in a ring of registers, one for each
// filter row.  So shared memory is read KW times per pixel, where an operand for each tap is read
// KH * KW times (patch.cuh), and weights not at all.  A finished output row takes the place of an
// input row that has been read: a warp owns its group's channels of the tile.
//
// Bound by latency (launch, one trip to memory, the walk, the stores; two or three blocks share an SM), from
// about 30 MB on by the rate at which those blocks keep loads in flight (2.7 TB/s read and
// written).  Shared memory's rows are whole eights of pixels, so that the swizzle of a lane's addresses
// is the same in every row: with addresses formed per tap, a 16-pixel step took 160 instructions and
// 32 groups of 8 on 32 images of 28 x 28 20.5 us, now 10.0 (17.8 in three launches on dense blocks;
// operands in L2, 11.5 us from memory).
#include <algorithm>
#include <atomic>
#include <cmath>

#include "direct.cuh"
#include "rows.h"

namespace plb {
namespace {

constexpr int kRowBytes = 128;  // of a pixel: 64 channels

struct RowsArgs {
  const uint8_t *act, *wgt;
  __half *out;
  const float *bias;
  float alpha;
  long long act_n, act_h, act_w;                  // bytes
  long long out_n, out_h, ldc;                    // elements
  long long wgt_tile, wgt_row;                    // bytes
  int tap_first, tap_step_h, tap_step_w, taps_stored;
  int in_w, in_h, width, height, images, chans;   // chans: of a pixel, all groups
  int pad_h, pad_w, b_mn;
  int tile_w, tile_h, tile_n;                     // output pixels of a block (tile_n: images side by side)
  int pitch, image_rows;                          // pixels of a row, rows of an image in shared memory
  uint32_t second;                                // bytes from a step's first eight pixels to the other eight
  int first_rows;                                 // input rows loaded first
  int slabs, tiles_w, tiles_h;
  FastDiv fd_slabs, fd_tiles_w, fd_tiles_h;
};

__device__ __forceinline__ void loadTwo(uint32_t at, uint32_t (&r)[2]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(at) : "memory");
}
__device__ __forceinline__ void multiplyOne(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(b0));
}

// A sum over the pixels that exist (products with padding make a NaN of an infinite weight).
template <int KH, int KW, int kC>
__device__ __noinline__ float rowsSum(const RowsArgs &g, int group, int n, int oh, int ow, int co) {
  float sum = 0.f;
#pragma unroll 1
  for (int t = 0; t < KH * KW; ++t) {
    const int r = t / KW, s = t - r * KW, ih = oh + r - g.pad_h, iw = ow + s - g.pad_w;
    if (ih < 0 || iw < 0 || ih >= g.in_h || iw >= g.in_w) continue;
    const uint8_t *x = g.act + n * g.act_n + ih * g.act_h + iw * g.act_w + group * kC * 2;
    const uint8_t *w = g.wgt + (g.tap_first + r * g.tap_step_h + s * g.tap_step_w + group * g.taps_stored) * g.wgt_tile;
#pragma unroll 1
    for (int k = 0; k < kC; ++k)
      sum += __half2float(*reinterpret_cast<const __half *>(x + 2 * k)) *
             __half2float(*reinterpret_cast<const __half *>(g.b_mn ? w + k * g.wgt_row + co * 2 : w + co * g.wgt_row + k * 2));
  }
  return sum;
}

// kC: channels of a group; kSteps: sixteens of pixels that a warp walks together.
template <int KH, int KW, int kC, int kSteps>
__global__ void __launch_bounds__(32 * 64 / kC, kC == 8 || KH == 5 ? 2 : 3)
rowsKernel(const __grid_constant__ RowsArgs g) {
  constexpr int kWarps = 64 / kC, kN = kC / 8;
  // operands of a row: two taps of 8 channels, or one of 16
  constexpr int kPairs = kC == 8 ? KW / 2 : KW;
  constexpr bool kOdd = kC == 8;  // (the last tap of a row alone)
  extern __shared__ __align__(128) uint8_t rows_smem[];
  const uint32_t smem = smem_u32(rows_smem);
  const int tid = int(threadIdx.x), lane = tid & 31, warp = tid >> 5;
  pdl_launch_dependents();
  // ---- the block's tile
  int u = int(blockIdx.x);
  const int t1 = int(fast_div(uint32_t(u), g.fd_slabs)), slab = u - t1 * g.slabs;
  const int t2 = int(fast_div(uint32_t(t1), g.fd_tiles_w)), tw = t1 - t2 * g.tiles_w;
  const int tn = int(fast_div(uint32_t(t2), g.fd_tiles_h)), th = t2 - tn * g.tiles_h;
  const int w0 = tw * g.tile_w, h0 = th * g.tile_h, n0 = tn * g.tile_n;
  const int rows = min(g.tile_h, g.height - h0);
  const int group = slab * (64 / kC) + warp;
  const bool mine = group * kC < g.chans;
  pdl_wait();  // operands may come from the previous kernel in the stream
  // ---- input: chunk c of column x lies at x * 128 + (c ^ x % 8) * 16 of its row (rows are whole
  // eights of pixels).  A warp loads a row at a time, four pixels an instruction.
  const int chunk = lane & 7, chan = slab * 64 + chunk * 8, column = lane >> 3;
  const uint32_t my_chunk = smem + uint32_t(column) * kRowBytes + (uint32_t(chunk ^ column) << 4);
  const uint32_t row_bytes = uint32_t(g.pitch) * kRowBytes;
  {
    const int cols = g.tile_w + KW - 1, iw0 = w0 - g.pad_w + column;
    auto load = [&](int first, int end) {  // input rows of every image
      for (int im = 0; im < g.tile_n; ++im)
#pragma unroll 1
        for (int y = first + warp; y < end; y += kWarps) {
          const int ih = h0 - g.pad_h + y;
          const bool there = uint32_t(ih) < uint32_t(g.in_h) && n0 + im < g.images && chan < g.chans;
          const uint8_t *src = g.act + (n0 + im) * g.act_n + ih * g.act_h + iw0 * g.act_w + chan * 2;
          uint32_t dst = my_chunk + uint32_t(im * g.image_rows + y) * row_bytes;
#pragma unroll 2
          for (int x = column, iw = iw0; x < cols; x += 4, iw += 4, src += 4 * g.act_w) {
            const bool in = there && uint32_t(iw) < uint32_t(g.in_w);
            copyAsync(dst, in ? src : g.act, in ? 16 : 0);
            dst = (dst + 4 * kRowBytes) ^ 64;
          }
        }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load(0, g.first_rows);
    load(g.first_rows, rows + KH - 1);
  }
  // ---- weights: operand b of (tap or pair of taps, eight output channels)
  uint32_t w[KH][kPairs][kN][2];
  [[maybe_unused]] uint32_t w_odd[KH];
  float bias[kN][2];
  {
    const uint8_t *const wg = g.wgt + (long long)(mine ? group : 0) * g.taps_stored * g.wgt_tile;
    const int k = 2 * (lane & 3), n = lane >> 2;
    // B[k0 + k, + 1][n0 + n] of tap (r, s), stored by columns, or by rows and turned round below
    auto two = [&](int r, int s, int k0, int n0) {
      const uint8_t *t = wg + (g.tap_first + r * g.tap_step_h + s * g.tap_step_w) * g.wgt_tile;
      return *reinterpret_cast<const uint32_t *>(g.b_mn ? t + (k0 + n) * g.wgt_row + (n0 + k) * 2 : t + (n0 + n) * g.wgt_row + (k0 + k) * 2);
    };
#pragma unroll
    for (int r = 0; r < KH; ++r) {
#pragma unroll
      for (int s = 0; s < kPairs; ++s)
#pragma unroll
        for (int j = 0; j < kN; ++j) {
          w[r][s][j][0] = kC == 8 ? two(r, 2 * s, 0, 0) : two(r, s, 0, j * 8);
          w[r][s][j][1] = kC == 8 ? two(r, 2 * s + 1, 0, 0) : two(r, s, 8, j * 8);
        }
      if constexpr (kOdd) w_odd[r] = two(r, KW - 1, 0, 0);
    }
    if (g.b_mn) {
      auto turn = [](uint32_t &v) { asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %0;" : "+r"(v)); };
#pragma unroll
      for (int r = 0; r < KH; ++r) {
#pragma unroll
        for (int s = 0; s < kPairs; ++s)
#pragma unroll
          for (int j = 0; j < kN; ++j) {
            turn(w[r][s][j][0]);
            turn(w[r][s][j][1]);
          }
        if constexpr (kOdd) turn(w_odd[r]);
      }
    }
#pragma unroll
    for (int j = 0; j < kN; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) bias[j][e] = g.bias && mine ? g.bias[group * kC + j * 8 + k + e] : 0.f;
  }
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncthreads();

  // ---- rows
  const int total = rows + KH - 1;  // input rows
  bool all = false;                 // have arrived
  const int steps = g.tile_w * g.tile_n / 16;
  // lane l of ldmatrix: pixel l % 16 of a step; the second half of the lanes, the pair's second part
  const int pixel = lane & 7, part = lane >> 4;
  const uint32_t half = lane & 8 ? g.second : 0;
  auto at = [&](int x, int c) { return smem + uint32_t(x) * kRowBytes + (uint32_t(c ^ (x & 7)) << 4); };
#pragma unroll 1
  for (int step0 = 0; step0 < steps; step0 += kSteps) {
    uint32_t a_at[kPairs], odd_at = 0, out_at[kN];
#pragma unroll
    for (int s = 0; s < kPairs; ++s)
      a_at[s] = half + uint32_t(step0) * 16 * kRowBytes + (kC == 8 ? at(pixel + 2 * s + part, warp) : at(pixel + s, 2 * warp + part));
    if constexpr (kOdd) odd_at = half + uint32_t(step0) * 16 * kRowBytes + at(pixel + KW - 1, warp);
#pragma unroll
    for (int n = 0; n < kN; ++n)
      out_at[n] = uint32_t(step0) * 16 * kRowBytes + at(lane >> 2, warp * kN + n) + 4 * (lane & 3) - (KH - 1) * row_bytes;
    float acc[KH][kSteps][kN][4];
#pragma unroll 1
    for (int y0 = 0; y0 < total; y0 += KH) {
      if (!all && y0 + KH > g.first_rows) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        all = true;
      }
      if (!mine) continue;
#pragma unroll
      for (int j = 0; j < KH; ++j) {
        if (y0 + j >= total) break;
#pragma unroll
        for (int i = 0; i < kSteps; ++i) {
#pragma unroll
          for (int n = 0; n < kN; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[j][i][n][e] = 0.f;
#pragma unroll
          for (int s = 0; s < kPairs; ++s) {
            uint32_t a[4];
            loadMatrices<false>(a_at[s] + i * 16 * kRowBytes, a);
#pragma unroll
            for (int r = 0; r < KH; ++r)
#pragma unroll
              for (int n = 0; n < kN; ++n) multiply<false>(acc[(j - r + KH) % KH][i][n], a, w[r][s][n][0], w[r][s][n][1]);
          }
          if constexpr (kOdd) {
            uint32_t a[2];
            loadTwo(odd_at + i * 16 * kRowBytes, a);
#pragma unroll
            for (int r = 0; r < KH; ++r) multiplyOne(acc[(j - r + KH) % KH][i][0], a[0], a[1], w_odd[r]);
          }
        }
        // output row y0 + j - KH + 1 is complete
        const int o = y0 + j - KH + 1;
        if (o >= 0) {
          float any = 0.f;
#pragma unroll
          for (int i = 0; i < kSteps; ++i)
#pragma unroll
            for (int n = 0; n < kN; ++n) {
              float (&d)[4] = acc[(j + 1) % KH][i][n];
              any += (d[0] + d[1]) + (d[2] + d[3]);
            }
          if (any * 0.f != 0.f) {
#pragma unroll 1
            for (int e = 0; e < kSteps * kN * 4; ++e) {
              const int x = (step0 + e / (4 * kN)) * 16 + (lane >> 2) + (e & 2) * 4, n = e / 4 % kN;
              const int im = g.tile_n > 1 ? x >> 3 : 0, ow = w0 + (g.tile_n > 1 ? x & 7 : x);
              float v = 0.f;
#pragma unroll
              for (int i = 0; i < kSteps * kN * 4; ++i) v = i == e ? acc[(j + 1) % KH][i / (4 * kN)][i / 4 % kN][i & 3] : v;
              if (isfinite(v) || ow >= g.width || n0 + im >= g.images) continue;
              v = rowsSum<KH, KW, kC>(g, group, n0 + im, h0 + o, ow, n * 8 + 2 * (lane & 3) + (e & 1));
#pragma unroll
              for (int i = 0; i < kSteps * kN * 4; ++i)
                if (i == e) acc[(j + 1) % KH][i / (4 * kN)][i / 4 % kN][i & 3] = v;
            }
          }
          __syncwarp();  // (its input rows have been read)
#pragma unroll
          for (int i = 0; i < kSteps; ++i)
#pragma unroll
            for (int n = 0; n < kN; ++n)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                float (&d)[4] = acc[(j + 1) % KH][i][n];
                const __half2 two = __floats2half2_rn(d[2 * h] * g.alpha + bias[n][0], d[2 * h + 1] * g.alpha + bias[n][1]);
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(out_at[n] + i * 16 * kRowBytes + (h ? g.second : 0)),
                             "r"(*reinterpret_cast<const uint32_t *>(&two)) : "memory");
              }
        }
#pragma unroll
        for (int s = 0; s < kPairs; ++s) a_at[s] += row_bytes;
        odd_at += row_bytes;
#pragma unroll
        for (int n = 0; n < kN; ++n) out_at[n] += row_bytes;
      }
    }
  }
  // ---- results
  __syncthreads();
  if (chan >= g.chans) return;
  for (int im = 0; im < g.tile_n && n0 + im < g.images; ++im)
#pragma unroll 1
    for (int y = warp; y < rows; y += kWarps) {
      __half *dst = g.out + (n0 + im) * g.out_n + (h0 + y) * g.out_h + (w0 + column) * g.ldc + chan;
      uint32_t src = my_chunk + uint32_t(im * g.image_rows + y) * row_bytes;
      const int cols = min(g.tile_w, g.width - w0);
#pragma unroll 4
      for (int x = column; x < cols; x += 4, dst += 4 * g.ldc) {
        uint4 v;
        asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(src));
        *reinterpret_cast<uint4 *>(dst) = v;
        src = (src + 4 * kRowBytes) ^ 64;
      }
    }
}

// The tile of the least estimated time: rounds of blocks (those of the last begin as others end),
// each its loads and stores, and the instructions of all the SM's warps or the latency of one
// warp's walk.  Fitted to 1900 tiles of 110 layers, whose times it is 16 % off; the tile that it takes is 1.2 %
// slower than a layer's best in the mean (with products alone for instructions, and whole rounds, 6 %).
bool rowsTiling(int sms, const IgemmProblem &p, RowsTiling *best) {
  const int K = p.taps_w, c = p.k_per_tap, most = c == 8 || K == 5 ? 2 : 3;
  const long slabs = upDiv(unsigned(p.groups * c), 64);
  // cycles of a 16-pixel step of a row: its products at the rate of the SM's four pipes
  const double products = c == 8 ? K * (8.3 * (K / 2) + 4.2) : 2 * K * K * 8.3;
  bool found = false;
  for (int steps = 1; steps <= 7 && (steps == 1 || 16 * (steps - 1) < p.out_w); ++steps)
    for (int images = 1; images <= (steps == 1 && p.out_w <= 8 ? 2 : 1); ++images) {
      const int tile_w = 16 * steps / images, pitch = (tile_w + K - 1 + 7) / 8 * 8, row_bytes = images * pitch * kRowBytes;
      const long columns = slabs * upDiv(p.out_w, tile_w) * upDiv(p.out_n, images);
      // (an even number of steps of 3x3 filters is walked by twos)
      const bool twos = steps % 2 == 0 && K == 3;
      const double load = 0.0413 * images * (tile_w + K - 1) * kRowBytes, store = 0.0192 * images * std::min(tile_w, p.out_w) * kRowBytes;
      const double all = steps * (0.747 * products + (twos ? 4.0 : 14.2)) * (64 / c) / 4, one = steps * (1.34 * products + (twos ? 84 : 168));
      for (int rows = std::min(p.out_h, 110 * 1024 / row_bytes - (K - 1)); rows >= 1; --rows) {
        const unsigned tiles = upDiv(p.out_h, rows);
        rows = int(upDiv(p.out_h, tiles));  // (the fewest that make as many tiles)
        const int smem = row_bytes * (rows + K - 1), resident = std::max(1, std::min(most, int(226u * 1024 / unsigned(smem + 1024))));
        const long blocks = columns * tiles;
        const double share = double(blocks) / (sms * resident), rounds = std::max(1.0, 0.425 * up(share) + 0.575 * share);
        const double here = std::min(double(resident), up(double(blocks) / sms)), walked = rows + K - 1;
        const float us = float(1.49 + rounds * (1781 + here * (load * walked + store * rows) + walked * std::max(all * here, one)) / 1900);
        if (!found || us <= best->us) *best = RowsTiling{tile_w, rows, images, pitch, steps, size_t(smem), blocks, us};
        found = true;
      }
    }
  return found;
}

}  // namespace

// Of 300 sampled layers of 0.1 to 134 MB (2 to 32 groups, 3x3 and 5x5), those within the limits below
// take 0.66 of their time on the other routes, a few passes of 600 more than 4 % longer, at most 13 %.
// Beyond them the persistent blocks of the tensor-core route stream better (3x3, 8 groups of 16, 34 images of
// 110 x 110, 105 MB, forward: 62 there, 81 here; 30.8 MB 26 and 28), 5x5 of 16 channels is bound by mma.sync
// (10 MB: 21 and 25), and two groups of 8 leave six of a block's warps idle (12 MB: 27 and 34).
bool rowsSuits(int sm_count, const IgemmProblem &p, int type, RowsTiling *t) {
  if (type != PLB_HALF || p.groups < 2 || p.out_f32 || p.beta != 0.f || p.addend || p.a_mn || p.plan_flags != 0 ||
      p.force_tile_n != 0 || p.force_split_k != 0)
    return false;
  const int c = p.k_per_tap;
  if ((c != 8 && c != 16) || p.n_total != c || p.taps_h != p.taps_w || (p.taps_h != 3 && p.taps_h != 5)) return false;
  if (p.stride_h != 1 || p.stride_w != 1 || p.dil_h != 1 || p.dil_w != 1) return false;
  if (p.act_group_stride != uint64_t(c) * 2 || p.out_group_stride != c) return false;
  uint64_t at = reinterpret_cast<uintptr_t>(p.act) | p.act_strides[0] | reinterpret_cast<uintptr_t>(p.out) | uint64_t(p.ldc) * 2;
  if (p.act_dims[2] > 1) at |= p.act_strides[1];
  if (p.out_h > 1) at |= uint64_t(p.out_stride_h) * 2;
  if (p.out_n > 1) at |= p.act_strides[2] | uint64_t(p.out_stride_n) * 2;
  if (at % 16 != 0 || (reinterpret_cast<uintptr_t>(p.wgt) | p.wgt_strides[0] | p.wgt_strides[1]) % 4 != 0) return false;
  if (p.out_w > 1 << 20 || p.out_h > 1 << 20 || std::abs(p.pad_h) > 1 << 20 || std::abs(p.pad_w) > 1 << 20) return false;
  const double megabytes = 2e-6 * p.groups * c * p.out_w * p.out_h * p.out_n;
  const double most = c == 16 ? (p.taps_w == 5 ? 5 : p.b_mn ? 60 : 28) : p.groups < 4 ? (p.taps_w == 5 ? 0.5 : 5) : p.taps_w == 5 || p.b_mn ? 1e9 : 100;
  return megabytes <= most && rowsTiling(sm_count, p, t) && t->blocks <= 0x3fffffff;
}

int launchRows(plb_context *ctx, const IgemmProblem &p, const RowsTiling &t) {
  RowsArgs g{};
  g.act = static_cast<const uint8_t *>(p.act);
  g.wgt = static_cast<const uint8_t *>(p.wgt);
  g.out = static_cast<__half *>(p.out);
  g.bias = p.bias;
  g.alpha = p.alpha;
  g.act_w = (long long)p.act_strides[0];
  g.act_h = (long long)p.act_strides[1];
  g.act_n = (long long)p.act_strides[2];
  g.ldc = p.ldc;
  g.out_h = p.out_stride_h ? p.out_stride_h : (long long)p.out_w * p.ldc;
  g.out_n = p.out_stride_n ? p.out_stride_n : (long long)p.out_h * p.out_w * p.ldc;
  g.wgt_row = (long long)p.wgt_strides[0];
  g.wgt_tile = (long long)p.wgt_strides[1];
  g.taps_stored = p.taps_stored ? p.taps_stored : p.taps_h * p.taps_w;
  const int pitch = p.tap_pitch_h ? p.tap_pitch_h : p.taps_w;
  g.tap_first = (p.tap_first_h + (p.flip_h ? (p.taps_h - 1) * p.tap_step_h : 0)) * pitch + p.tap_first_w +
                (p.flip_w ? (p.taps_w - 1) * p.tap_step_w : 0);
  g.tap_step_h = (p.flip_h ? -p.tap_step_h : p.tap_step_h) * pitch;
  g.tap_step_w = p.flip_w ? -p.tap_step_w : p.tap_step_w;
  g.in_w = int(p.act_dims[1]);
  g.in_h = int(p.act_dims[2]);
  g.width = p.out_w;
  g.height = p.out_h;
  g.images = p.out_n;
  g.chans = p.groups * p.k_per_tap;
  g.pad_h = p.pad_h;
  g.pad_w = p.pad_w;
  g.b_mn = p.b_mn ? 1 : 0;
  g.tile_w = t.tile_w;
  g.tile_h = t.tile_h;
  g.tile_n = t.tile_n;
  g.pitch = t.pitch;
  g.image_rows = t.tile_h + p.taps_h - 1;
  g.second = uint32_t(t.tile_n > 1 ? g.image_rows * t.pitch : 8) * kRowBytes;
  g.first_rows = std::min(t.tile_h + p.taps_h - 1, std::max(p.taps_h, (t.tile_h / 2 + p.taps_h - 1) / p.taps_h * p.taps_h));
  g.slabs = int(upDiv(g.chans, 64));
  g.tiles_w = int(upDiv(p.out_w, t.tile_w));
  g.tiles_h = int(upDiv(p.out_h, t.tile_h));
  g.fd_slabs = make_fastdiv(uint32_t(g.slabs));
  g.fd_tiles_w = make_fastdiv(uint32_t(g.tiles_w));
  g.fd_tiles_h = make_fastdiv(uint32_t(g.tiles_h));
  auto launch = [&](auto kernel, std::atomic<bool> *configured) {
    std::atomic<bool> &done = configured[ctx->device & 63];
    if (!done) {
      PLB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024));
      done = true;
    }
    return launchPdl(ctx, kernel, dim3(unsigned(t.blocks)), dim3(unsigned(32 * 64 / p.k_per_tap)), t.smem, g);
  };
  static std::atomic<bool> configured[8][64] = {};  // (contexts may live on several threads)
  const bool two = t.steps % 2 == 0;
  if (p.k_per_tap == 8) {
    if (p.taps_w == 3) return two ? launch(rowsKernel<3, 3, 8, 2>, configured[0]) : launch(rowsKernel<3, 3, 8, 1>, configured[1]);
    return launch(rowsKernel<5, 5, 8, 1>, configured[2]);
  }
  if (p.taps_w == 3) return two ? launch(rowsKernel<3, 3, 16, 2>, configured[3]) : launch(rowsKernel<3, 3, 16, 1>, configured[4]);
  return launch(rowsKernel<5, 5, 16, 1>, configured[5]);
}

}  // namespace plb
