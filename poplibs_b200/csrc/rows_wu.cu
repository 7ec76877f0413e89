// Weight gradients of channel groups of 8 or 16, filters of 3x3 (and 5x5 of 8) with unit strides.
//
//   dW[r, s][co, ci] = sum over pixels of dY[pixel, co] * X[pixel + (r, s) - pad, ci]
//
// As a dense block of 128 channels the tensor core forms 16 or 8 times the sums that are
// wanted, and stores a good part of them.  Here a block takes 64 channels of a share of the tiles of
// output pixels, and a warp a whole group of them, whose sums, 9 to 25 taps of 8 x 8 or 16 x 16,
// stay in its registers until the end.  It walks down the rows of a tile with both operands in
// shared memory: a row of activations, read once by ldmatrix for each horizontal tap (turned round:
// the pixels are the reduction; two taps of 8 channels are the sixteen rows of an
// instruction), is multiplied with the output gradients of all the rows that it meets, which are
// kept in a ring of registers, one for each filter row.  Rows beyond the tile are skipped, pixels
// beyond the output are zero in both operands, so that an infinite activation meets no gradients that do not
// exist.  Padding is multiplied as zeros: an infinite gradient makes NaNs of the sums of the taps that
// reach padding from its pixel, as in the contraction (wu_sm100.cuh).  A second kernel adds the
// shares in their order (wu_reduce4_kernel).
//
// Bound by latency and the loads' rate: two or three blocks share an SM, one multiplies while
// another loads.  32 groups of 8 on 32 images of 28 x 28: 18.3 -> 14.9 us with the second kernel (operands
// in L2, 17.0 from memory).
#include <algorithm>
#include <atomic>
#include <cmath>

#include "direct.cuh"
#include "rows.h"

namespace plb {
namespace {

constexpr int kRowBytes = 128;  // of a pixel: 64 channels

struct RowsWuArgs {
  const uint8_t *x, *dy;
  float *partial;                                 // [split][group][tap][co][ci]
  long long x_n, x_h, x_w, dy_n, dy_h, dy_w;      // bytes
  int in_w, in_h, width, height, images, chans, groups;
  int pad_h, pad_w;
  int tile_w, tile_h, tile_n, tiles_w, tiles_h, tiles, slabs, splits;
  int pitch, image_rows;                          // of the activations in shared memory: pixels of a row, rows of an image
  uint32_t second, dy_second, dy_at;              // bytes from a step's first eight pixels to the other eight; to the gradients
  FastDiv fd_slabs, fd_tiles_w, fd_tiles_h;
};

__device__ __forceinline__ void loadTwoTurned(uint32_t at, uint32_t (&r)[2]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(at) : "memory");
}

template <int K, int kC>
__global__ void __launch_bounds__(32 * 64 / kC, kC == 8 ? 2 : 3)
rowsWuKernel(const __grid_constant__ RowsWuArgs g) {
  constexpr int kWarps = 64 / kC, kN = kC / 8;
  constexpr int kPairs = kC == 8 ? K / 2 : K;
  constexpr bool kOdd = kC == 8;
  extern __shared__ __align__(128) uint8_t rows_smem[];
  const uint32_t smem = smem_u32(rows_smem);
  const int tid = int(threadIdx.x), lane = tid & 31, warp = tid >> 5;
  pdl_launch_dependents();
  const int split = int(fast_div(blockIdx.x, g.fd_slabs)), slab = int(blockIdx.x) - split * g.slabs;
  const int group = slab * kWarps + warp;
  const bool mine = group < g.groups;
  const int chunk = lane & 7, chan = slab * 64 + chunk * 8, column = lane >> 3;
  const uint32_t my_chunk = smem + uint32_t(column) * kRowBytes + (uint32_t(chunk ^ column) << 4);
  const uint32_t row_bytes = uint32_t(g.pitch) * kRowBytes, dy_row_bytes = uint32_t(g.tile_w) * kRowBytes;
  float acc[K][kPairs][kN][4];
  [[maybe_unused]] float odd[K][4];
#pragma unroll
  for (int r = 0; r < K; ++r) {
#pragma unroll
    for (int s = 0; s < kPairs; ++s)
#pragma unroll
      for (int n = 0; n < kN; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[r][s][n][e] = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) odd[r][e] = 0.f;
  }
  pdl_wait();  // operands may come from the previous kernel in the stream
  const int first = int((long long)g.tiles * split / g.splits), last = int((long long)g.tiles * (split + 1) / g.splits);
#pragma unroll 1
  for (int tile = first; tile < last; ++tile) {
    const int t2 = int(fast_div(uint32_t(tile), g.fd_tiles_w)), tw = tile - t2 * g.tiles_w;
    const int tn = int(fast_div(uint32_t(t2), g.fd_tiles_h)), th = t2 - tn * g.tiles_h;
    const int w0 = tw * g.tile_w, h0 = th * g.tile_h, n0 = tn * g.tile_n;
    const int rows = min(g.tile_h, g.height - h0), total = rows + K - 1;
    if (tile != first) __syncthreads();  // (the last tile has been read)
    // ---- operands: chunk c of column x lies at x * 128 + (c ^ x % 8) * 16 of its row; a warp loads a
    // row at a time, four pixels an instruction
    auto load = [&](const uint8_t *src0, long long step_n, long long step_h, long long step_w, int ih0, int iw0, int in_h, int in_w,
                    int end, int cols, uint32_t at, int image_rows, uint32_t bytes) {
      for (int im = 0; im < g.tile_n; ++im)
#pragma unroll 1
        for (int y = warp; y < end; y += kWarps) {
          const int ih = ih0 + y;
          const bool there = uint32_t(ih) < uint32_t(in_h) && n0 + im < g.images && chan < g.chans;
          const uint8_t *src = src0 + (n0 + im) * step_n + ih * step_h + (iw0 + column) * step_w + chan * 2;
          uint32_t dst = my_chunk + at + uint32_t(im * image_rows + y) * bytes;
#pragma unroll 2
          for (int x = column, iw = iw0 + column; x < cols; x += 4, iw += 4, src += 4 * step_w) {
            const bool in = there && uint32_t(iw) < uint32_t(in_w);
            copyAsync(dst, in ? src : src0, in ? 16 : 0);
            dst = (dst + 4 * kRowBytes) ^ 64;
          }
        }
    };
    load(g.x, g.x_n, g.x_h, g.x_w, h0 - g.pad_h, w0 - g.pad_w, g.in_h, g.in_w, total, g.tile_w + K - 1, 0, g.image_rows, row_bytes);
    load(g.dy, g.dy_n, g.dy_h, g.dy_w, h0, w0, g.height, g.width, rows, g.tile_w, g.dy_at, g.tile_h, dy_row_bytes);
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (!mine) continue;

    // ---- rows
    const int left = g.width - w0;  // columns that exist (of one image)
    const int steps = min(g.tile_w * g.tile_n / 16, g.tile_n > 1 ? 1 : (left + 15) / 16);
    auto at = [&](int x, int c) { return smem + uint32_t(x) * kRowBytes + (uint32_t(c ^ (x & 7)) << 4); };
    const int pixel = lane & 7;
#pragma unroll 1
    for (int step = 0; step < steps; ++step) {
      // lanes of ldmatrix: kC 8: taps (lanes 8-15, 24-31 the second of a pair), then the other eight
      // pixels (16-31); kC 16: channels, then pixels
      const uint32_t x_half = lane & 16 ? g.second : 0, x_step = uint32_t(step) * 16 * kRowBytes;
      uint32_t a_at[kPairs], odd_at = 0, b_at;
#pragma unroll
      for (int s = 0; s < kPairs; ++s)
        a_at[s] = x_step + x_half + (kC == 8 ? at(pixel + 2 * s + (lane >> 3 & 1), warp) : at(pixel + s, 2 * warp + (lane >> 3 & 1)));
      if constexpr (kOdd) odd_at = x_step + (lane & 8 ? g.second : 0) + at(pixel + K - 1, warp);
      // gradients: the other eight pixels (lanes 8-15), then the other eight channels (16-31)
      b_at = g.dy_at + x_step + (lane & 8 ? g.dy_second : 0) + (kC == 8 ? at(pixel, warp) : at(pixel, 2 * warp + (lane >> 4)));
      // pixels beyond the image are no products: zero in the activations, too
      const int valid = g.tile_n > 1 ? min(left, 8) : min(left - step * 16, 16), k = 2 * (lane & 3);
      const bool whole = valid == (g.tile_n > 1 ? 8 : 16);
      auto keep = [&](int k0) { return (k0 + k < valid ? 0xffffu : 0u) | (k0 + k + 1 < valid ? 0xffff0000u : 0u); };
      const uint32_t mask_lo = keep(0), mask_hi = keep(g.tile_n > 1 ? 0 : 8);
      uint32_t b[K][kN][2];
#pragma unroll 1
      for (int y0 = 0; y0 < total; y0 += K) {
#pragma unroll
        for (int j = 0; j < K; ++j) {
          const int y = y0 + j;
          if (y >= total) break;
          if (y < rows) {
            if constexpr (kC == 8) {
              loadTwoTurned(b_at, b[j][0]);
            } else {
              uint32_t v[4];
              loadMatrices<true>(b_at, v);
              b[j][0][0] = v[0];
              b[j][0][1] = v[1];
              b[j][kN - 1][0] = v[2];
              b[j][kN - 1][1] = v[3];
            }
            b_at += dy_row_bytes;
          }
          const bool every = y >= K - 1 && y < rows;
#pragma unroll
          for (int s = 0; s < kPairs + (kOdd ? 1 : 0); ++s) {
            uint32_t a[4];
            if (s < kPairs) {
              loadMatrices<true>(a_at[s < kPairs ? s : 0], a);
              a_at[s < kPairs ? s : 0] += row_bytes;
            } else {
              uint32_t f[2];
              loadTwoTurned(odd_at, f);
              odd_at += row_bytes;
              a[0] = f[0];
              a[2] = f[1];
              a[1] = a[3] = 0u;
            }
            if (!whole) {
              a[0] &= mask_lo;
              a[1] &= mask_lo;
              a[2] &= mask_hi;
              a[3] &= mask_hi;
            }
#pragma unroll
            for (int r = 0; r < K; ++r) {
              if (!every && (y - r < 0 || y - r >= rows)) continue;
#pragma unroll
              for (int n = 0; n < kN; ++n) {
                uint32_t (&bb)[2] = b[(j - r + K) % K][n];
                multiply<false>(s < kPairs ? acc[r][s < kPairs ? s : 0][n] : odd[r], a, bb[0], bb[1]);
              }
            }
          }
        }
      }
    }
  }
  if (!mine) return;
  // ---- sums: row m of an instruction is (tap, channel in), column n a channel out
  float *const out = g.partial + ((long long)split * g.groups + group) * (K * K * kC * kC);
  const int ci = lane >> 2, co = 2 * (lane & 3);
#pragma unroll
  for (int r = 0; r < K; ++r)
#pragma unroll
    for (int s = 0; s < kPairs + (kOdd ? 1 : 0); ++s)
#pragma unroll
      for (int n = 0; n < kN; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (s == kPairs && e >= 2) continue;
          const float v = s < kPairs ? acc[r][s < kPairs ? s : 0][n][e] : odd[r][e];
          const int tap = r * K + (kC == 8 ? 2 * s + (e >> 1) : s);
          out[(tap * kC + n * 8 + co + (e & 1)) * kC + ci + (kC == 16 ? (e >> 1) * 8 : 0)] = v;
        }
}

bool rowsWuTiling(int sms, const RowsWuProblem &p, RowsWuTiling *best) {
  const int K = p.kernel, c = p.chans, most = c == 8 ? 2 : 3;
  const long slabs = rowsWuSlabs(p);
  // cycles of a 16-pixel step of a row
  const double step = (c == 8 ? K * (K / 2 + 1) : 2 * K * K) * 8.3;
  const double sums = 1.0e-6 * p.groups * K * K * c * c * 4 / 2.5;
  bool found = false;
  for (int steps = 1; steps <= 7 && (steps == 1 || 16 * (steps - 1) < p.width); ++steps)
    for (int images = 1; images <= (steps == 1 && p.width <= 8 ? 2 : 1); ++images) {
      const int tile_w = 16 * steps / images, pitch = (tile_w + K - 1 + 7) / 8 * 8;
      const int x_row = images * pitch * kRowBytes, dy_row = images * tile_w * kRowBytes;
      const long columns = long(upDiv(p.width, tile_w)) * upDiv(p.images, images);
      const double load = images * kRowBytes / 30.0;
      for (int rows = std::min(p.height, (110 * 1024 - x_row * (K - 1)) / (x_row + dy_row)); rows >= 1; --rows) {
        const unsigned parts = upDiv(p.height, rows);
        rows = int(upDiv(p.height, parts));  // (the fewest that make as many tiles)
        const int x_bytes = x_row * (rows + K - 1), smem = x_bytes + dy_row * rows;
        const int resident = std::max(1, std::min(most, int(226u * 1024 / unsigned(smem + 1024))));
        const long tiles = columns * parts, splits = std::max<long>(1, std::min<long>(tiles, sms * resident / slabs));
        const double rounds = up(double(tiles) / double(splits)), here = std::min(double(resident), up(double(splits * slabs) / sms));
        const double bytes = load * ((rows + K - 1) * (tile_w + K - 1) + rows * tile_w), walk = (rows + K - 1) * steps * step;
        const double busy = std::max(walk * (64 / c) * here / 4, walk * 1.6 + (rows + K - 1) * steps * 60.0);
        const float us = float(2.3 + rounds * (1200 + here * bytes + busy) / 1900 + 2.5 + double(splits) * sums);
        if (!found || us <= best->us)
          *best = RowsWuTiling{tile_w, rows, images, pitch, size_t(x_bytes), size_t(smem), tiles, int(splits), us};
        found = true;
      }
    }
  return found;
}

}  // namespace

// Of 300 sampled layers (see rows.cu) 0.78 of the tensor-core route's time in all.  With 16 channels
// the dense block wastes half as much, and rows that fill their sixteens of pixels badly, or large
// layers, are quicker there (4 groups, 45 images of 20 x 20 10.6 us there, 13.4 here; 8 groups, 87 of 42 x 42 38.5 and 43).
bool rowsWuSuits(int sm_count, const RowsWuProblem &p, RowsWuTiling *t) {
  if ((p.chans != 8 && p.chans != 16) || p.groups < 2 || (p.kernel != 3 && !(p.kernel == 5 && p.chans == 8))) return false;
  if (p.width < 1 || p.height < 1 || p.images < 1) return false;
  if ((reinterpret_cast<uintptr_t>(p.x) | reinterpret_cast<uintptr_t>(p.dy)) % 16 != 0) return false;
  if (p.width > 1 << 20 || p.height > 1 << 20 || std::abs(p.pad_h) > 1 << 20 || std::abs(p.pad_w) > 1 << 20) return false;
  if (p.chans == 16) {
    const int stepped = p.width <= 8 ? 8 : (p.width + 15) / 16 * 16;
    if (4 * p.width < 3 * stepped || 2e-6 * p.groups * 16 * p.width * p.height * p.images > 8) return false;
  }
  return rowsWuTiling(sm_count, p, t) && t->tiles <= 0x3fffffff;
}

int launchRowsWu(plb_context *ctx, const RowsWuProblem &p, const RowsWuTiling &t, float *partial) {
  RowsWuArgs g{};
  g.x = static_cast<const uint8_t *>(p.x);
  g.dy = static_cast<const uint8_t *>(p.dy);
  g.partial = partial;
  g.chans = p.groups * p.chans;
  g.groups = p.groups;
  g.x_w = g.dy_w = (long long)g.chans * 2;
  g.x_h = g.x_w * p.in_pitch_w;
  g.x_n = g.x_h * p.in_pitch_h;
  g.dy_h = g.dy_w * p.width;
  g.dy_n = g.dy_h * p.height;
  g.in_w = p.in_w;
  g.in_h = p.in_h;
  g.width = p.width;
  g.height = p.height;
  g.images = p.images;
  g.pad_h = p.pad_h;
  g.pad_w = p.pad_w;
  g.tile_w = t.tile_w;
  g.tile_h = t.tile_h;
  g.tile_n = t.tile_n;
  g.tiles_w = int(upDiv(p.width, t.tile_w));
  g.tiles_h = int(upDiv(p.height, t.tile_h));
  g.tiles = int(t.tiles);
  g.slabs = rowsWuSlabs(p);
  g.splits = t.splits;
  g.pitch = t.pitch;
  g.image_rows = t.tile_h + p.kernel - 1;
  g.second = uint32_t(t.tile_n > 1 ? g.image_rows * t.pitch : 8) * kRowBytes;
  g.dy_second = uint32_t(t.tile_n > 1 ? t.tile_h * t.tile_w : 8) * kRowBytes;
  g.dy_at = uint32_t(t.x_bytes);
  g.fd_slabs = make_fastdiv(uint32_t(g.slabs));
  g.fd_tiles_w = make_fastdiv(uint32_t(g.tiles_w));
  g.fd_tiles_h = make_fastdiv(uint32_t(g.tiles_h));
  auto launch = [&](auto kernel, std::atomic<bool> *configured) {
    std::atomic<bool> &done = configured[ctx->device & 63];
    if (!done) {
      PLB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024));
      done = true;
    }
    return launchPdl(ctx, kernel, dim3(unsigned(t.splits * g.slabs)), dim3(unsigned(32 * 64 / p.chans)), t.smem, g);
  };
  static std::atomic<bool> configured[3][64] = {};  // (contexts may live on several threads)
  if (p.chans == 16) return launch(rowsWuKernel<3, 16>, configured[0]);
  return p.kernel == 3 ? launch(rowsWuKernel<3, 8>, configured[1]) : launch(rowsWuKernel<5, 8>, configured[2]);
}

}  // namespace plb
