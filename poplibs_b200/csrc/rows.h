// Convolutions of narrow channel groups, a warp to a group (rows.cu), and their weight
// gradients (rows_wu.cu).
#pragma once

#include "runtime.h"

namespace plb {

// For the searches of tilings, which every call makes: quotients of positive numbers below 2^31
// rounded up, and the ceiling of one below 2^62 (std::ceil is a call).
inline unsigned upDiv(unsigned a, unsigned b) { return (a + b - 1) / b; }
inline double up(double v) {
  const double whole = double((long long)v);
  return whole < v ? whole + 1 : whole;
}

// Output pixels of a block, `steps` sixteens of them to a row of its images.
struct RowsTiling {
  int tile_w, tile_h, tile_n, pitch, steps;
  size_t smem;
  long blocks;
  float us;
};
// Whether this problem (`type`: the operands' element type, all pointers the caller's) runs
// on the kernel that walks the rows of a group with its weights in registers, and how.
bool rowsSuits(int sm_count, const IgemmProblem &p, int type, RowsTiling *t);
int launchRows(plb_context *ctx, const IgemmProblem &p, const RowsTiling &t);

// Weight gradient of half channel groups, `chans` in and out each, of a kernel x kernel filter with
// unit strides and dilations.
struct RowsWuProblem {
  const void *x, *dy;
  int groups, chans, kernel, images;
  int in_w, in_h;              // extent that is read, of rows and images of in_pitch_w, in_pitch_h pixels
  int in_pitch_w, in_pitch_h;
  int width, height;           // output pixels
  int pad_w, pad_h;
};
// Tiles of output pixels, and the shares of them whose sums lie apart, [share][group][tap][out][in].
struct RowsWuTiling {
  int tile_w, tile_h, tile_n, pitch;
  size_t x_bytes, smem;
  long tiles;
  int splits;
  float us;
};
// Whether it suits, and how.
bool rowsWuSuits(int sm_count, const RowsWuProblem &p, RowsWuTiling *t);
int launchRowsWu(plb_context *ctx, const RowsWuProblem &p, const RowsWuTiling &t, float *partial);
// Blocks of a share, 64 channels each.
inline int rowsWuSlabs(const RowsWuProblem &p) { return (p.groups * p.chans + 63) / 64; }

}  // namespace plb
