// Which convolutions run on the patch kernel, their tiling and launch.
#include <algorithm>
#include <cmath>

#include "patch.cuh"

namespace plb {

namespace {

struct Tiling {
  int group_block, n_block, tile_w, tile_h, tile_n, patch_w, patch_h, pixel_chunks, mt, nt;
  long tiles;
  size_t table_bytes, pixel_bytes, patch_pixel_bytes, weight_bytes, patch_bytes, smem;
  int stage_pitch, resident;
  float us, us_later;
};

int ceilDiv(long a, long b) { return int((a + b - 1) / b); }

// What all tilings share.
struct Shape {
  int groups, units, weight_chunks, n_total, max_w, max_h, images, planes, chunks[kPatchMaxPhases], first_h, first_w, reach_h, reach_w;
  int es, os;
};

bool shapeOf(const IgemmProblem *p, int n, int type, Shape *s) {
  *s = Shape{};
  s->groups = std::max(1, p->groups);
  s->units = (p->k_per_tap + 7) / 8;
  const int stored = p->taps_stored ? p->taps_stored : p->taps_h * p->taps_w;
  if (stored > 0xffff) return false;
  s->n_total = p->n_total;
  s->images = p->out_n;
  s->planes = type == PLB_FLOAT ? 2 : 1;
  s->es = int(dtypeBytes(type));
  s->os = p->out_f32 ? 4 : 2;
  s->first_h = s->first_w = 1 << 30;
  for (int i = 0; i < n; ++i) {
    s->max_w = std::max(s->max_w, p[i].out_w);
    s->max_h = std::max(s->max_h, p[i].out_h);
    s->chunks[i] = p[i].taps_h * p[i].taps_w * s->units;
    s->weight_chunks += s->chunks[i];
    if (s->chunks[i] == 0) continue;
    s->first_h = std::min(s->first_h, -p[i].pad_h);
    s->first_w = std::min(s->first_w, -p[i].pad_w);
  }
  // (no filter tap reaches any output, or there are no channels: nothing to multiply, and the
  // general route clears the outputs or refuses the layer)
  if (s->weight_chunks == 0) return false;
  for (int i = 0; i < n; ++i) {
    if (s->chunks[i] == 0) continue;
    s->reach_h = std::max(s->reach_h, -p[i].pad_h + (p[i].taps_h - 1) * p[i].dil_h - s->first_h);
    s->reach_w = std::max(s->reach_w, -p[i].pad_w + (p[i].taps_w - 1) * p[i].dil_w - s->first_w);
  }
  if (s->weight_chunks > 8192) return false;
  return s->reach_h < 4096 && s->reach_w < 4096;
}

// Parts of about equal size, none above `most`.
int evenly(int total, int most) { return ceilDiv(total, ceilDiv(total, std::max(1, most))); }

// A tile of about `pixels` output pixels: whole rows, images or parts of rows.
bool setTile(const Shape &s, const IgemmProblem &p, int n, int pixels, Tiling *t) {
  t->tile_w = s.max_w <= std::max(32, pixels / 4) ? std::min(s.max_w, evenly(s.max_w, pixels)) : evenly(s.max_w, std::min(32, pixels));
  t->tile_h = evenly(s.max_h, std::min(s.max_h, std::max(1, pixels / t->tile_w)));
  t->tile_n = t->tile_h == s.max_h && t->tile_w == s.max_w
                  ? evenly(s.images, std::max(1, std::min(s.images, std::min(255, pixels / (t->tile_w * t->tile_h))))) : 1;
  t->patch_w = (t->tile_w - 1) * p.stride_w + s.reach_w + 1;
  t->patch_h = (t->tile_h - 1) * p.stride_h + s.reach_h + 1;
  if (t->patch_w > 4095 || t->patch_h > 4095) return false;
  const size_t patch_pixels = size_t(t->tile_n) * t->patch_w * t->patch_h, m = size_t(t->tile_n) * t->tile_w * t->tile_h;
  t->patch_bytes = patch_pixels * t->pixel_chunks * 16;
  t->pixel_bytes = (m + 63) / 64 * 64 * 8;
  t->patch_pixel_bytes = (patch_pixels * 4 + 15) & ~size_t(15);
  t->tiles = long(ceilDiv(s.max_w, t->tile_w)) * ceilDiv(s.max_h, t->tile_h) * ceilDiv(s.images, t->tile_n);
  // (the last: reads past the last weights)
  t->smem = t->table_bytes + t->pixel_bytes + t->patch_pixel_bytes + s.planes * (t->weight_bytes + t->patch_bytes) +
            size_t(n) * m * t->stage_pitch * s.os + 4096;
  t->resident = std::max(1, std::min(2, int(226 * 1024 / (t->smem + 1024))));
  return t->smem <= 220 * 1024 && t->tiles <= 0x3fffffff;
}

bool tilingOf(int sms, const IgemmProblem *p, int n, int type, bool vec, Tiling *t) {
  Shape s;
  if (!shapeOf(p, n, type, &s)) return false;
  *t = Tiling{};
  t->table_bytes = (size_t(s.weight_chunks) * 8 + 15) & ~size_t(15);
  // groups: as many neighbours as make up 128 bytes of a pixel
  t->n_block = s.n_total <= 64 ? s.n_total : s.n_total % 64 == 0 || s.n_total > 256 ? 64 : evenly(s.n_total, 64) + 7 & ~7;
  const int n8 = ceilDiv(t->n_block, 8);
  const size_t group_weights = size_t(s.weight_chunks) * (p->b_mn ? 8 * (n8 | 1) : 8 * n8) * 16;
  t->group_block = 1;
  if (t->n_block == s.n_total)
    for (int gb = 2; gb <= std::min(s.groups, 16); ++gb)
      if (s.groups % gb == 0 && gb * s.units <= 8 && gb * s.n_total <= 128 && s.planes * gb * group_weights <= 64 * 1024) t->group_block = gb;
  t->weight_bytes = t->group_block * group_weights;
  if (t->group_block * s.units > kPatchThreads / 2) return false;
  if (s.planes * t->weight_bytes > 112 * 1024) return false;
  t->pixel_chunks = (t->group_block * s.units) | 1;
  t->stage_pitch = (t->group_block * t->n_block + 15) / 8 * 8;
  // pixels: 256 to a tile, fewer while that leaves SMs idle or does not fit twice
  const long columns = long(s.groups / t->group_block) * ceilDiv(s.n_total, t->n_block);
  const long pixels = long(s.max_w) * s.max_h * s.images;
  int want = int(std::max<long>(32, std::min<long>(256, pixels * columns / (2 * sms))));
  while (!setTile(s, *p, n, want, t) || (t->resident < 2 && want > 96)) {
    if (want <= 16) return false;
    want = want * 3 / 4;
  }
  const int m = t->tile_w * t->tile_h * t->tile_n;
  t->nt = n8 <= 4 ? n8 : n8 % 4 == 0 ? 4 : n8 % 3 == 0 ? 3 : n8 % 4 == 3 ? 4 : 3;
  // (enough shares for eight warps)
  const int combos = n * t->group_block;
  if (combos * ceilDiv(n8, t->nt) * ceilDiv(m, 32) < kPatchWarps && t->nt > 2) t->nt = 2;
  if (combos * ceilDiv(n8, t->nt) * ceilDiv(m, 32) < kPatchWarps && t->nt > 1) t->nt = 1;
  // (64 pixels an item where that wastes no more than an eighth and leaves enough items)
  t->mt = type != PLB_FLOAT && ceilDiv(m, 64) * 64 * 8 <= 9 * m && combos * ceilDiv(n8, t->nt) * ceilDiv(m, 64) >= kPatchWarps ? 4 : 2;
  const long sets = std::max<long>(1, std::min<long>(t->tiles, long(sms) * t->resident / columns));
  const double rounds = double(ceilDiv(t->tiles, sets)), resident = t->resident;
  const int items = combos * ceilDiv(n8, t->nt) * ceilDiv(m, 16 * t->mt), deep = ceilDiv(items, kPatchWarps);
  const double chunks = double(s.weight_chunks) / n;
  // (an even stride: pixels' rows meet in the same banks)
  const double matrices = (t->mt * (p->stride_w % 2 == 0 ? 2 : 1) + (t->nt == 1 ? 0.5 : ceilDiv(t->nt, 2))) * s.planes * 4, products = t->mt * t->nt * (type == PLB_FLOAT ? 3 : 1) * 2.1;
  const double rate = items * chunks / 2 * std::max(matrices, products) / 1000, latency = deep * chunks / 2 * 0.1;
  // (loads through registers, four of a thread in flight)
  const double loads = vec ? 0 : double(t->tile_n) * t->patch_w * t->patch_h * t->group_block * s.units / 1000;
  const double stores = double(n) * m * t->group_block * t->n_block * s.os / 16000;
  t->us = float(1.6 + 0.0025 * t->group_block * s.weight_chunks * n8 +
                rounds * (2.35 + 0.72 * rate * resident + 0.33 * std::max(latency - rate, 0.0) +
                          1.5 * std::ceil(loads * 1000 / (4 * kPatchThreads)) + (0.45 * loads + 1.2 * stores) * resident));
  // and fitted to ten times as many passes, larger ones among them: with what all blocks fetch
  // of the same weights at once from L2, and as many blocks to an SM as there are
  const bool f = type == PLB_FLOAT;
  const double blocks = double(sets) * columns, weights = double(t->group_block) * s.weight_chunks * n8;
  const double fetched = blocks * weights * 64 * s.es / 1e6, shared = std::min(resident, std::max(1.0, std::ceil(blocks / sms)));
  t->us_later = float((f ? 3.08 + 0.0088 * weights : 1.71 + 0.0046 * weights) + fetched * (p->b_mn ? 0.034 : 0.136) + 0.28 * (shared - 1) +
                      rounds * (1.84 + 0.33 * (n - 1) + (f ? 0.794 : 0.624) * rate * shared + (f ? 1.09 : 0.49) * std::max(latency - rate, 0.0) +
                                1.84 * std::ceil(loads * 1000 / (4 * kPatchThreads)) + (0.22 * loads + 1.34 * stores) * shared));
  return true;
}

bool wholeLoads(const IgemmProblem &p, int type) {
  const uint64_t load = type == PLB_QUARTER ? 8 : 16;
  uint64_t at = reinterpret_cast<uintptr_t>(p.act) | p.act_strides[0];
  if (p.act_dims[2] > 1) at |= p.act_strides[1];
  if (p.out_n > 1) at |= p.act_strides[2];
  if (p.groups > 1) at |= p.act_group_stride;
  return at % load == 0;
}

bool patchable(const IgemmProblem *p, int n, int type) {
  if (n < 1 || n > kPatchMaxPhases || p->a_mn || p->plan_flags != 0 || p->force_tile_n != 0 || p->force_split_k != 0) return false;
  if (type != PLB_HALF && type != PLB_FLOAT && type != PLB_QUARTER) return false;
  if (p->beta != 0.f) return false;
  const uint64_t limit = 0x3fffffffull;
  for (int i = 0; i < n; ++i) {
    if (uint64_t(p[i].out_w) * p[i].out_h * p[i].out_n > limit || p[i].out_n <= 0) return false;
    if (p[i].dil_h > 1024 || p[i].dil_w > 1024 || p[i].taps_h > 1024 || p[i].taps_w > 1024) return false;
    if (std::abs(p[i].pad_h) > 4096 || std::abs(p[i].pad_w) > 4096) return false;
  }
  if (p->stride_h > 64 || p->stride_w > 64 || p->out_w > 1 << 20 || p->out_h > 1 << 20) return false;
  if (p->act_strides[0] * p->act_dims[1] > limit || p->act_strides[1] * p->act_dims[2] > limit) return false;
  if (p->groups > 1 && p->out_group_stride != p->n_total) return false;
  return true;
}

}  // namespace

// Layers whose time on the patch kernel, as tilingOf estimates it (fitted to 478 passes of
// small and grouped layers of every type, median error 11 %), is below what the general route
// takes at least, less a sixteenth: 3.6 us, 2.4 for each launch besides the contraction (block-diagonal
// weights, repair, copies, phases of a strided layer), and the tensor-core steps of the
// groups contracted together (`packed`: of all taps of a row together).  Of the 478 it takes
// 127, which run in 0.59 of their time, two of them slower (by 6 and 11 %; 3x3, 2 groups of 8,
// 3 images of 14 x 95 8.5 -> 4.4 us; 3x3/2, 32 groups of 8, 2 of 8 x 108, input gradient 20.6 ->
// 9.3); ungrouped layers that are one launch stay (56 x 56, 64 channels: 5.3 against 11.2).
// Groups of 8 and 16 that the row kernel takes (rows.cu) are not estimated.
// Unless the general route packs its operand rows, both times are estimated once more, fitted to
// 4200 passes (median errors 7 and 8 %, a tenth of them 20 and 23 %): of 1800 that the first
// estimates took, 103 were more than 8 % slower than on the general route, up to 1.7 times; the second
// leave 26 of those, and give up 22 that gain (3x3, 2 groups of 32, 42 images of 13 x 13, where 294 blocks
// wait for the same weights, 13.0 -> 7.5 us; 1x1, 2 groups of 32, 8 of 35 x 35 8.8 -> 5.6).
bool patchSuits(int sm_count, const IgemmProblem *p, int n, int type, int contractions, int together, bool copied, bool packed,
                bool slower_too, RowsTiling *rows) {
  rows->blocks = 0;
  if (!patchable(p, n, type)) return false;
  if (n == 1 && rowsSuits(sm_count, *p, type, rows)) return true;
  rows->blocks = 0;
  const double operand = (type == PLB_FLOAT ? 6.0 : type == PLB_QUARTER ? 1.0 : 2.0) * together * p->k_per_tap;
  const double columns = double(together) * p->n_total, wide = columns <= 64 ? 1 : columns <= 128 ? 1.6 : 2.6;
  const double tile_n = columns <= 64 ? 64 : columns <= 128 ? 128 : 256;
  double steps = 0, tiles = 0;
  bool several_taps = false;
  for (int i = 0; i < n; ++i) {
    const double pixels = std::ceil(double(p[i].out_w) * p[i].out_h * p[i].out_n / 128);
    tiles += pixels;
    steps += pixels * p[i].taps_h * (packed ? std::ceil(operand * p[i].taps_w / 128) : p[i].taps_w * std::ceil(operand / 128));
    several_taps |= p[i].taps_h * p[i].taps_w > 1;
  }
  const double waves = std::ceil(columns / tile_n) * std::max(1, p->groups) / together / sm_count;
  steps *= wide * waves;
  const int launches = contractions + (together > 1 ? 2 : 0) + (copied ? 1 : 0);
  const float general = float(3.4 + 2.25 * (launches - 1) + 0.134 * steps);
  // a contraction and further ones, steps and tiles, of which a device's first few cost most;
  // block-diagonal weights and repair; copies
  tiles = std::max(0.0, tiles * waves - 0.5);
  double later = 2.37 + 3.54 * (contractions - 1) + 0.166 * steps + 0.116 * std::min(steps, 20.0) + 0.17 * tiles + 0.8 * std::min(tiles, 4.0);
  if (together > 1) {
    const int stored = p->taps_stored ? p->taps_stored : p->taps_h * p->taps_w;
    later += 3.11 + (several_taps ? 1.68 : 0) + 3.81e-6 * p->groups * stored * double(p->k_per_tap) * p->n_total * together * dtypeBytes(type);
  }
  if (copied)
    later += type == PLB_FLOAT ? 3.44 + 0.16e-6 * double(p->act_strides[2]) * p->out_n : type == PLB_QUARTER ? 1.92 : 2.72;
  Tiling t;
  // (no tiling takes less than 4 us)
  return general > 4.0f && tilingOf(sm_count, p, n, type, wholeLoads(*p, type), &t) && t.us < general &&
         (packed || slower_too || t.us_later < 0.98 * later);
}

int launchPatch(plb_context *ctx, const IgemmProblem *p, int n, int type, bool repair) {
  Tiling t;
  const bool act_vec = wholeLoads(*p, type);
  if (!tilingOf(ctx->sm_count, p, n, type, act_vec, &t)) return fail(PLB_ERR_UNSUPPORTED, "no tiling of the patch kernel");
  Shape s;
  shapeOf(p, n, type, &s);
  PatchArgs g{};
  g.act = static_cast<const uint8_t *>(p->act);
  g.wgt = static_cast<const uint8_t *>(p->wgt);
  g.act_n = (long long)p->act_strides[2];
  g.act_group = s.groups > 1 ? (long long)p->act_group_stride : 0;
  g.wgt_tile = (long long)p->wgt_strides[1];
  g.wgt_row = (long long)p->wgt_strides[0];
  g.act_w = int(p->act_strides[0]);
  g.act_h = p->act_dims[2] > 1 ? int(p->act_strides[1]) : 0;
  g.in_w = int(p->act_dims[1]);
  g.in_h = int(p->act_dims[2]);
  g.images = p->out_n;
  g.stride_h = p->stride_h;
  g.stride_w = p->stride_w;
  g.k = p->k_per_tap;
  g.n_total = p->n_total;
  g.groups = s.groups;
  g.taps_stored = p->taps_stored ? p->taps_stored : p->taps_h * p->taps_w;
  g.units = s.units;
  g.group_block = t.group_block;
  const int group_blocks = s.groups / t.group_block;
  g.n_block = t.n_block;
  g.n_blocks = ceilDiv(s.n_total, t.n_block);
  g.tile_w = t.tile_w;
  g.tile_h = t.tile_h;
  g.tile_n = t.tile_n;
  g.tiles_w = ceilDiv(s.max_w, t.tile_w);
  g.tiles_h = ceilDiv(s.max_h, t.tile_h);
  g.tiles = int(t.tiles);
  g.patch_w = t.patch_w;
  g.patch_h = t.patch_h;
  g.pixel_chunks = t.pixel_chunks;
  g.first_h = s.first_h;
  g.first_w = s.first_w;
  g.m = t.tile_w * t.tile_h * t.tile_n;
  g.m_chunks = ceilDiv(g.m, 16 * t.mt);
  const int n8 = ceilDiv(t.n_block, 8);
  g.n_parts = ceilDiv(n8, t.nt);
  g.weight_chunks = s.weight_chunks;
  g.weight_row = n8 | 1;
  g.at_pixels = int(t.table_bytes);
  g.at_patch_pixels = int(t.table_bytes + t.pixel_bytes);
  g.at_weights = int(t.table_bytes + t.pixel_bytes + t.patch_pixel_bytes);
  g.patch_pixels = t.tile_n * t.patch_w * t.patch_h;
  g.weight_bytes = int(t.weight_bytes);
  g.patch_bytes = int(t.patch_bytes);
  g.stage_pitch = t.stage_pitch;
  g.fd_units = make_fastdiv(uint32_t(s.units));
  g.fd_patch_w = make_fastdiv(uint32_t(t.patch_w));
  g.fd_patch_h = make_fastdiv(uint32_t(t.patch_h));
  g.fd_tile_w = make_fastdiv(uint32_t(t.tile_w));
  g.fd_tile_h = make_fastdiv(uint32_t(t.tile_h));
  g.fd_tiles_w = make_fastdiv(uint32_t(g.tiles_w));
  g.fd_tiles_h = make_fastdiv(uint32_t(g.tiles_h));
  g.fd_group_weights = make_fastdiv(uint32_t(s.weight_chunks * n8 * 8));
  g.fd_chunk_weights = make_fastdiv(uint32_t(n8 * 8));
  g.fd_weight_cols = make_fastdiv(uint32_t(n8));
  g.blocks_per_set = group_blocks * g.n_blocks;
  g.fd_blocks = make_fastdiv(uint32_t(g.blocks_per_set));
  g.act_vec = act_vec;
  g.wgt_vec = (reinterpret_cast<uintptr_t>(p->wgt) | p->wgt_strides[0] | p->wgt_strides[1]) % 16 == 0;
  g.fmt_a = p->fmt_a;
  g.fmt_b = p->fmt_b;
  g.out = p->out;
  g.ldc = p->ldc;
  g.out_h = p->out_stride_h ? p->out_stride_h : (long long)p->out_w * p->ldc;
  g.out_n = p->out_stride_n ? p->out_stride_n : (long long)p->out_h * p->out_w * p->ldc;
  g.out_group = s.groups > 1 ? p->out_group_stride : 0;
  g.bias = p->bias;
  g.alpha = p->alpha;
  g.out_f32 = p->out_f32 ? 1 : 0;
  g.repair = repair ? 1 : 0;
  g.phases = n;
  // a pixel's run of channels in one block: all its groups', or a part of one group's
  uint64_t run = uint64_t(t.group_block) * t.n_block * s.os, at = uint64_t(g.ldc | g.out_h | g.out_n) * s.os | run;
  if (group_blocks > 1) at |= uint64_t(t.group_block) * uint64_t(g.out_group) * s.os;
  if (g.n_blocks > 1) at |= uint64_t(s.n_total % t.n_block) * s.os;
  int table = 0;
  for (int i = 0; i < n; ++i) {
    const IgemmProblem &q = p[i];
    PatchPhase &ph = g.phase[i];
    ph.out_w = q.out_w;
    ph.out_h = q.out_h;
    ph.taps_h = q.taps_h;
    ph.taps_w = std::max(1, q.taps_w);
    ph.dil_h = q.dil_h;
    ph.dil_w = q.dil_w;
    ph.pad_h = q.pad_h;
    ph.pad_w = q.pad_w;
    ph.row0 = -q.pad_h - s.first_h;
    ph.col0 = -q.pad_w - s.first_w;
    const int pitch = q.tap_pitch_h ? q.tap_pitch_h : q.taps_w;
    ph.tap_first = (q.tap_first_h + (q.flip_h ? (q.taps_h - 1) * q.tap_step_h : 0)) * pitch + q.tap_first_w +
                   (q.flip_w ? (q.taps_w - 1) * q.tap_step_w : 0);
    ph.tap_step_h = (q.flip_h ? -q.tap_step_h : q.tap_step_h) * pitch;
    ph.tap_step_w = q.flip_w ? -q.tap_step_w : q.tap_step_w;
    ph.table = table;
    ph.chunks = s.chunks[i];
    table += s.chunks[i];
    ph.out = (static_cast<const uint8_t *>(q.out) - static_cast<const uint8_t *>(p->out)) / (long long)s.os;
    at |= reinterpret_cast<uintptr_t>(q.out);
  }
  g.run_vec = at % 16 == 0 ? 16 : at % 8 == 0 ? 8 : at % 4 == 0 ? 4 : 2;
  PatchVariant v{};
  v.b_mn = p->b_mn;
  v.mt = t.mt;
  v.nt = t.nt;
  v.smem = t.smem;
  const long sets = std::max<long>(1, std::min<long>(t.tiles, long(ctx->sm_count) * t.resident / g.blocks_per_set));
  v.grid = unsigned(sets * g.blocks_per_set);
  switch (type) {
    case PLB_FLOAT: return launchPatchFloat(ctx, v, g);
    case PLB_QUARTER: return launchPatchQuarter(ctx, v, g);
    default: return launchPatchHalf(ctx, v, g);
  }
}

}  // namespace plb
