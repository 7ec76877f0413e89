// Planning and launch of the implicit-GEMM kernel: CTA tile selection, pixel
// box selection, TMA tensor maps.  This replaces, for the GPU, the search the
// reference's planner does over IPU tile partitions
// (lib/poplin/ConvPlan.cpp:1100-1224, 1674-1768): the quantities chosen here
// are the CTA tile (128 pixels x 64/128/256 channels), the pixel box that makes
// up the 128 rows, the pipeline depth and the number of persistent CTAs.
#include "igemm_dispatch.cuh"
#include "igemm_sm100.cuh"
#include "runtime.h"

#include <algorithm>
#include <cstdlib>
#include <cstring>

namespace plb {

namespace {

int stagesFor(int bn, int a_stage_bytes, int b_tiles, bool resident, int resident_bytes,
              bool pair) {
  const int a = a_stage_bytes;
#define PLB_STAGES(BN)                                                                         \
  return resident ? (pair ? IgemmSmem<BN, true, true>::stagesFor(a, b_tiles, resident_bytes)   \
                          : IgemmSmem<BN, true, false>::stagesFor(a, b_tiles, resident_bytes)) \
                  : (pair ? IgemmSmem<BN, false, true>::stagesFor(a, b_tiles, 0)               \
                          : IgemmSmem<BN, false, false>::stagesFor(a, b_tiles, 0));
  switch (bn) {
    case 64: PLB_STAGES(64)
    case 128: PLB_STAGES(128)
    default: PLB_STAGES(256)
  }
#undef PLB_STAGES
}

// Weights stay in shared memory when one N tile covers all output channels,
// every CTA gets several pixel tiles to amortise the load over, and the
// weights leave room for a pipeline of at least six activation stages.
constexpr int kMaxResidentBytes = 96 * 1024;
// Groups beside which a grid that is a multiple of their number still fills the device.
constexpr int kMaxResidentGroups = 16;
// Bytes that all CTAs together may ask for at their start.
constexpr long kMostFirstBytes = 16L << 20;

}  // namespace

int planIgemm(const IgemmProblem &p, int sm_count, plb_plan *plan) {
  const int elem = p.fp8 ? 1 : 2;
  if (p.n_total <= 0 || p.out_w <= 0 || p.out_h <= 0 || p.out_n <= 0 || p.k_per_tap <= 0)
    return fail(PLB_ERR_INVALID_PARAMS, "empty contraction reached the kernel planner");
  if (p.fp8 && p.b_mn)
    return fail(PLB_ERR_UNSUPPORTED, "MN-major right operand is only implemented for half");
  if (p.a_mn && (p.fp8 || p.taps_h * p.taps_w != 1 || p.out_h != 1 || p.out_n != 1))
    return fail(PLB_ERR_UNSUPPORTED, "a transposed left operand is only implemented for half matrix products");
  const long groups = std::max(1, p.groups);
  // ---- N tile ---------------------------------------------------------------
  // Cost model: waves of tiles over the SMs times the measured duration of a
  // 128 x BN x 16 tensor-core instruction (operand fetch bound: 75 / 95 / 155
  // cycles for BN = 64 / 128 / 256).  Wide tiles win whenever the grid fills
  // the device; a grid of a few tiles (small matrix products) finishes sooner
  // with narrow ones, which also spread it over more SMs.
  int bn = 0;
  if (p.force_tile_n) {
    bn = p.force_tile_n;
    if (bn != 64 && bn != 128 && bn != 256)
      return fail(PLB_ERR_INVALID_OPTION, "tile_n must be 64, 128 or 256");
  } else {
    const long sms = sm_count > 0 ? sm_count : 148;
    const long pixel_tiles = (long(p.out_w) * p.out_h * p.out_n + kTileM - 1) / kTileM;  // lower bound
    long best = -1;
    for (int cand : {256, 128, 64}) {
      const long n_tiles_c = (p.n_total + cand - 1) / cand;
      const long waves = (pixel_tiles * n_tiles_c * groups + sms - 1) / sms;
      const long cost = waves * (cand == 256 ? 155 : cand == 128 ? 95 : 75);
      if (best < 0 || cost < best) {
        best = cost;
        bn = cand;
      }
    }
  }
  // ---- pixel box: bw*bh*bn == 128, fewest tiles, then widest rows ------------
  int bw = 0, bh = 0, bb = 0;
  long best_tiles = -1;
  for (int w = 128; w >= 1; w >>= 1)
    for (int h = 128 / w; h >= 1; h >>= 1) {
      const int n = 128 / (w * h);
      if ((w - 1) * p.stride_w + 1 > 256 || (h - 1) * p.stride_h + 1 > 256) continue;
      const long tiles = long((p.out_w + w - 1) / w) * ((p.out_h + h - 1) / h) *
                         ((p.out_n + n - 1) / n);
      if (best_tiles < 0 || tiles < best_tiles) {
        best_tiles = tiles;
        bw = w;
        bh = h;
        bb = n;
      }
    }
  const int n_tiles = (p.n_total + bn - 1) / bn;
  if (best_tiles * n_tiles * groups > 0x7fffffffL)
    return fail(PLB_ERR_UNSUPPORTED, "too many output tiles for one launch");
  plan->kernel = 0;
  plan->tile_m = kTileM;
  plan->tile_n = bn;
  plan->tile_k_bytes = kStageKBytes;
  plan->box_w = bw;
  plan->box_h = bh;
  plan->box_n = bb;
  plan->split_k = 1;
  plan->tiles = int(best_tiles * n_tiles * groups);
  // CTA pairs: two M tiles share one 256-row MMA, each CTA holding half of the
  // weight tile.  Needs two M tiles and, for a row-major B, a whole 64-column
  // block per CTA.
  // Worth it, with a K loop that is not short, when every CTA pair gets several tile
  // pairs: the two SMs advance in lockstep per tile, which costs short tiles more than the
  // halved weight traffic saves.  With 256-column tiles the weight tile is two thirds of a
  // stage's bytes and half the K length already pays (1x1 stride-2 layer 256 -> 512: 71 ->
  // 67 us).  With fewer tiles, as long as the pairs need no wave more:
  //  - filters of several rows: half the weights also make room for a halo strip, which a
  //    vertical stride has not (3x3/2, 392 channels, 2 images of 59x59: 22.7 -> 24.2)
  //    (3x3, 208 channels, 2 images of 76x76, 95 tiles: 20.6 -> 16.7 us; 3x3, 96 -> 176,
  //    4 images of 29x20, 60 tiles: 7.2 -> 6.3); not short tiles of 64 columns in a second
  //    wave that is mostly empty (3x3, 48 channels, 42 images of 8x84, 231 tiles: 8.7 -> 9.2;
  //    11 sampled layers 5 % slower);
  //  - more than a wave of wide tiles, whatever the taps, stride and groups: products
  //    (2048 x 4096 x 4096, 256 tiles: 65 -> 60 us), strided filters (3x3/2, 128 channels, 32
  //    images of 56x56, 196 tiles: 13.0 -> 12.0; 256 channels, 12 of 56x56, 168 tiles: 17.4 ->
  //    16.5), groups (3x3, 2 groups of 128, 12 of 28x28, 168 tiles: 11.4 -> 9.2); 63 sampled
  //    strided and grouped layers 0.86 of their time, one 5 % longer;
  //  - wide tiles whose rows start at odd multiples of 16 bytes, which take the copy engine
  //    longer (1500 x 3000 x 3000, 144 tiles: 39 -> 31 us; with whole lines, 2238 x 1216 x
  //    1792, 126 tiles: 11.2 -> 11.9).
  const int k_elems_stage = kStageKBytes / elem;
  const int taps = p.taps_h * p.taps_w;
  const long k_steps_per_tile = long(taps) * ((p.k_per_tap + k_elems_stage - 1) / k_elems_stage);
  const long sms_for_pair = sm_count > 0 ? sm_count : 148;
  const long units_single = best_tiles * n_tiles * groups, units_pair = (best_tiles + 1) / 2 * n_tiles * groups;
  const bool no_more_waves = (units_pair + sms_for_pair / 2 - 1) / (sms_for_pair / 2) <= (units_single + sms_for_pair - 1) / sms_for_pair;
  const bool odd_rows = p.act_strides[0] % 32 != 0 || p.wgt_strides[0] % 32 != 0;
  const bool several_taps = p.taps_h > 1 && p.stride_h == 1 && groups == 1 && k_steps_per_tile >= 8 && units_single >= 48 &&
                            !(bn <= 64 && k_steps_per_tile < 16 && units_single > sms_for_pair);
  const bool wide_tiles = bn >= 128 && k_steps_per_tile >= 7 &&
                          (units_single > sms_for_pair || (odd_rows && 2 * units_single >= sms_for_pair));
  const bool pair = (p.plan_flags & PLB_PLAN_NO_CTA_PAIR) == 0 && (!p.b_mn || bn >= 128) &&
                    ((p.plan_flags & PLB_PLAN_FORCE_CTA_PAIR) != 0
                         ? best_tiles >= 2
                         : (k_steps_per_tile >= (bn >= 256 ? 4 : 8) && units_single >= 2 * sms_for_pair) ||
                               (best_tiles >= 2 && no_more_waves && (several_taps || wide_tiles)));
  plan->cta_pair = pair ? 1 : 0;
  auto grid_for = [&](long m_tiles) {
    const int sms = sm_count > 0 ? sm_count : 148;
    // (with resident weights a CTA, or pair, keeps to one group)
    const long units = pair ? std::min<long>(((m_tiles + 1) / 2) * n_tiles * groups, sms / 2)
                            : std::min<long>(m_tiles * n_tiles * groups, sms);
    return int((pair ? 2 : 1) * (plan->resident_weights ? units / groups * groups : units));
  };
  plan->resident_weights = 0;
  plan->grid = grid_for(best_tiles);
  const int k_elems = kStageKBytes / elem;
  const long k_iters = long(p.taps_h) * p.taps_w * ((p.k_per_tap + k_elems - 1) / k_elems);
  // per CTA
  const long resident_bytes = k_iters * (bn / (pair ? 2 : 1)) * kStageKBytes;
  const bool force_resident = (p.plan_flags & PLB_PLAN_FORCE_RESIDENT_WEIGHTS) != 0;
  const bool want_resident = force_resident || plan->tiles >= 2 * plan->grid;
  // With several groups a CTA (pair) works on one of them alone: as many as can run
  // side by side if residency is asked for, and no K splits, which are neighbouring
  // units (a tile's splits would be different groups' units to the CTAs).
  const long side_by_side = pair ? sms_for_pair / 2 : sms_for_pair;
  const long most_groups = force_resident ? side_by_side : std::min<long>(kMaxResidentGroups, side_by_side);
  plan->resident_weights =
      ((p.plan_flags & PLB_PLAN_NO_RESIDENT_WEIGHTS) == 0 && n_tiles == 1 && groups <= most_groups && !p.a_mn &&
       (groups == 1 || p.force_split_k <= 1) && resident_bytes <= kMaxResidentBytes && want_resident)
          ? 1
          : 0;
  plan->grid = grid_for(best_tiles);
  plan->halo_rows = 0;
  plan->stages = stagesFor(bn, kTileM * kStageKBytes, 1, plan->resident_weights != 0,
                           plan->resident_weights ? int(resident_bytes) : 0, pair);
  // Halo mode: with resident weights and a filter taller than one row (unit
  // vertical stride), load (box_h + halo) input rows once per horizontal tap
  // instead of box_h rows per tap.  The tile rows are ordered (w, n, h) so that
  // a vertical shift is a whole number of 8-row groups: box_w * box_n % 8 == 0.
  const int halo = (p.taps_h - 1) * p.dil_h;
  if ((p.plan_flags & PLB_PLAN_NO_HALO) == 0 && p.taps_h > 1 &&
      p.stride_h == 1) {
    // Shared-memory fill per pixel tile and channel chunk, the quantity that
    // bounds a layer whose tensor-core work is short: activation rows plus,
    // unless the weights are resident, one weight tile per filter tap.
    const bool res = plan->resident_weights != 0;
    const long b_tile = res ? 0 : long(bn / (pair ? 2 : 1)) * kStageKBytes;
    const long base_cost =
        best_tiles * p.taps_h * p.taps_w * (long(kTileM) * kStageKBytes + b_tile);
    long best_cost = -1, best_t = -1;
    int hw = 0, hh = 0, hn = 0;
    for (int w = 128; w >= 1; w >>= 1)
      for (int n = 128 / w; n >= 1; n >>= 1) {
        const int h = 128 / (w * n);
        if ((w * n) % 8 != 0 || h + halo > 256 || (w - 1) * p.stride_w + 1 > 256) continue;
        const long tiles = long((p.out_w + w - 1) / w) * ((p.out_h + h - 1) / h) *
                           ((p.out_n + n - 1) / n);
        // without much more tensor-core work (padded tiles)
        if (tiles * 8 > best_tiles * 9) continue;
        const long cost =
            tiles * p.taps_w * (long(w) * n * (h + halo) * kStageKBytes + p.taps_h * b_tile);
        if (best_cost < 0 || cost < best_cost || (cost == best_cost && tiles < best_t)) {
          best_cost = cost;
          best_t = tiles;
          hw = w;
          hh = h;
          hn = n;
        }
      }
    if (best_cost > 0) {
      const int a_stage = hw * hn * (hh + halo) * kStageKBytes;
      const int st = stagesFor(bn, a_stage, res ? 1 : p.taps_h, res, res ? int(resident_bytes) : 0,
                               pair);
      // worthwhile only if it really fills less and still leaves a pipeline
      if (st >= 3 && best_cost < base_cost) {
        plan->halo_rows = halo;
        plan->box_w = hw;
        plan->box_h = hh;
        plan->box_n = hn;
        plan->stages = st;
        plan->tiles = int(best_t * n_tiles * groups);
        plan->grid = grid_for(best_t);
      }
    }
  }
  plan->b_mn_major = p.b_mn ? 1 : 0;
  plan->workspace_bytes = 0;
  // ---- split-K ---------------------------------------------------------------
  // A product with few output tiles and a long reduction leaves most SMs idle:
  // let several CTAs share a tile, each taking a range of its pipeline steps,
  // and add their fp32 partial sums in a second kernel.  Model (microseconds): a
  // pipeline step of one CTA takes about 0.15 per weight tile that it streams, more
  // where an operand's rows begin at odd multiples of 16 bytes (0.24 for a left operand
  // of 1800 columns, 0.28 with a right one of 200 too: such rows are copied in more,
  // partly filled sectors); the second kernel 3.4 plus the partial sums written and read at 4 TB/s (MB per
  // microsecond below); the split must save more than it costs.  From sweeps of long
  // products and of small images: 128 x 2048 x 64 splits (8.3 -> 7.0 us), so do 3x3
  // layers of 256 and 512 channels on one 14 x 14 image (8.6 -> 7.5, 13.7 -> 9.3);
  // 512 x 1024 x 1024 and 256 channels on four such images stay whole (6.1 against
  // 7.8, 8.7 against 9.7).
  {
    const long units = plan->tiles / (pair ? 2 : 1) + (pair ? plan->tiles % 2 : 0);
    const long steps = plan->halo_rows > 0 ? long(p.taps_w) * ((p.k_per_tap + k_elems - 1) / k_elems)
                                           : k_iters;
    const long sms = sm_count > 0 ? sm_count : 148;
    const int b_tiles = plan->halo_rows > 0 && !plan->resident_weights ? p.taps_h : 1;
    // The cheapest split of `tiles` units of work, at most one per SM or (pairs) two per
    // pair of SMs.
    auto cheapest = [&](long tiles) {
      if (tiles * 2 > sms || steps * b_tiles < 20 || (plan->resident_weights && groups > 1)) return 1;
      int split = 1;
      const double out_mb = double(groups) * p.out_w * p.out_h * p.out_n * p.n_total * 4 / 1e6;
      const double odd_rows = (p.act_strides[0] % 32 != 0 ? 0.09 : 0.0) + (p.wgt_strides[0] % 32 != 0 ? 0.045 : 0.0);
      const double step_us = 0.15 * b_tiles + odd_rows;
      double best = step_us * double(steps);
      for (long sp = 2; sp <= std::min<long>(steps * b_tiles / 4, std::min(steps, sms / tiles)); ++sp) {
        const double t = step_us * double((steps + sp - 1) / sp) + 3.4 + out_mb * double(sp + 1) / 4.0;
        if (t < best) {
          best = t;
          split = int(sp);
        }
      }
      return split;
    };
    // Pairs are split where their tiles would be on single SMs.  There they run in up to
    // two waves and are quicker for it (3x3, 512 channels, one 28 x 28 image, 28 pairs:
    // 5 splits 12.7 us, 2 splits 14.0, unpaired 13.0).  Elsewhere the second wave, the
    // partial sums and the second kernel cost more than the shorter ranges save (5x5, 304 -> 368
    // channels, 11 images of 16 x 16, 66 pairs: 2 splits 23.4 us, whole 17.5, unpaired 20.7;
    // 180 sampled passes 0.92 of their time with every pair split as the model has it, 0.85
    // of it unpaired).  A few would still gain (5x5, 499 -> 308, 3 of 20 x 20, 38 pairs:
    // 3 splits 26.5, whole 30.9, unpaired 36.5), but take no scratch this way.
    int split = 1;
    if (p.force_split_k > 0)
      split = int(std::min<long>(p.force_split_k, steps));
    else if (!pair || cheapest(plan->tiles) > 1)
      split = cheapest(units);
    if (split > 1 && long(plan->tiles) * split > 0x3fffffffL) split = 1;
    plan->split_k = split;
    if (split > 1) {
      const long units_total = units * split;
      plan->grid = pair ? int(2 * std::min<long>(units_total, sms / 2)) : int(std::min<long>(units_total, sms));
      const size_t ld_p = (size_t(p.n_total) + 31) / 32 * 32;
      plan->workspace_bytes = uint64_t(split) * groups * p.out_w * p.out_h * p.out_n * ld_p * sizeof(float);
    }
  }
  return PLB_OK;
}

namespace {

// Second kernel of a split-K product: adds the splits' partial sums in split
// order (a fixed order, so the result does not depend on timing) and applies
// what the implicit-GEMM kernel's own epilogue would have: alpha, bias, the
// beta-scaled addend, the cast.  One thread per four consecutive channels of
// one output pixel.
struct SplitKReduceArgs {
  const float *partial;
  int split_k;
  long long split_stride;  // elements between splits
  int ld_p;                // elements between pixels in the partial sums
  int groups, n_total, out_w, out_h, out_n;
  void *out;
  long long ldc, out_stride_h, out_stride_n, out_group_stride;
  const void *addend;
  long long ld_addend, addend_group_stride;
  const float *bias;
  float alpha, beta;
  int out_is_f32;
};

__global__ void __launch_bounds__(256) igemm_splitk_reduce_kernel(const SplitKReduceArgs a) {
  pdl_launch_dependents();
  pdl_wait();  // the partial sums come from the previous kernel in the stream
  const int quads = (a.n_total + 3) / 4;
  const long long pixels = (long long)a.out_w * a.out_h * a.out_n;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < a.groups * pixels * quads;
       i += (long long)gridDim.x * blockDim.x) {
    const long long row = i / quads, g = row / pixels, pixel = row - g * pixels;
    const int c = int(i - row * quads) * 4;
    const float *src = a.partial + row * a.ld_p + c;
    float4 s = *reinterpret_cast<const float4 *>(src);
    for (int k = 1; k < a.split_k; ++k) {
      const float4 v = *reinterpret_cast<const float4 *>(src + k * a.split_stride);
      s.x += v.x;
      s.y += v.y;
      s.z += v.z;
      s.w += v.w;
    }
    float f[4] = {s.x, s.y, s.z, s.w};
    const int valid = min(4, a.n_total - c);
    if (a.alpha != 1.f)
      for (int j = 0; j < 4; ++j) f[j] *= a.alpha;
    if (a.bias != nullptr)
      for (int j = 0; j < valid; ++j) f[j] += a.bias[g * a.n_total + c + j];
    if (a.addend != nullptr) {
      if (a.out_is_f32) {
        const float *ad = static_cast<const float *>(a.addend) + g * a.addend_group_stride + pixel * a.ld_addend + c;
        for (int j = 0; j < valid; ++j) f[j] += a.beta * ad[j];
      } else {
        const __half *ad = static_cast<const __half *>(a.addend) + g * a.addend_group_stride + pixel * a.ld_addend + c;
        for (int j = 0; j < valid; ++j) f[j] += a.beta * __half2float(ad[j]);
      }
    }
    const long long ow = pixel % a.out_w, rest = pixel / a.out_w;
    const long long oh = rest % a.out_h, on = rest / a.out_h;
    const long long off = g * a.out_group_stride + on * a.out_stride_n + oh * a.out_stride_h + ow * a.ldc + c;
    if (a.out_is_f32) {
      float *dst = static_cast<float *>(a.out) + off;
      if (valid == 4 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0)
        *reinterpret_cast<float4 *>(dst) = make_float4(f[0], f[1], f[2], f[3]);
      else
        for (int j = 0; j < valid; ++j) dst[j] = f[j];
    } else {
      __half *dst = static_cast<__half *>(a.out) + off;
      if (valid == 4 && (reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
        const __half2 lo = __floats2half2_rn(f[0], f[1]), hi = __floats2half2_rn(f[2], f[3]);
        *reinterpret_cast<uint2 *>(dst) = make_uint2(*reinterpret_cast<const uint32_t *>(&lo),
                                                     *reinterpret_cast<const uint32_t *>(&hi));
      } else {
        for (int j = 0; j < valid; ++j) dst[j] = __float2half_rn(f[j]);
      }
    }
  }
}

}  // namespace

int launchIgemm(plb_context *ctx, const IgemmProblem &p, const plb_plan &plan) {
  const int elem = p.fp8 ? 1 : 2;
  const int k_elems_per_stage = kStageKBytes / elem;
  const CUtensorMapDataType dt =
      p.fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;

  const bool halo = plan.halo_rows > 0;
  // In halo mode the pixel dimensions are ordered (w, n, h) in every tensor map.
  auto order = [&](uint64_t w, uint64_t h, uint64_t n, uint64_t *out3) {
    out3[0] = w;
    out3[1] = halo ? n : h;
    out3[2] = halo ? h : n;
  };
  const int groups = std::max(1, p.groups);
  // The kernel instance for groups, also taken where a short K (one chunk, not
  // full) saves instructions on every tile.  Its copies and stores carry the group
  // coordinate whatever the number of groups, so the tensor maps of activations
  // and output must have the dimension.
  const int k_chunks = (p.k_per_tap + k_elems_per_stage - 1) / k_elems_per_stage;
  const int k_elems_mma = 32 / elem;
  const int k_last = (p.k_per_tap - (k_chunks - 1) * k_elems_per_stage + k_elems_mma - 1) / k_elems_mma;
  const bool with_groups =
      groups > 1 || (!plan.resident_weights && k_chunks == 1 && k_last < 4 && p.taps_h * p.taps_w > 1);
  // Rows of an activation box.  A single tile along the slowest dimension of the
  // box loads only what the output needs of it: a product of 16 rows would
  // otherwise spend most of its copy time filling 112 rows with zeros.  (What the
  // unused rows of shared memory hold reaches unused accumulator rows alone.)
  int load_w = plan.box_w, load_h = plan.box_h, load_n = plan.box_n;
  if (!plan.cta_pair) {
    int *slowest = halo ? (load_h > 1 ? &load_h : load_n > 1 ? &load_n : &load_w)
                        : (load_n > 1 ? &load_n : load_h > 1 ? &load_h : &load_w);
    *slowest = std::min(*slowest, slowest == &load_w ? p.out_w : slowest == &load_h ? p.out_h : p.out_n);
  }
  const int a_blocks = p.a_mn ? (load_w + 63) / 64 : 0;
  CUtensorMap ta, tb;
  if (p.a_mn) {
    // [group][k][m], rows of m: boxes of 64 K rows x 64 output rows
    const uint64_t dims[3] = {p.act_dims[1], p.act_dims[0], uint64_t(groups)};
    const uint64_t strides[2] = {p.act_strides[0], groups > 1 ? uint64_t(p.act_group_stride) : p.act_strides[1]};
    const uint32_t box[3] = {64, 64, 1}, es[3] = {1, 1, 1};
    if (int rc = encodeTensorMap(&ta, dt, 3, p.act, dims, strides, box, es)) return rc;
  } else {
    // (k, w, h, n), with groups (k, group, w, h, n)
    uint64_t dims[5] = {p.act_dims[0]}, strides[4], b3[3], e3[3];
    uint32_t box[5] = {uint32_t(k_elems_per_stage)}, es[5] = {1};
    int rank = 1;
    if (with_groups) {
      dims[1] = uint64_t(groups);
      strides[0] = groups > 1 ? p.act_group_stride : p.act_strides[0];
      box[1] = es[1] = 1;
      rank = 2;
    }
    order(p.act_dims[1], p.act_dims[2], p.act_dims[3], dims + rank);
    strides[rank - 1] = p.act_strides[0];
    strides[rank] = halo ? p.act_strides[2] : p.act_strides[1];
    strides[rank + 1] = halo ? p.act_strides[1] : p.act_strides[2];
    order(uint64_t((load_w - 1) * p.stride_w + 1), uint64_t((load_h + plan.halo_rows - 1) * p.stride_h + 1),
          uint64_t(load_n), b3);
    order(uint64_t(p.stride_w), uint64_t(p.stride_h), 1, e3);
    for (int i = 0; i < 3; ++i) {
      box[rank + i] = uint32_t(b3[i]);
      es[rank + i] = uint32_t(e3[i]);
    }
    if (int rc = encodeTensorMap(&ta, dt, rank + 3, p.act, dims, strides, box, es)) return rc;
  }
  // One narrow tile covering all output channels: the instruction computes, and
  // a K-major weight box loads, only the columns that exist (16 at least, 32 for
  // a pair, whose CTAs hold half of them each).
  const int n_quantum = plan.cta_pair ? 32 : 16;
  const int n_mma = plan.cta_pair && p.b_mn ? plan.tile_n
                                            : std::min(plan.tile_n, (p.n_total + n_quantum - 1) / n_quantum * n_quantum);
  const int b_rows = p.b_mn ? plan.tile_n / (plan.cta_pair ? 2 : 1) : n_mma / (plan.cta_pair ? 2 : 1);
  {
    uint32_t box[3];
    if (p.b_mn) {
      box[0] = 64;
      box[1] = 64;
      box[2] = 1;
    } else {
      box[0] = uint32_t(k_elems_per_stage);
      box[1] = uint32_t(b_rows);
      box[2] = 1;
    }
    const uint32_t es[3] = {1, 1, 1};
    if (int rc = encodeTensorMap(&tb, dt, 3, p.wgt, p.wgt_dims, p.wgt_strides, box, es)) return rc;
  }

  IgemmArgs a{};
  a.split_k = std::max(1, int(plan.split_k));
  a.fd_split = make_fastdiv(uint32_t(a.split_k));
  const bool split = a.split_k > 1;
  const size_t ld_p = (size_t(p.n_total) + 31) / 32 * 32;
  float *partial = nullptr;
  if (split) {
    void *ws = nullptr;
    a.split_stride = (long long)groups * p.out_w * p.out_h * p.out_n * (long long)ld_p;
    if (int rc = scratch(ctx, kSlotSplitK, size_t(a.split_k) * size_t(a.split_stride) * sizeof(float), &ws))
      return rc;
    partial = static_cast<float *>(ws);
  }
  // Output through TMA when the tensor can be described to it: 16-byte aligned
  // base and pixel stride, and rows that end on 16 bytes (a shorter last vector is written whole,
  // over what lies between the rows of a result with a leading dimension).  Each epilogue warp stores a (columns, w, h, n) box
  // holding its 32 pixels and 32 columns: 128-byte rows of fp32, 64-byte rows
  // (64-byte swizzle) of half.
  CUtensorMap tout;
  std::memset(&tout, 0, sizeof tout);
  const size_t out_es = p.out_f32 ? 4 : 2;
  const long long out_stride_h = p.out_stride_h ? p.out_stride_h : (long long)p.out_w * p.ldc;
  const long long out_stride_n =
      p.out_stride_n ? p.out_stride_n : (long long)p.out_h * p.out_w * p.ldc;
  // the 32 rows of one epilogue warp as a box over the tile's row order
  const int d2 = halo ? plan.box_n : plan.box_h;
  a.sub_w = std::min(plan.box_w, 32);
  a.sub_h = std::min(d2, 32 / a.sub_w);  // extent along the second row dimension
  const int sub_3 = 32 / (a.sub_w * a.sub_h);
  a.use_tma_store = 0;
  if (!split && (p.plan_flags & PLB_PLAN_NO_TMA_STORE) == 0 &&
      (reinterpret_cast<uintptr_t>(p.out) & 15) == 0 && (size_t(p.n_total) * out_es) % 16 == 0 &&
      (size_t(p.ldc) * out_es) % 16 == 0 && (size_t(out_stride_h) * out_es) % 16 == 0 &&
      (size_t(out_stride_n) * out_es) % 16 == 0 && (groups == 1 || (size_t(p.out_group_stride) * out_es) % 16 == 0)) {
    uint64_t dims[5] = {uint64_t(p.n_total)}, strides[4];
    uint32_t box[5] = {32u};
    int rank = 1;
    if (with_groups) {
      dims[1] = uint64_t(groups);
      strides[0] = uint64_t(groups > 1 ? p.out_group_stride : p.ldc) * out_es;
      box[1] = 1;
      rank = 2;
    }
    order(uint64_t(p.out_w), uint64_t(p.out_h), uint64_t(p.out_n), dims + rank);
    const uint64_t sw = uint64_t(p.ldc) * out_es, sh = uint64_t(out_stride_h) * out_es,
                   sn = uint64_t(out_stride_n) * out_es;
    strides[rank - 1] = sw;
    strides[rank] = halo ? sn : sh;
    strides[rank + 1] = halo ? sh : sn;
    box[rank] = uint32_t(a.sub_w);
    box[rank + 1] = uint32_t(a.sub_h);
    box[rank + 2] = uint32_t(sub_3);
    const uint32_t es[5] = {1, 1, 1, 1, 1};
    if (int rc = encodeTensorMap(&tout,
                                 p.out_f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                           : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                                 rank + 3, p.out, dims, strides, box, es, p.out_f32 ? 128 : 64))
      return rc;
    a.use_tma_store = 1;
  }
  a.box_w = plan.box_w;
  a.box_h = plan.box_h;
  a.box_n = plan.box_n;
  a.tiles_w = (p.out_w + plan.box_w - 1) / plan.box_w;
  a.tiles_h = (p.out_h + plan.box_h - 1) / plan.box_h;
  a.tiles_n = (p.out_n + plan.box_n - 1) / plan.box_n;
  a.out_w = p.out_w;
  a.out_h = p.out_h;
  a.out_n = p.out_n;
  a.n_tiles = (p.n_total + plan.tile_n - 1) / plan.tile_n;
  a.n_total = p.n_total;
  a.taps_h = p.taps_h;
  a.taps_w = p.taps_w;
  a.k_chunks = k_chunks;
  a.k_last = k_last;
  a.groups = groups;
  a.fd_groups = make_fastdiv(uint32_t(groups));
  a.out_group_stride = groups > 1 ? p.out_group_stride : 0;
  a.addend_group_stride = groups > 1 ? p.addend_group_stride : 0;
  a.n_mma = n_mma;
  a.b_box_bytes = b_rows * kStageKBytes;
  a.tap_first_h = p.tap_first_h;
  a.tap_step_h = p.tap_step_h;
  a.tap_pitch_h = p.tap_pitch_h ? p.tap_pitch_h : p.taps_w;
  a.tap_first_w = p.tap_first_w;
  a.tap_step_w = p.tap_step_w;
  a.taps_stored = p.taps_stored ? p.taps_stored : p.taps_h * p.taps_w;
  a.pad_h = p.pad_h;
  a.pad_w = p.pad_w;
  a.dil_h = p.dil_h;
  a.dil_w = p.dil_w;
  a.stride_h = p.stride_h;
  a.stride_w = p.stride_w;
  a.flip_h = p.flip_h;
  a.flip_w = p.flip_w;
  a.group_m = plan.cta_pair ? 8 : 16;  // M tiles (pairs of them) per band
  a.h_outer = halo ? 1 : 0;
  a.fd_band = make_fastdiv(uint32_t(std::max(1, a.group_m * a.n_tiles)));
  a.fd_gm = make_fastdiv(uint32_t(std::max(1, a.group_m)));
  a.fd_tw = make_fastdiv(uint32_t(std::max(1, a.tiles_w)));
  a.fd_inner = make_fastdiv(uint32_t(std::max(1, a.h_outer ? a.tiles_n : a.tiles_h)));
  a.a_stage_bytes = plan.box_w * plan.box_n * (plan.box_h + plan.halo_rows) * kStageKBytes;
  a.b_tiles_per_stage = (halo && !plan.resident_weights) ? p.taps_h : 1;
  a.a_blocks = a_blocks;
  a.stage_tx_bytes = (p.a_mn ? a_blocks * 64 * 64 * 2 : load_w * load_n * (load_h + plan.halo_rows) * kStageKBytes) +
                     (plan.resident_weights ? 0 : a.b_tiles_per_stage * a.b_box_bytes);
  a.halo_step_bytes = p.dil_h * plan.box_w * plan.box_n * kStageKBytes;
  a.num_stages = plan.stages;
  // Short tiles (few tensor-core instructions each) are bound by what one
  // thread can issue and wait for per tile: let two issuers take alternate tiles.
  {
    const int steps_per_tile = halo ? a.taps_w * a.k_chunks : a.taps_h * a.taps_w * a.k_chunks;
    const int mmas_per_tile = a.taps_h * a.taps_w * a.k_chunks * 4;
    // (only with CTA pairs and 64-column tiles, the case it was built and
    // verified for: weights resident or streamed, halo strips)
    const int stages = dualIssueStages(plan.stages, steps_per_tile);
    a.dual_issue = ((p.plan_flags & PLB_PLAN_NO_DUAL_ISSUE) == 0 && steps_per_tile <= 4 && mmas_per_tile <= 48 &&
                    plan.tiles >= 2 * plan.grid && plan.cta_pair && plan.tile_n == 64 && !split && stages > 0)
                       ? 1
                       : 0;
    if (a.dual_issue) a.num_stages = stages;
  }
  // The first steps of every CTA, issued at once by idle warps and pulled towards L2
  // before the predecessor has ended, save a short product most of its time (16 x 512 x
  // 512 with operands from memory 4.34 -> 3.84 us) as long as what they ask for together
  // is small.  Beyond, they only delay one another's first stage: with all 25 MB of its
  // first steps requested at once 1024 x 1024 x 1024 took 7.4 us, without the prefetch and
  // with three steps (as many as there are producers) 6.3.  Stages of 24 KB that hold the
  // whole reduction are better loaded in order too (512 x 512 x 512 4.56 -> 4.42 us).
  {
    const long unit_steps = ((halo ? 1L : a.taps_h) * a.taps_w * a.k_chunks + a.split_k - 1) / a.split_k;
    const long steps = std::min<long>(plan.stages, unit_steps);
    const bool small = plan.grid * steps * a.stage_tx_bytes <= kMostFirstBytes;
    const bool at_once = small && (a.stage_tx_bytes <= 16 * 1024 || unit_steps > plan.stages);
    a.first_prefetches = small ? int(steps) : 0;
    a.first_loads = int(at_once ? steps : std::min<long>(steps, kIgemmProducers));
  }
  const int resident_bytes =
      plan.resident_weights ? a.taps_h * a.taps_w * a.k_chunks *
                                  (plan.tile_n / (plan.cta_pair ? 2 : 1)) * kStageKBytes
                            : 0;
  a.out = p.out;
  a.ldc = p.ldc;
  a.out_stride_h = out_stride_h;
  a.out_stride_n = out_stride_n;
  a.addend = p.beta != 0.f ? p.addend : nullptr;
  a.ld_addend = p.ld_addend;
  a.bias = p.bias;
  if (split) {
    // raw fp32 sums, dense in pixels, into this split's slice of the scratch
    a.out = partial;
    a.ldc = (long long)ld_p;
    a.out_stride_h = (long long)p.out_w * a.ldc;
    a.out_stride_n = (long long)p.out_h * a.out_stride_h;
    a.out_group_stride = (long long)p.out_n * a.out_stride_n;
    a.addend = nullptr;
    a.bias = nullptr;
  }
  a.idesc_formats = p.bf16 ? make_idesc(0, 0, 1, 1, false, false) & ~(1u << 4)
                    : p.fp8 ? make_idesc(0, 0, uint32_t(p.fmt_a & 1), uint32_t(p.fmt_b & 1), false, false) & ~(1u << 4)
                          : 0u;
  a.alpha = split ? 1.f : p.alpha;
  a.beta = split ? 0.f : p.beta;
  a.out_is_f32 = split || p.out_f32 ? 1 : 0;
  a.nonfinite = p.nonfinite;
  a.chain = split ? kChainNone : p.chain;
  a.status = ctx->d_status;
  a.trace = ctx->trace;

  const bool pdl = (p.plan_flags & PLB_PLAN_NO_PDL) == 0;
  const IgemmVariant variant{p.fp8, p.a_mn, p.b_mn, plan.resident_weights != 0, halo, plan.cta_pair != 0, with_groups, plan.grid,
                             plan.resident_weights ? groups : 1,
                             resident_bytes, pdl};
  int rc = PLB_OK;
  switch (plan.tile_n) {
    case 64: rc = launchIgemm64(ctx, ta, tb, tout, a, variant); break;
    case 128: rc = launchIgemm128(ctx, ta, tb, tout, a, variant); break;
    case 256: rc = launchIgemm256(ctx, ta, tb, tout, a, variant); break;
    default: return fail(PLB_ERR_INVALID_OPTION, "unsupported tile_n in plan");
  }
  if (rc) return rc;
  if (!split) return PLB_OK;
  SplitKReduceArgs r{};
  r.partial = partial;
  r.split_k = a.split_k;
  r.split_stride = a.split_stride;
  r.ld_p = int(ld_p);
  r.groups = groups;
  r.out_group_stride = p.out_group_stride;
  r.addend_group_stride = p.addend_group_stride;
  r.n_total = p.n_total;
  r.out_w = p.out_w;
  r.out_h = p.out_h;
  r.out_n = p.out_n;
  r.out = p.out;
  r.ldc = p.ldc;
  r.out_stride_h = out_stride_h;
  r.out_stride_n = out_stride_n;
  r.addend = p.beta != 0.f ? p.addend : nullptr;
  r.ld_addend = p.ld_addend;
  r.bias = p.bias;
  r.alpha = p.alpha;
  r.beta = p.beta;
  r.out_is_f32 = p.out_f32 ? 1 : 0;
  const long long work = (long long)groups * p.out_w * p.out_h * p.out_n * ((p.n_total + 3) / 4);
  cudaLaunchAttribute pdl_attr[1];
  pdl_attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  pdl_attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(std::max<long long>(1, std::min<long long>((work + 255) / 256,
                                                                         (long long)ctx->sm_count * 8))));
  cfg.blockDim = dim3(256);
  cfg.stream = ctx->stream;
  cfg.attrs = pdl_attr;
  cfg.numAttrs = pdl ? 1 : 0;
  PLB_CUDA(cudaLaunchKernelEx(&cfg, igemm_splitk_reduce_kernel, r));
  PLB_CUDA(cudaGetLastError());
  ctx->launches++;
  return PLB_OK;
}

}  // namespace plb
