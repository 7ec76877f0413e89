// Weight-update pass: planning and launch of the weight-gradient kernel.
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <string>
#include <type_traits>

#include "conv_geometry.h"
#include "rows.h"
#include "runtime.h"
#include "small_channel.h"
#include "wu_sm100.cuh"

namespace plb {
namespace {

struct WuShape {
  int H, W, OH, OW, KH, KW, padH, padW, dilH, dilW, strH, strW;
  // views: input truncation (tH, tW; extent He x We), output padding (opH, opW;
  // computed extent OHc x OWc); padH/padW already include the output truncation
  int tH, tW, He, We, opH, opW, OHc, OWc;
};

int wuShape(const plb_conv_params &p, WuShape *s) {
  const std::string err = validate(p);
  if (!err.empty()) return fail(PLB_ERR_INVALID_PARAMS, err);
  if (p.num_field_dims > 2)
    return fail(PLB_ERR_UNSUPPORTED, "3-D convolutions are not implemented on this path yet");
  if (!is16BitFloat(p.input_type) && p.input_type != PLB_FLOAT)
    // the reference never runs the weight update in quarter either
    // (tools/single_conv_layer.cpp:725-733)
    return fail(PLB_ERR_UNSUPPORTED, "weight update is implemented for half and float input only");
  for (unsigned d = 0; d != p.num_field_dims; ++d) {
    // (kernel truncation and flip are resolved by plb_conv_wu before it gets here)
    if (p.in_dilation[d] != 1 || p.in_flip[d] || p.k_trunc_lo[d] || p.k_trunc_hi[d] || p.k_flip[d])
      return fail(PLB_ERR_UNSUPPORTED,
                  "input dilation/flip are not implemented on this path yet (kernel truncation "
                  "and flip only through plb_conv_wu)");
    if (p.stride[d] > 8) return fail(PLB_ERR_UNSUPPORTED, "strides above 8 are not implemented");
  }
  const unsigned hd = p.num_field_dims == 2 ? 0 : ~0u, wd = p.num_field_dims - 1;
  auto get = [&](const uint32_t *v, unsigned d, int dflt) { return d == ~0u ? dflt : int(v[d]); };
  s->H = get(p.field, hd, 1);
  s->W = get(p.field, wd, 1);
  s->KH = get(p.kernel, hd, 1);
  s->KW = get(p.kernel, wd, 1);
  s->padH = get(p.in_pad_lo, hd, 0);
  s->padW = get(p.in_pad_lo, wd, 0);
  s->dilH = get(p.k_dilation, hd, 1);
  s->dilW = get(p.k_dilation, wd, 1);
  s->strH = get(p.stride, hd, 1);
  s->strW = get(p.stride, wd, 1);
  s->OH = hd == ~0u ? 1 : int(outputSize(p, hd));
  s->OW = int(outputSize(p, wd));
  s->tH = get(p.in_trunc_lo, hd, 0);
  s->tW = get(p.in_trunc_lo, wd, 0);
  s->He = s->H - s->tH - get(p.in_trunc_hi, hd, 0);
  s->We = s->W - s->tW - get(p.in_trunc_hi, wd, 0);
  // kernel padding only shifts where the taps land
  s->padH -= get(p.out_trunc_lo, hd, 0) + get(p.k_pad_lo, hd, 0);
  s->padW -= get(p.out_trunc_lo, wd, 0) + get(p.k_pad_lo, wd, 0);
  s->opH = get(p.out_pad_lo, hd, 0);
  s->opW = get(p.out_pad_lo, wd, 0);
  s->OHc = s->OH - s->opH - get(p.out_pad_hi, hd, 0);
  s->OWc = s->OW - s->opW - get(p.out_pad_hi, wd, 0);
  return PLB_OK;
}

// One contraction of the weight-gradient kernel: the operands as it reads them.
struct WuProblem {
  bool bf16 = false;
  int batch = 0;
  int ci = 0, co = 0;               // channels of a super-group (as stored)
  int sgroups = 1, sub = 1;         // super-groups, groups in each
  int sub_ci = 0, sub_co = 0;       // stored channels per group
  WuShape s;                        // field, taps, padding, stride
  // base address, channels of a pixel, byte strides of w, h, n
  const void *x = nullptr, *dy = nullptr;
  uint64_t x_chans = 0, dy_chans = 0, x_strides[3] = {}, dy_strides[3] = {};
};

// Whether narrow channel groups run on the kernel that keeps a group's sums in a warp's registers.
bool narrowGroups(int sm_count, const plb_conv_params &p, const WuShape &s, int force_split, unsigned plan_flags,
                  const void *x, const void *dy, RowsWuProblem *q, RowsWuTiling *t) {
  if (p.input_type != PLB_HALF || force_split != 0 || plan_flags != 0 || p.in_chans_per_group != p.out_chans_per_group) return false;
  if (s.KH != s.KW || s.strH != 1 || s.strW != 1 || s.dilH != 1 || s.dilW != 1 || s.opH || s.opW || s.OHc != s.OH || s.OWc != s.OW) return false;
  const int c = int(p.in_chans_per_group);
  *q = RowsWuProblem{static_cast<const uint8_t *>(x) + (size_t(s.tH) * s.W + s.tW) * p.groups * c * 2, dy, int(p.groups), c, s.KH,
                     int(p.batch), s.We, s.He, s.W, s.H, s.OW, s.OH, s.padW, s.padH};
  return rowsWuSuits(sm_count, *q, t);
}

// How the channels of a pixel lie in the operands the kernel reads, and how many
// groups are contracted together (every sub'th group starts a super-group).
struct WuLayout {
  uint32_t sub, ci_pitch, co_pitch;  // channels from one group to the next
  uint64_t x_pixel, dy_pixel;        // from one pixel to the next
};

// Groups together: as many as fill the 128 output-channel rows of the tensor-core
// tile without exceeding 128 input channels.  32 groups of 8 channels run as two
// dense blocks of 128 x 128 instead of 32 launches whose tiles are 15/16 padding.
// A super-group has to start on a 16-byte boundary; only where no number of groups
// does are the channels of each group rounded up.
WuLayout wuLayout(uint32_t groups, uint32_t ci, uint32_t co, bool copied = false) {
  WuLayout l{};
  const uint32_t most = std::max<uint32_t>(1, std::min(groups, std::min(128 / std::max(co, 1u), 128 / std::max(ci, 1u))));
  auto quantum = [](uint32_t c) {
    uint32_t q = 1;
    while ((q * c) % 8 != 0) q *= 2;
    return q;
  };
  const uint32_t q = std::max(quantum(ci), quantum(co));
  l.sub = most == groups ? groups : most / q * q;
  l.ci_pitch = ci;
  l.co_pitch = co;
  if (l.sub == 0) {
    l.ci_pitch = roundToVec(ci, 2);
    l.co_pitch = roundToVec(co, 2);
    l.sub = std::max<uint32_t>(1, std::min(groups, std::min(128 / l.co_pitch, 128 / l.ci_pitch)));
  }
  // (`copied`: both tensors are copied in any case)
  auto pixel = [&](uint64_t chans) { return copied || chans % 8 != 0 ? roundToRow(chans, 2) : uint32_t(chans); };
  // where each group is rounded up on its own, pixels are those rows side by side
  l.x_pixel = l.ci_pitch != ci ? groups * l.ci_pitch : pixel(uint64_t(groups) * ci);
  l.dy_pixel = l.co_pitch != co ? groups * l.co_pitch : pixel(uint64_t(groups) * co);
  return l;
}

// The layer's tensors [N][H][W][x_pixel] with the channels laid out as `l` says.
WuProblem wuProblem(const plb_conv_params &p, const WuShape &s, const WuLayout &l, uint32_t groups) {
  const uint32_t ci_pitch = l.ci_pitch, co_pitch = l.co_pitch, sub = l.sub;
  const size_t es = 2;
  WuProblem q;
  q.bf16 = p.input_type == PLB_BFLOAT16;
  q.batch = int(p.batch);
  q.sub = int(sub);
  q.sgroups = int((groups + sub - 1) / sub);
  q.sub_ci = int(ci_pitch);
  q.sub_co = int(co_pitch);
  // (a single super-group may include the channels the pixel was rounded up by)
  q.ci = int(q.sgroups == 1 ? roundToVec(sub * ci_pitch, 2) : sub * ci_pitch);
  q.co = int(q.sgroups == 1 ? roundToVec(sub * co_pitch, 2) : sub * co_pitch);
  q.s = s;
  // what a super-group reads beyond its own channels only meets sums that nothing
  // reads; the end of the pixel is the end of the tensor
  q.x_chans = std::max<uint64_t>(uint64_t(groups) * ci_pitch, l.x_pixel * (p.groups == groups ? 1 : 0));
  q.dy_chans = std::max<uint64_t>(uint64_t(groups) * co_pitch, l.dy_pixel * (p.groups == groups ? 1 : 0));
  const uint64_t xp = l.x_pixel * es, yp = l.dy_pixel * es;
  q.x_strides[0] = xp;
  q.x_strides[1] = uint64_t(s.W) * xp;
  q.x_strides[2] = uint64_t(s.H) * s.W * xp;
  q.dy_strides[0] = yp;
  q.dy_strides[1] = uint64_t(s.OW) * yp;
  q.dy_strides[2] = uint64_t(s.OH) * s.OW * yp;
  return q;
}

// Tiling of a weight update.
void planWu(const WuProblem &p, int sm_count, int force_split, unsigned plan_flags, WuArgs *a, plb_plan *plan) {
  const WuShape &s = p.s;
  const int co = p.co, ci = p.ci;
  const int taps = s.KH * s.KW;
  a->taps_h = s.KH;
  a->taps_w = s.KW;
  a->pad_h = s.padH;
  a->pad_w = s.padW;
  a->dil_h = s.dilH;
  a->dil_w = s.dilW;
  a->stride_h = s.strH;
  a->stride_w = s.strW;
  a->sgroups = p.sgroups;
  a->x_step = ci;
  a->dy_step = co;
  a->sub = p.sub;
  a->sub_ci = p.sub_ci;
  a->sub_co = p.sub_co;
  a->co_total = co;
  a->ci_total = ci;
  a->co_blocks = (co + 127) / 128;
  a->ci_blk = std::min(256, (ci + 31) / 32 * 32);
  a->ci_blk64 = (a->ci_blk + 63) / 64;
  a->ci_blocks = (ci + a->ci_blk - 1) / a->ci_blk;
  a->taps_per_group = std::max(1, std::min(taps, 512 / a->ci_blk));
  // two pipeline stages of (outGrad tile + one activation box per tap) must fit
  while (a->taps_per_group > 1 &&
         2 * (2 + a->taps_per_group * a->ci_blk64) * kWuBlockBytes > 200 * 1024)
    --a->taps_per_group;
  a->tap_groups = (taps + a->taps_per_group - 1) / a->taps_per_group;
  // even out the groups (9 taps, 4 per group -> 3 groups of 3)
  a->taps_per_group = (taps + a->tap_groups - 1) / a->tap_groups;
  int cols = a->taps_per_group * a->ci_blk, pow2 = 32;
  while (pow2 < cols) pow2 <<= 1;
  a->tmem_cols = pow2;
  // pixel box: 64 pixels, fewest tiles, then widest rows
  long best = -1;
  for (int w = 64; w >= 1; w >>= 1)
    for (int h = 64 / w; h >= 1; h >>= 1) {
      const int n = 64 / (w * h);
      if ((w - 1) * s.strW + 1 > 256 || (h - 1) * s.strH + 1 > 256) continue;
      const long tiles =
          long((s.OWc + w - 1) / w) * ((s.OHc + h - 1) / h) * ((long(p.batch) + n - 1) / n);
      if (best < 0 || tiles < best) {
        best = tiles;
        a->box_w = w;
        a->box_h = h;
        a->box_n = n;
      }
    }
  int stage_bytes = (2 + a->taps_per_group * a->ci_blk64) * kWuBlockBytes;
  // Strip mode: one tap group per filter column, the activations of a K step
  // loaded once for all filter rows.  Needs a unit vertical stride, all filter
  // rows' accumulators in TMEM at once and box_w * box_n a multiple of 8; taken
  // when it costs at most 1/8 more pixel tiles than the best box.
  a->strip_mode = 0;
  // PLB_PLAN_NO_A_COLLECTOR: fetch the outGrad tile for every instruction (A/B timing)
  a->reuse_a = (plan_flags & PLB_PLAN_NO_A_COLLECTOR) ? 0 : 1;
  a->idesc_formats = p.bf16 ? (make_idesc(0, 0, 1, 1, false, false) & ~(1u << 4)) : 0u;
  const int halo = (s.KH - 1) * s.dilH;
  if (s.KH > 1 && s.strH == 1 && s.KH * a->ci_blk <= 512 && (plan_flags & PLB_PLAN_NO_HALO) == 0) {
    long sbest = -1;
    int sw = 0, sh = 0, sn = 0;
    for (int h = 64; h >= 1; h >>= 1)  // tallest first: least halo per row
      for (int w = 64 / h; w >= 1; w >>= 1) {
        const int n = 64 / (w * h);
        if ((w * n) % 8 != 0 || h + halo > 256 || (w - 1) * s.strW + 1 > 256) continue;
        const long tiles =
            long((s.OWc + w - 1) / w) * ((s.OHc + h - 1) / h) * ((long(p.batch) + n - 1) / n);
        if (sbest < 0 || tiles < sbest) {
          sbest = tiles;
          sw = w;
          sh = h;
          sn = n;
        }
      }
    const int strip_rows = sw * sn * (sh + halo);
    const int sbytes = 2 * kWuBlockBytes + a->ci_blk64 * strip_rows * 128;
    if (sbest > 0 && sbest * 8 <= best * 9 && 2 * sbytes <= 200 * 1024) {
      a->strip_mode = 1;
      a->box_w = sw;
      a->box_h = sh;
      a->box_n = sn;
      a->strip_rows = strip_rows;
      a->halo_step_bytes = s.dilH * sw * sn * 128;
      a->taps_per_group = s.KH;
      a->tap_groups = s.KW;
      a->tmem_cols = 32;
      while (a->tmem_cols < s.KH * a->ci_blk) a->tmem_cols <<= 1;
      stage_bytes = sbytes;
      best = sbest;
    }
  }
  // Both halves of the instruction's rows for 64 output channels (fewer: the copies take longer
  // than the instructions): where a 16-pixel step lies in one row, and all tiles then take less.  A tile
  // takes what its instructions do (one of n columns about 35 + 0.47 n cycles: measured 75, 95, 155 at 64,
  // 128 and 256), its way into and out of shared memory at 100 bytes a cycle (measured 91 to 110), or
  // its copies by pixel (3.1 cycles, 7.5 where its channels do not fill 128 bytes); and the tiles of a CTA
  // have to win 2000 cycles for clearing the accumulators and the edge rows.  (That is on the safe side:
  // it leaves 5x5, 64 channels, 2 images of 56 x 56 unpaired, 9.6 us, paired 8.7, and 3x3, 4 of 33 x 29, 7.4
  // and 7.3; it was found with 40 output channels, 12.6 us unpaired and 13.3 paired, which are not paired
  // now.)  Boxes are eight pixels wide and more: of single columns of 16 images, 3x3, 4 groups of 16, 16 images
  // of 107 x 107 took 44 us, unpaired 34.
  a->pair_rows = a->pair_shift = 0;
  if (a->strip_mode && co == 64) {
    const int rows = (s.KH + 1) / 2, shift = rows * s.dilH;
    auto cost = [&](int filter_rows, int dy_rows, int x_rows) {
      const int each = a->ci_blk == 64 ? std::min(4, filter_rows) : 1, count = (filter_rows + each - 1) / each;
      const double columns = filter_rows * a->ci_blk, fill = (dy_rows + a->ci_blk64 * x_rows) * 128.0;
      const double copies = dy_rows * 3.1 + a->ci_blk64 * x_rows * (ci % 64 ? 7.5 : 3.1);
      return std::max({4 * (35 * count + 0.47 * columns), (fill + 4 * (4096 * count + 32 * columns)) / 100, copies});
    };
    const double before = best * cost(s.KH, 64, a->strip_rows);
    const int columns = a->sgroups * a->ci_blocks * s.KW;
    // (a constraint to as many CTAs as there are tiles may be the saved plan of a call that had SMs for more:
    // it is weighed as that call was, and leads to the same kernel)
    const int room = std::max(1, (sm_count > 0 ? sm_count : 148) / columns);
    const double splits = force_split <= 0 ? room : force_split < best ? force_split : std::max(force_split, room);
    double least = std::min(0.94 * before, before - 2000 * splits);
    for (int h = 4; h >= 1; h >>= 1)
      for (int w = 64 / h; w >= 1; w >>= 1) {
        const int n = 64 / (w * h), dy_rows = w * n * (h + shift), strip_rows = w * n * (h + (rows - 1) * s.dilH);
        const int bytes = (dy_rows + a->ci_blk64 * strip_rows) * 128;
        if (h + shift > 256 || (w - 1) * s.strW + 1 > 256 || 3 * bytes > 200 * 1024) continue;
        const long tiles = long((s.OWc + w - 1) / w) * ((s.OHc + shift + h - 1) / h) * ((long(p.batch) + n - 1) / n);
        if (w < 8 || tiles * cost(rows, dy_rows, strip_rows) >= least) continue;
        least = tiles * cost(rows, dy_rows, strip_rows);
        a->box_w = w;
        a->box_h = h;
        a->box_n = n;
        a->pair_rows = rows;
        a->pair_shift = shift;
        a->dy_rows = dy_rows;
        a->strip_rows = strip_rows;
        stage_bytes = bytes;
        best = tiles;
      }
    if (a->pair_rows) {
      a->halo_step_bytes = s.dilH * a->box_w * a->box_n * 128;
      a->taps_per_group = rows;
      a->tmem_cols = 32;
      while (a->tmem_cols < rows * a->ci_blk) a->tmem_cols <<= 1;
      a->last_row = s.OHc;
    }
  }
  a->tiles_w = (s.OWc + a->box_w - 1) / a->box_w;
  a->tiles_h = (s.OHc + a->pair_shift + a->box_h - 1) / a->box_h;
  a->tiles_n = (int(p.batch) + a->box_n - 1) / a->box_n;
  a->stage_bytes = stage_bytes;
  a->stages = std::max(2, std::min(kWuMaxStages, (200 * 1024) / stage_bytes));
  const int units = a->sgroups * a->co_blocks * a->ci_blocks * a->tap_groups;
  int ksplit = force_split > 0 ? force_split : std::max(1, (sm_count > 0 ? sm_count : 148) / units);
  ksplit = int(std::min<long>(ksplit, std::max<long>(best, 1)));
  a->ksplit = ksplit;
  if (plan) {
    plan->kernel = 1;
    // (paired: a CTA's tile is 64 output channels' sums of all filter rows, in instructions of 128 rows and half
    // the columns)
    plan->tile_m = a->pair_rows ? 64 : 128;
    plan->tile_n = (a->pair_rows ? s.KH : a->taps_per_group) * a->ci_blk;
    plan->tile_k_bytes = kWuPixelsPerStage * 2;
    plan->box_w = a->box_w;
    plan->box_h = a->box_h;
    plan->box_n = a->box_n;
    plan->stages = a->stages;
    plan->split_k = ksplit;
    plan->tiles = units;
    plan->grid = units * ksplit;
    plan->b_mn_major = 1;
    plan->halo_rows = a->pair_rows ? (a->pair_rows - 1) * s.dilH : a->strip_mode ? halo : 0;
    plan->workspace_bytes = size_t(ksplit) * p.sgroups * taps * co * ci * sizeof(float);
  }
}

// Gradient of the used taps -> gradient of the stored filter: tap (th, tw) of
// the [G][JH*JW][inner] source goes to tap (r0h + th', r0w + tw') of the
// zero-initialised [G][KH*KW][inner] destination, th' = JH-1-th when the
// kernel is used flipped in that dimension.  `vec_bytes` is 4 or 2.
template <typename T>
__global__ void scatterTapsKernel(const T *__restrict__ src, T *__restrict__ dst, int groups, int KH,
                                  int KW, int JH, int JW, int r0h, int r0w, int flip_h, int flip_w,
                                  size_t inner) {
  const size_t total = size_t(groups) * JH * JW * inner;
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < total;
       i += size_t(gridDim.x) * blockDim.x) {
    const size_t v = i % inner;
    size_t t = i / inner;
    const int tw = int(t % JW);
    t /= JW;
    const int th = int(t % JH);
    const int g = int(t / JH);
    const int oh = r0h + (flip_h ? JH - 1 - th : th), ow = r0w + (flip_w ? JW - 1 - tw : tw);
    dst[(size_t(g) * KH * KW + size_t(oh) * KW + ow) * inner + v] = src[i];
  }
}

// The wu kernel needs more dynamic shared memory than the default limit: raised
// once per device, for every entry point alike.
int configureWuKernel(int device) {
  static std::mutex mutex;
  static bool configured[64] = {};
  if (device < 0 || device >= 64) return fail(PLB_ERR_INVALID_PARAMS, "device ordinal out of range");
  std::lock_guard<std::mutex> lock(mutex);
  if (!configured[device]) {
    // the caller has made `device` current
    for (auto *kernel : {wu_kernel<false>, wu_kernel<true>})
      PLB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured[device] = true;
  }
  return PLB_OK;
}

cudaLaunchConfig_t wuReduceConfig(cudaStream_t stream, size_t blocks, cudaLaunchAttribute *pdl) {
  pdl->id = cudaLaunchAttributeProgrammaticStreamSerialization;
  pdl->val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(blocks));
  cfg.blockDim = dim3(32, kWuReduceLanes);
  cfg.stream = stream;
  cfg.attrs = pdl;
  cfg.numAttrs = 1;
  return cfg;
}

// Reduction over the K splits (and, with `peer`, over the ranks) into one
// gradient of w_elems.  The partial sums are in the gradient's order unless
// `gather` says otherwise.
int launchWuReduce(cudaStream_t stream, const WuArgs &a, size_t w_elems, void *d_weight_grads,
                   float *d_weight_grads_f32, const WuGather *gather, const WuPeerArgs *peer = nullptr,
                   unsigned group = 0) {
  cudaLaunchAttribute pdl[1];
  __half *out16 = static_cast<__half *>(d_weight_grads);
  const bool vec = w_elems % 4 == 0 && (reinterpret_cast<uintptr_t>(d_weight_grads_f32) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(out16) & 7) == 0;
  const size_t count4 = w_elems / 4;
  if (peer != nullptr) {
    const unsigned rgrid = unsigned((count4 + kWuFusedChunk - 1) / kWuFusedChunk);
    WuPeerArgs pa = *peer;
    for (int r = 0; r < pa.world; ++r) {
      pa.grads[r] += size_t(group) * count4;
      if (pa.results[r] != nullptr) pa.results[r] += size_t(group) * count4;
    }
    pa.chunk_base = group * rgrid;
    const cudaLaunchConfig_t cfg = wuReduceConfig(stream, rgrid, pdl);
    PLB_CUDA(cudaLaunchKernelEx(&cfg, wu_reduce_allreduce_kernel, reinterpret_cast<const float4 *>(a.partial),
                                a.ksplit, count4, pa, reinterpret_cast<float4 *>(d_weight_grads_f32),
                                reinterpret_cast<uint2 *>(out16)));
  } else if (gather == nullptr && vec) {
    // (up to 8 splits, one thread per sum adds in the same order as eight lanes)
    const bool single = a.ksplit <= kWuReduceLanes && count4 >= size_t(148) * 512;
    cudaLaunchConfig_t cfg = wuReduceConfig(stream, single ? (count4 + 255) / 256 : (count4 + 31) / 32, pdl);
    if (single) cfg.blockDim = dim3(256, 1);
    PLB_CUDA(cudaLaunchKernelEx(&cfg, single ? wu_reduce4_kernel<1> : wu_reduce4_kernel<kWuReduceLanes>, reinterpret_cast<const float4 *>(a.partial), a.ksplit,
                                count4, reinterpret_cast<float4 *>(d_weight_grads_f32),
                                reinterpret_cast<uint2 *>(out16)));
  } else {
    WuGather g{};
    if (gather) {
      g = *gather;
    } else {
      g.taps = g.p_taps = uint32_t(a.taps_h * a.taps_w);
      g.co = g.co_pitch = g.p_co = uint32_t(a.co_total);
      g.ci = g.ci_pitch = g.p_ci = uint32_t(a.ci_total);
      g.sub = 1;
    }
    g.split_stride = (unsigned long long)a.sgroups * a.taps_h * a.taps_w * a.co_total * a.ci_total;
    g.total = w_elems;
    // four channels at once where they are neighbours on both sides
    const int V = vec && g.ci % 4 == 0 && g.ci_pitch % 4 == 0 ? 4 : 1;
    const size_t vectors = w_elems / V;
    g.fd_ci = make_fastdiv(g.ci / V);
    g.fd_co = make_fastdiv(g.co);
    g.fd_taps = make_fastdiv(g.taps);
    g.fd_sub = make_fastdiv(g.sub);
    // as few threads per sum as fill the device: each then has several loads in flight
    int lanes = 1;
    while (lanes < 8 && lanes < a.ksplit && vectors * lanes < size_t(148) * 1024) lanes *= 2;
    auto launch = [&](auto kernel, int L) {
      const size_t per_block = size_t(kWuReduceThreads / L);
      cudaLaunchConfig_t cfg = wuReduceConfig(stream, (vectors + per_block - 1) / per_block, pdl);
      cfg.blockDim = dim3(kWuReduceThreads);
      return cudaLaunchKernelEx(&cfg, kernel, (const float *)a.partial, a.ksplit, g, d_weight_grads_f32, out16);
    };
    auto dispatch = [&](auto v) {
      constexpr int kV = decltype(v)::value;
      if (vectors >= (size_t(1) << 31)) return launch(wu_gather_kernel<kV, 8, true>, 8);
      switch (lanes) {
        case 1: return launch(wu_gather_kernel<kV, 1, false>, 1);
        case 2: return launch(wu_gather_kernel<kV, 2, false>, 2);
        case 4: return launch(wu_gather_kernel<kV, 4, false>, 4);
        default: return launch(wu_gather_kernel<kV, 8, false>, 8);
      }
    };
    if (V == 4)
      PLB_CUDA(dispatch(std::integral_constant<int, 4>()));
    else
      PLB_CUDA(dispatch(std::integral_constant<int, 1>()));
  }
  PLB_CUDA(cudaGetLastError());
  return PLB_OK;
}

// Launches the weight-gradient kernel.  `a.partial` and `a.status` are set by the caller.
int launchWuKernel(cudaStream_t stream, const WuProblem &p, const WuArgs &a) {
  const WuShape &s = p.s;
  const int taps = s.KH * s.KW;
  const int smem = a.stages * a.stage_bytes + 256 + 1024;
  const uint32_t ones[4] = {1, 1, 1, 1};
  CUtensorMap tout, tdy, tx;
  {
    // partial sums [ksplit][sgroups * taps][co][ci] fp32, stored in blocks of 32 x 32
    const uint64_t w_elems = uint64_t(p.sgroups) * taps * p.co * p.ci;
    const uint64_t dims[4] = {uint64_t(p.ci), uint64_t(p.co), uint64_t(p.sgroups) * taps, uint64_t(a.ksplit)};
    const uint64_t strides[3] = {uint64_t(p.ci) * 4, uint64_t(p.co) * p.ci * 4, w_elems * 4};
    const uint32_t box[4] = {32, 32, 1, 1};
    if (int rc = encodeTensorMap(&tout, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a.partial, dims, strides, box, ones))
      return rc;
  }
  // pixel dimensions (w, h, n); strip mode orders them (w, n, h)
  const bool strip = a.strip_mode != 0;
  const int halo = strip ? ((a.pair_rows ? a.pair_rows : s.KH) - 1) * s.dilH : 0;
  const uint64_t batch = uint64_t(p.batch);
  {
    const uint64_t dims[4] = {p.dy_chans, uint64_t(s.OWc), strip ? batch : uint64_t(s.OHc),
                              strip ? uint64_t(s.OHc) : batch};
    const uint64_t strides[3] = {p.dy_strides[0], p.dy_strides[strip ? 2 : 1], p.dy_strides[strip ? 1 : 2]};
    const uint32_t box[4] = {64, uint32_t(a.box_w), uint32_t(strip ? a.box_n : a.box_h),
                             uint32_t(strip ? a.box_h + a.pair_shift : a.box_n)};
    if (int rc = encodeTensorMap(&tdy, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
                                 static_cast<const uint8_t *>(p.dy) + uint64_t(s.opH) * p.dy_strides[1] +
                                     uint64_t(s.opW) * p.dy_strides[0],
                                 dims, strides, box, ones))
      return rc;
  }
  {
    const uint64_t dims[4] = {p.x_chans, uint64_t(s.We), strip ? batch : uint64_t(s.He),
                              strip ? uint64_t(s.He) : batch};
    const uint64_t strides[3] = {p.x_strides[0], p.x_strides[strip ? 2 : 1], p.x_strides[strip ? 1 : 2]};
    const uint32_t bw = uint32_t((a.box_w - 1) * s.strW + 1);
    const uint32_t bh = strip ? uint32_t(a.box_h + halo) : uint32_t((a.box_h - 1) * s.strH + 1);
    const uint32_t box[4] = {64, bw, strip ? uint32_t(a.box_n) : bh, strip ? bh : uint32_t(a.box_n)};
    const uint32_t estr[4] = {1, uint32_t(s.strW), strip ? 1u : uint32_t(s.strH), 1};
    if (int rc = encodeTensorMap(&tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
                                 static_cast<const uint8_t *>(p.x) + uint64_t(s.tH) * p.x_strides[1] +
                                     uint64_t(s.tW) * p.x_strides[0],
                                 dims, strides, box, estr))
      return rc;
  }
  const int grid = a.sgroups * a.co_blocks * a.ci_blocks * a.tap_groups * a.ksplit;
  // programmatic stream serialization: the kernel's set-up overlaps the tail of
  // whatever runs before it; it waits before touching global memory
  cudaLaunchAttribute pdl[1];
  pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  pdl[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(grid));
  cfg.blockDim = dim3(kWuThreads);
  cfg.dynamicSmemBytes = size_t(smem);
  cfg.stream = stream;
  cfg.attrs = pdl;
  cfg.numAttrs = 1;
  PLB_CUDA(cudaLaunchKernelEx(&cfg, a.pair_rows ? wu_kernel<true> : wu_kernel<false>, tdy, tx, tout, a));
  PLB_CUDA(cudaGetLastError());
  return PLB_OK;
}

// One group of a layer whose groups are contracted one after the other.
WuLayout oneGroup(const plb_conv_params &p) {
  const uint32_t ci = p.in_chans_per_group, co = p.out_chans_per_group;
  return WuLayout{1, ci, co, uint64_t(p.groups) * ci, uint64_t(p.groups) * co};
}

// Few input channels (an image network's first layer): the rearranged input of
// the forward pass, whose pixels hold a window of the filter's columns, so that
// the KW taps of a filter row are 64 channels of one tap.  (On channels padded to
// 8 the layer 7x7, stride 2, 3 -> 64 channels, 256 images of 224x224, took
// 49 taps of 5/8 padding and 5.5 ms.)  Returns whether it applies.
bool rearrangedProblem(const plb_conv_params &p, const WuShape &s, S2dShape *g, WuProblem *q) {
  const uint32_t ci = p.in_chans_per_group, co = p.out_chans_per_group;
  if (ci % 8 == 0 || co % 8 != 0 || p.input_type == PLB_FLOAT || smallChannelShape(p, g) != PLB_OK) return false;
  WuShape s2 = s;
  s2.H = s2.He = g->H2;
  s2.W = g->W2;
  s2.We = g->OW;  // windows per row
  s2.KH = g->K2h;
  s2.KW = 1;
  s2.padH = s2.padW = 0;
  s2.strH = s2.strW = 1;
  *q = wuProblem(p, s2, WuLayout{1, 64, co, 64, uint64_t(co)}, 1);
  q->x_strides[0] = uint64_t(g->C2) * 2;
  q->x_strides[1] = uint64_t(g->W2) * g->C2 * 2;
  q->x_strides[2] = uint64_t(g->H2) * g->W2 * g->C2 * 2;
  return true;
}
size_t rearrangedBytes(const S2dShape &g) { return smallChannelElems(g) * 2 + 256; }

// The general form: channel counts TMA cannot address (a pixel must be a multiple of
// 16 bytes) run on copies with the channels rounded up; float operands as three
// batches of bfloat16 pieces side by side.  The padded rows and columns of the
// partial sums are not read.  `x` and `dy` become the operands as the kernel reads
// them; up to two copies are left to do in `jobs`, `bytes` of scratch in all.
struct WuOperands {
  WuLayout layout;
  Repack jobs[2];
  const void **operand[2];
  size_t offset[2];
  int copies = 0;
  size_t bytes = 0;
};
WuProblem generalProblem(const plb_conv_params &p, const WuShape &s, const void **x, const void **dy, WuOperands *o) {
  const uint32_t ci = p.in_chans_per_group, co = p.out_chans_per_group;
  const bool is_float = p.input_type == PLB_FLOAT;
  const WuLayout l = wuLayout(p.groups, ci, co, is_float);
  // whole pixels, or where the groups' channels are rounded up, each group's
  auto add = [&](const void **base, uint64_t pixels, uint32_t chans, uint32_t chans_pitch, uint64_t pixel, bool second) {
    if (!is_float && chans == chans_pitch && pixel == uint64_t(p.groups) * chans &&
        (reinterpret_cast<uintptr_t>(*base) & 15) == 0)
      return;
    const bool whole = chans == chans_pitch;
    const uint32_t cols = whole ? p.groups * chans : chans;
    o->jobs[o->copies] = Repack{*base, nullptr, whole ? pixels : pixels * p.groups, cols, cols, whole ? uint32_t(pixel) : chans_pitch,
                                is_float ? 4u : 2u, is_float ? kRepackSplitPlanes : kRepackCopy, second, 0, {}};
    o->offset[o->copies] = o->bytes;
    o->bytes += (repackBytes(o->jobs[o->copies]) + 255) & ~size_t(255);
    o->operand[o->copies++] = base;
  };
  add(x, uint64_t(p.batch) * s.H * s.W, ci, l.ci_pitch, l.x_pixel, false);
  add(dy, uint64_t(p.batch) * s.OH * s.OW, co, l.co_pitch, l.dy_pixel, true);
  o->layout = l;
  plb_conv_params q16 = p;
  if (is_float) {
    q16.input_type = PLB_BFLOAT16;
    q16.batch *= 3;
  }
  return wuProblem(q16, s, l, p.groups);
}

// The groups of a layer one after the other, through one group's worth of scratch
// (the entry points that cannot hold more).  With `peer` the reduction also adds
// the gradients of the other ranks; the caller has checked that the shapes allow it.
int launchWuPerGroup(cudaStream_t stream, const plb_conv_params &p, const WuShape &s, const WuArgs &a,
                     const void *d_acts, const void *d_out_grads, void *d_weight_grads,
                     float *d_weight_grads_f32, uint64_t *launches, const WuPeerArgs *peer = nullptr) {
  const uint32_t co = p.out_chans_per_group, ci = p.in_chans_per_group;
  const size_t w_elems = size_t(s.KH) * s.KW * co * ci, es = 2;
  for (unsigned g = 0; g < p.groups; ++g) {
    WuProblem q = wuProblem(p, s, oneGroup(p), 1);
    q.x = static_cast<const uint8_t *>(d_acts) + size_t(g) * ci * es;
    q.dy = static_cast<const uint8_t *>(d_out_grads) + size_t(g) * co * es;
    if (int rc = launchWuKernel(stream, q, a)) return rc;
    if (int rc = launchWuReduce(
            stream, a, w_elems, d_weight_grads ? static_cast<uint8_t *>(d_weight_grads) + g * w_elems * es : nullptr,
            d_weight_grads_f32 ? d_weight_grads_f32 + g * w_elems : nullptr, nullptr, peer, g))
      return rc;
    if (launches) *launches += 2;
  }
  return PLB_OK;
}

}  // namespace
}  // namespace plb

using namespace plb;

extern "C" {

int plb_conv_wu_plan(const plb_conv_params *p_in, const plb_conv_options *opt, plb_plan *plan) {
  if (!p_in || !plan) return fail(PLB_ERR_INVALID_PARAMS, "null argument");
  if (p_in->num_field_dims == 3) return conv3dPlan(*p_in, opt, PLB_PASS_TRAINING_WU, plan);
  // plan what plb_conv_wu runs: flipped inputs are reversed first, truncated /
  // flipped kernels are computed as ordinary kernels of the truncated extent
  plb_conv_params q;
  unflippedInputParams(*p_in, &q);
  {
    plb_conv_params undilated;
    DilatedField df;
    if (undilatedInputParams(q, &undilated, &df)) q = undilated;
  }
  for (unsigned d = 0; d != q.num_field_dims && d < PLB_MAX_FIELD_DIMS; ++d) {
    q.kernel[d] -= std::min(q.kernel[d], q.k_trunc_lo[d] + q.k_trunc_hi[d]);
    q.k_trunc_lo[d] = q.k_trunc_hi[d] = 0;
    if (q.k_flip[d]) std::swap(q.k_pad_lo[d], q.k_pad_hi[d]);
    q.k_flip[d] = 0;
  }
  const plb_conv_params *p = &q;
  WuShape s;
  if (int rc = wuShape(*p, &s)) return rc;
  *plan = plb_plan{};
  WuArgs a{};
  if (p->groups == 0 || p->in_chans_per_group == 0 || p->out_chans_per_group == 0 || p->batch == 0 || s.OHc <= 0 ||
      s.OWc <= 0 || s.He <= 0 || s.We <= 0)
    return PLB_OK;  // nothing is contracted
  S2dShape g2{};
  WuProblem w;
  const void *x = nullptr, *dy = nullptr;  // (as aligned as they need to be)
  WuOperands operands;
  const bool rearranged = rearrangedProblem(*p, s, &g2, &w);
  if (!rearranged) w = generalProblem(*p, s, &x, &dy, &operands);
  planWu(w, 148, opt ? opt->split_k : 0, opt ? opt->plan_flags : 0, &a, plan);
  plan->workspace_bytes += rearranged ? rearrangedBytes(g2) : operands.bytes;
  RowsWuProblem rows;
  RowsWuTiling t;
  if (!rearranged && narrowGroups(148, *p, s, opt ? opt->split_k : 0, opt ? unsigned(opt->plan_flags) : 0u, nullptr, nullptr, &rows, &t)) {
    // 64 output channels a block, and with each those of its own group at every tap
    *plan = plb_plan{};
    plan->kernel = 3;
    plan->tile_m = 64;
    plan->tile_n = s.KH * s.KW * rows.chans;
    plan->tile_k_bytes = t.tile_w * t.tile_h * t.tile_n * 2;
    plan->box_w = t.tile_w;
    plan->box_h = t.tile_h;
    plan->box_n = t.tile_n;
    plan->stages = 1;
    plan->split_k = t.splits;
    plan->tiles = rowsWuSlabs(rows);
    plan->grid = plan->tiles * t.splits;
    plan->b_mn_major = 1;
    plan->halo_rows = s.KH - 1;
    plan->workspace_bytes = size_t(t.splits) * p->groups * s.KH * s.KW * rows.chans * rows.chans * sizeof(float);
  }
  plan->flops = 2 * numberOfMacs(*p);
  const uint64_t es = dtypeBytes(p->input_type);
  plan->bytes = es * (uint64_t(p->batch) * s.H * s.W * p->groups * p->in_chans_per_group +
                      uint64_t(p->batch) * s.OH * s.OW * p->groups * p->out_chans_per_group +
                      uint64_t(p->groups) * s.KH * s.KW * p->in_chans_per_group *
                          p->out_chans_per_group);
  return PLB_OK;
}

int plb_conv_wu(plb_context *ctx, const plb_conv_params *p, const plb_conv_options *opt,
                const void *d_acts, const void *d_out_grads, void *d_weight_grads,
                float *d_weight_grads_f32) {
  TraceRange trace_range("plb_conv_wu");
  if (int rc = activate(ctx)) return rc;
  if (!p) return fail(PLB_ERR_INVALID_PARAMS, "null params");
  {
    size_t n_in, n_w, n_out;
    convElementCounts(*p, &n_in, &n_w, &n_out);
    if (n_in == 0 || n_out == 0) n_in = n_out = 0;  // nothing is read: the gradient is zero
    const void *result = d_weight_grads ? d_weight_grads : static_cast<const void *>(d_weight_grads_f32);
    if (int rc = checkConvRequest(*p, true, d_acts, n_w ? n_in : 0, d_out_grads, n_w ? n_out : 0, result, n_w))
      return rc;
  }
  if (p->input_type == PLB_FLOAT && d_weight_grads) {
    // a float layer's weight gradient is float either way
    float *result = d_weight_grads_f32 ? d_weight_grads_f32 : static_cast<float *>(d_weight_grads);
    if (int rc = plb_conv_wu(ctx, p, opt, d_acts, d_out_grads, nullptr, result)) return rc;
    size_t n_in, n_w, n_out;
    convElementCounts(*p, &n_in, &n_w, &n_out);
    if (n_w && d_weight_grads != static_cast<void *>(result))
      PLB_CUDA(cudaMemcpyAsync(d_weight_grads, result, n_w * sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
    return PLB_OK;
  }
  if (p->input_type == PLB_BFLOAT16 && d_weight_grads)
    return fail(PLB_ERR_UNSUPPORTED, "a bfloat16 layer's weight gradient is returned as fp32 only");
  if (p->num_field_dims == 3)
    return conv3dWu(ctx, *p, opt, d_acts, d_out_grads, d_weight_grads, d_weight_grads_f32);
  {
    // a flipped input: reverse it once, then an ordinary weight update
    plb_conv_params q;
    if (unflippedInputParams(*p, &q) && p->num_field_dims <= 2) {
      const std::string err = validate(*p);
      if (!err.empty()) return fail(PLB_ERR_INVALID_PARAMS, err);
      const bool two = p->num_field_dims == 2;
      const uint32_t H = two ? p->field[0] : 1, W = p->field[two ? 1 : 0];
      const size_t px = size_t(p->groups) * p->in_chans_per_group * dtypeBytes(p->input_type);
      void *xf = nullptr;
      if (int rc = scratch(ctx, kSlotFlipped, size_t(p->batch) * H * W * px + 256, &xf)) return rc;
      if (int rc = flipField(ctx, d_acts, xf, p->batch, H, W, px, two && p->in_flip[0],
                             p->in_flip[two ? 1 : 0] != 0))
        return rc;
      return plb_conv_wu(ctx, &q, opt, xf, d_out_grads, d_weight_grads, d_weight_grads_f32);
    }
  }
  {
    // a dilated input: write the zero-stuffed tensor once
    plb_conv_params q;
    DilatedField df;
    if (undilatedInputParams(*p, &q, &df)) {
      const std::string err = validate(*p);
      if (!err.empty()) return fail(PLB_ERR_INVALID_PARAMS, err);
      const size_t px = size_t(p->groups) * p->in_chans_per_group * dtypeBytes(p->input_type);
      void *xd = nullptr;
      if (int rc = scratch(ctx, kSlotDilated, size_t(p->batch) * df.Hd * df.Wd * px + 256, &xd)) return rc;
      if (int rc = dilateField(ctx, d_acts, xd, p->batch, df, px, false)) return rc;
      return plb_conv_wu(ctx, &q, opt, xd, d_out_grads, d_weight_grads, d_weight_grads_f32);
    }
  }
  {
    // A truncated and / or flipped kernel: the gradient of the used taps is
    // that of an ordinary kernel of the truncated extent (with the kernel
    // padding of a flipped dimension swapped), scattered back into the stored
    // filter, whose unused taps get zero.
    bool special = false;
    for (unsigned d = 0; d != p->num_field_dims && d < PLB_MAX_FIELD_DIMS; ++d)
      special |= p->k_trunc_lo[d] || p->k_trunc_hi[d] || p->k_flip[d];
    if (special) {
      const std::string err = validate(*p);
      if (!err.empty()) return fail(PLB_ERR_INVALID_PARAMS, err);
      if (p->num_field_dims > 2)
        return fail(PLB_ERR_UNSUPPORTED, "3-D convolutions are not implemented on this path yet");
      plb_conv_params q = *p;
      int K[2] = {1, 1}, J[2] = {1, 1}, r0[2] = {0, 0}, fl[2] = {0, 0};
      for (unsigned d = 0; d != p->num_field_dims; ++d) {
        const unsigned slot = p->num_field_dims == 2 ? d : 1;  // 1-D: the width
        K[slot] = int(p->kernel[d]);
        J[slot] = int(p->kernel[d]) - int(p->k_trunc_lo[d]) - int(p->k_trunc_hi[d]);
        r0[slot] = int(p->k_trunc_lo[d]);
        fl[slot] = p->k_flip[d] ? 1 : 0;
        q.kernel[d] = uint32_t(J[slot]);
        q.k_trunc_lo[d] = q.k_trunc_hi[d] = 0;
        q.k_flip[d] = 0;
        if (p->k_flip[d]) std::swap(q.k_pad_lo[d], q.k_pad_hi[d]);
      }
      const size_t inner = size_t(p->out_chans_per_group) * p->in_chans_per_group;
      const size_t full = size_t(p->groups) * K[0] * K[1] * inner, used = size_t(p->groups) * J[0] * J[1] * inner;
      const size_t es = dtypeBytes(p->input_type);
      if (d_weight_grads) PLB_CUDA(cudaMemsetAsync(d_weight_grads, 0, full * es, ctx->stream));
      if (d_weight_grads_f32) PLB_CUDA(cudaMemsetAsync(d_weight_grads_f32, 0, full * sizeof(float), ctx->stream));
      if (used == 0 || full == 0) return PLB_OK;
      void *tmp = nullptr;
      const size_t used16 = (used * es + 255) & ~size_t(255);
      if (int rc = scratch(ctx, kSlotUsedTaps, used16 + used * sizeof(float) + 256, &tmp)) return rc;
      void *t16 = tmp;
      float *t32 = reinterpret_cast<float *>(static_cast<uint8_t *>(tmp) + used16);
      if (int rc = plb_conv_wu(ctx, &q, opt, d_acts, d_out_grads, d_weight_grads ? t16 : nullptr,
                               d_weight_grads_f32 ? t32 : nullptr))
        return rc;
      const int grid = int(std::min<size_t>((used + 255) / 256, size_t(ctx->sm_count) * 8));
      if (d_weight_grads) {
        scatterTapsKernel<uint16_t><<<grid, 256, 0, ctx->stream>>>(
            static_cast<const uint16_t *>(t16), static_cast<uint16_t *>(d_weight_grads), int(p->groups),
            K[0], K[1], J[0], J[1], r0[0], r0[1], fl[0], fl[1], inner);
        PLB_CUDA(cudaGetLastError());
        ctx->launches++;
      }
      if (d_weight_grads_f32) {
        scatterTapsKernel<float><<<grid, 256, 0, ctx->stream>>>(
            t32, d_weight_grads_f32, int(p->groups), K[0], K[1], J[0], J[1], r0[0], r0[1], fl[0], fl[1],
            inner);
        PLB_CUDA(cudaGetLastError());
        ctx->launches++;
      }
      return PLB_OK;
    }
  }
  WuShape s;
  if (int rc = wuShape(*p, &s)) return rc;
  const int co = int(p->out_chans_per_group), ci = int(p->in_chans_per_group);
  const int taps = s.KH * s.KW;
  const size_t w_elems = size_t(taps) * co * ci;
  if (p->groups == 0 || w_elems == 0) return PLB_OK;
  if (p->batch == 0 || s.OHc <= 0 || s.OWc <= 0 || s.He <= 0 || s.We <= 0) {
    // empty reduction: the gradient is zero
    const size_t n = size_t(p->groups) * w_elems;
    if (d_weight_grads) PLB_CUDA(cudaMemsetAsync(d_weight_grads, 0, n * dtypeBytes(p->input_type), ctx->stream));
    if (d_weight_grads_f32) PLB_CUDA(cudaMemsetAsync(d_weight_grads_f32, 0, n * sizeof(float), ctx->stream));
    return PLB_OK;
  }
  if (int rc = configureWuKernel(ctx->device)) return rc;
  const int force_split = opt ? opt->split_k : 0;
  const unsigned plan_flags = unsigned((opt ? opt->plan_flags : 0) | ctx->plan_flags);
  WuGather gather{};
  gather.taps = gather.p_taps = uint32_t(taps);
  gather.co = uint32_t(co);
  gather.ci = uint32_t(ci);
  auto run = [&](const WuProblem &q, const WuGather *g, const WuFold *fold = nullptr) -> int {
    WuArgs a{};
    planWu(q, ctx->sm_count, force_split, plan_flags, &a, nullptr);
    a.status = ctx->d_status;
    a.trace = ctx->trace;
    void *ws = nullptr;
    const size_t partial = size_t(a.ksplit) * q.sgroups * q.s.KH * q.s.KW * q.co * q.ci * sizeof(float);
    if (int rc = scratch(ctx, kSlotWuPartials, partial, &ws)) return rc;
    a.partial = static_cast<float *>(ws);
    if (int rc = launchWuKernel(ctx->stream, q, a)) return rc;
    ctx->launches += 2;
    if (fold) {
      WuFold f = *fold;
      f.split_stride = (unsigned long long)q.s.KH * q.co * q.ci;
      cudaLaunchAttribute pdl[1];
      const cudaLaunchConfig_t cfg = wuReduceConfig(ctx->stream, (size_t(f.p_taps) * f.co * 16 + 31) / 32, pdl);
      PLB_CUDA(cudaLaunchKernelEx(&cfg, wu_fold_kernel, (const float *)a.partial, a.ksplit, f, d_weight_grads_f32,
                                  static_cast<__half *>(d_weight_grads)));
      PLB_CUDA(cudaGetLastError());
      return PLB_OK;
    }
    return launchWuReduce(ctx->stream, a, p->groups * w_elems, d_weight_grads, d_weight_grads_f32, g);
  };
  S2dShape g2{};
  WuProblem q;
  // (output gradients off the 16-byte alignment have to be copied: the general form does)
  if ((reinterpret_cast<uintptr_t>(d_out_grads) & 15) == 0 && rearrangedProblem(*p, s, &g2, &q)) {
    void *ws = nullptr;
    if (int rc = scratch(ctx, kSlotOperands, rearrangedBytes(g2), &ws)) return rc;
    if (int rc = smallChannelPrepare(ctx, g2, d_acts, static_cast<__half *>(ws), nullptr, nullptr, co)) return rc;
    q.x = ws;
    q.dy = d_out_grads;
    const WuFold fold{uint32_t(s.KH), uint32_t(s.KW), uint32_t(co), uint32_t(ci), uint32_t(g2.s), uint32_t(g2.Cp),
                      uint32_t(g2.K2h), 0};
    return run(q, nullptr, &fold);
  }
  RowsWuProblem rows;
  RowsWuTiling tiling;
  if (narrowGroups(ctx->sm_count, *p, s, force_split, plan_flags, d_acts, d_out_grads, &rows, &tiling)) {
    WuArgs a{};
    a.sgroups = int(p->groups);
    a.taps_h = s.KH;
    a.taps_w = s.KW;
    a.co_total = co;
    a.ci_total = ci;
    a.ksplit = tiling.splits;
    void *ws = nullptr;
    if (int rc = scratch(ctx, kSlotWuPartials, size_t(tiling.splits) * p->groups * w_elems * sizeof(float), &ws)) return rc;
    a.partial = static_cast<float *>(ws);
    if (int rc = launchRowsWu(ctx, rows, tiling, a.partial)) return rc;
    ctx->launches++;
    return launchWuReduce(ctx->stream, a, p->groups * w_elems, d_weight_grads, d_weight_grads_f32, nullptr);
  }
  const void *x = d_acts, *dy = d_out_grads;
  WuOperands operands;
  q = generalProblem(*p, s, &x, &dy, &operands);
  if (operands.copies) {
    void *ws = nullptr;
    if (int rc = scratch(ctx, kSlotRepacked, operands.bytes + 256, &ws)) return rc;
    for (int i = 0; i < operands.copies; ++i)
      *operands.operand[i] = operands.jobs[i].dst = static_cast<uint8_t *>(ws) + operands.offset[i];
    if (int rc = repack(ctx, operands.jobs, operands.copies)) return rc;
  }
  const WuLayout &l = operands.layout;
  q.x = x;
  q.dy = dy;
  gather.sub = uint32_t(q.sub);
  gather.co_pitch = l.co_pitch;
  gather.ci_pitch = l.ci_pitch;
  gather.p_co = uint32_t(q.co);
  gather.p_ci = uint32_t(q.ci);
  const bool same_order = q.sub == 1 && q.ci == ci && q.co == co;
  return run(q, same_order ? nullptr : &gather);
}

// Chunks (= blocks of the fused reduction, = flags per sender) of one call.
static size_t wuPeerChunks(const plb_conv_params &p, const WuShape &s) {
  const size_t w_elems = size_t(s.KH) * s.KW * p.out_chans_per_group * p.in_chans_per_group;
  return size_t(p.groups) * ((w_elems / 4 + kWuFusedChunk - 1) / kWuFusedChunk);
}

uint64_t plb_conv_wu_allreduce_flag_bytes(const plb_conv_params *p) {
  WuShape s;
  if (!p || p->input_type == PLB_FLOAT || wuShape(*p, &s)) return 0;  // (the fused pass takes half operands)
  // per chunk a word per sender, then a word per chunk for the owner's "sum complete"
  return uint64_t(wuPeerChunks(*p, s)) * (kWuPeerMaxWorld + 1) * sizeof(uint32_t);
}

}  // extern "C"

static int wuAllreduce(plb_context *ctx, const plb_conv_params *p, const plb_conv_options *opt,
                       const void *d_acts, const void *d_out_grads, int32_t rank, int32_t world,
                       void *const *d_peer_grads, void *const *d_peer_results,
                       void *const *d_peer_flags, uint32_t epoch, void *d_weight_grads,
                       float *d_weight_grads_f32) {
  TraceRange trace_range("plb_conv_wu_allreduce");
  if (int rc = activate(ctx)) return rc;
  if (!p) return fail(PLB_ERR_INVALID_PARAMS, "null params");
  if (world < 1 || world > kWuPeerMaxWorld || rank < 0 || rank >= world)
    return fail(PLB_ERR_INVALID_PARAMS, "rank / world size out of range (at most " +
                                            std::to_string(kWuPeerMaxWorld) + " ranks)");
  if (!d_peer_grads || !d_peer_flags) return fail(PLB_ERR_INVALID_PARAMS, "null pointer table");
  if (epoch == 0 || (epoch & 0x80000000u))
    return fail(PLB_ERR_INVALID_PARAMS, "steps are numbered from 1 to 2^31 - 1 (flags start at zero)");
  const char *other = "; use plb_conv_wu and plb_allreduce_f32_p2p for this layer";
  if (p->input_type != PLB_HALF)
    return fail(PLB_ERR_UNSUPPORTED, std::string("plb_conv_wu_allreduce takes half operands") + other);
  WuShape s;
  if (int rc = wuShape(*p, &s)) return rc;   // 1-D / 2-D, half, no input dilation / flip, plain kernel
  const int co = int(p->out_chans_per_group), ci = int(p->in_chans_per_group);
  const size_t w_elems = size_t(s.KH) * s.KW * co * ci;
  if (p->groups == 0 || w_elems == 0) return PLB_OK;
  if (ci % 8 != 0 || co % 8 != 0)
    return fail(PLB_ERR_UNSUPPORTED,
                std::string("the fused weight update needs channel counts that are multiples of 8") + other);
  // all blocks of the reduction wait for their peers' blocks: keep the grid resident
  if (wuPeerChunks(*p, s) / p->groups > size_t(ctx->sm_count) * 4)
    return fail(PLB_ERR_UNSUPPORTED,
                std::string("weight gradient too large for the fused reduction over ranks") + other);
  WuPeerArgs pa{};
  for (int r = 0; r < world; ++r) {
    if (!d_peer_grads[r] || !d_peer_flags[r]) return fail(PLB_ERR_INVALID_PARAMS, "null peer pointer");
    if ((reinterpret_cast<uintptr_t>(d_peer_grads[r]) & 15) != 0)
      return fail(PLB_ERR_INVALID_PARAMS, "peer gradient buffers must be 16-byte aligned");
    pa.grads[r] = static_cast<float4 *>(d_peer_grads[r]);
    pa.flags[r] = static_cast<uint32_t *>(d_peer_flags[r]);
    if (d_peer_results) {
      if (!d_peer_results[r] || (reinterpret_cast<uintptr_t>(d_peer_results[r]) & 15) != 0)
        return fail(PLB_ERR_INVALID_PARAMS, "peer result buffers must be non-null and 16-byte aligned");
      pa.results[r] = static_cast<float4 *>(d_peer_results[r]);
    }
  }
  pa.result_flags = uint32_t(wuPeerChunks(*p, s) * kWuPeerMaxWorld);
  if ((reinterpret_cast<uintptr_t>(d_weight_grads_f32) & 15) != 0 ||
      (reinterpret_cast<uintptr_t>(d_weight_grads) & 7) != 0)
    return fail(PLB_ERR_INVALID_PARAMS, "outputs must be 16-byte (fp32) / 8-byte (half) aligned");
  pa.rank = rank;
  pa.world = world;
  pa.epoch = epoch;
  pa.status = ctx->d_status;
  WuArgs a{};
  a.status = ctx->d_status;
  a.trace = ctx->trace;
  if (int rc = configureWuKernel(ctx->device)) return rc;
  uint64_t launches = 0;
  if (p->batch == 0 || s.OHc <= 0 || s.OWc <= 0 || s.He <= 0 || s.We <= 0) {
    // this rank has no share of the batch: it contributes zeros, through one
    // split of zero partial sums, so that the peers still get its flags
    planWu(wuProblem(*p, s, oneGroup(*p), 1), ctx->sm_count, 1, opt ? opt->plan_flags : 0, &a, nullptr);
    a.ksplit = 1;
    void *ws = nullptr;
    if (int rc = scratch(ctx, kSlotWuPartials, w_elems * sizeof(float), &ws)) return rc;
    PLB_CUDA(cudaMemsetAsync(ws, 0, w_elems * sizeof(float), ctx->stream));
    a.partial = static_cast<float *>(ws);
    for (unsigned g = 0; g < p->groups; ++g) {
      if (int rc = launchWuReduce(
              ctx->stream, a, w_elems,
              d_weight_grads ? static_cast<uint8_t *>(d_weight_grads) + g * w_elems * 2 : nullptr,
              d_weight_grads_f32 ? d_weight_grads_f32 + g * w_elems : nullptr, nullptr, &pa, g))
        return rc;
      ++launches;
    }
    ctx->launches += launches;
    return PLB_OK;
  }
  planWu(wuProblem(*p, s, oneGroup(*p), 1), ctx->sm_count, opt ? opt->split_k : 0,
         opt ? opt->plan_flags : 0, &a, nullptr);
  void *ws = nullptr;
  if (int rc = scratch(ctx, kSlotWuPartials, size_t(a.ksplit) * w_elems * sizeof(float), &ws)) return rc;
  a.partial = static_cast<float *>(ws);
  if (int rc = launchWuPerGroup(ctx->stream, *p, s, a, d_acts, d_out_grads, d_weight_grads, d_weight_grads_f32,
                        &launches, &pa))
    return rc;
  ctx->launches += launches;
  return PLB_OK;
}

extern "C" int plb_conv_wu_allreduce(plb_context *ctx, const plb_conv_params *p,
                                     const plb_conv_options *opt, const void *d_acts,
                                     const void *d_out_grads, int32_t rank, int32_t world,
                                     void *const *d_peer_grads, void *const *d_peer_flags,
                                     uint32_t epoch, void *d_weight_grads,
                                     float *d_weight_grads_f32) {
  return wuAllreduce(ctx, p, opt, d_acts, d_out_grads, rank, world, d_peer_grads, nullptr,
                     d_peer_flags, epoch, d_weight_grads, d_weight_grads_f32);
}

extern "C" int plb_conv_wu_allreduce_owners(plb_context *ctx, const plb_conv_params *p,
                                            const plb_conv_options *opt, const void *d_acts,
                                            const void *d_out_grads, int32_t rank, int32_t world,
                                            void *const *d_peer_grads,
                                            void *const *d_peer_results,
                                            void *const *d_peer_flags, uint32_t epoch,
                                            void *d_weight_grads, float *d_weight_grads_f32) {
  if (!d_peer_results) return fail(PLB_ERR_INVALID_PARAMS, "null pointer table");
  return wuAllreduce(ctx, p, opt, d_acts, d_out_grads, rank, world, d_peer_grads, d_peer_results,
                     d_peer_flags, epoch, d_weight_grads, d_weight_grads_f32);
}

// ---------------------------------------------------------------------------
// Weight update for callers that must not allocate device memory
// ---------------------------------------------------------------------------
// Some callers of this library cannot call cudaMalloc when they need a weight
// gradient: code running inside a framework's allocator hooks or under a
// caching allocator that owns all device memory, real-time loops that may not
// take the allocator's global lock, and processes whose memory budget was fixed
// at start-up.  plb_conv_wu grows a scratch buffer with cudaMalloc on demand;
// this entry point instead keeps the split-K partial sums in a fixed array that
// is part of the library's device image.  Every GPU that loads the library
// holds these bytes until the process exits, so the size is kept modest.

namespace {

constexpr size_t kStaticScratchBytes = size_t(32) << 20;  // 32 MiB
static __device__ __align__(256) unsigned char g_wu_static_scratch[kStaticScratchBytes];
static __device__ int g_wu_static_status;

// Device addresses of the two symbols, looked up once per device.  In host code
// the arrays' names are only host-side handles for the symbols, not device
// addresses: kernels must be given what cudaGetSymbolAddress returns.
struct StaticScratch {
  bool ready = false;
  float *partial = nullptr;
  int *status = nullptr;
  int sm_count = 0;
};
StaticScratch g_static_scratch[64];
std::mutex g_static_scratch_mutex;

int staticScratchFor(int device, StaticScratch *out) {
  if (device < 0 || device >= 64) return fail(PLB_ERR_INVALID_PARAMS, "device ordinal out of range");
  std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
  StaticScratch &s = g_static_scratch[device];
  if (!s.ready) {
    // the caller has made `device` current
    void *scratch_ptr = nullptr, *status_ptr = nullptr;
    PLB_CUDA(cudaGetSymbolAddress(&scratch_ptr, g_wu_static_scratch));
    PLB_CUDA(cudaGetSymbolAddress(&status_ptr, g_wu_static_status));
    PLB_CUDA(cudaDeviceGetAttribute(&s.sm_count, cudaDevAttrMultiProcessorCount, device));
    s.partial = static_cast<float *>(scratch_ptr);
    s.status = static_cast<int *>(status_ptr);
    s.ready = true;
  }
  *out = s;
  return PLB_OK;
}

}  // namespace

extern "C" int plb_conv_wu_static_scratch(int device, void *cuda_stream, const plb_conv_params *p,
                                          const plb_conv_options *opt, const void *d_acts,
                                          const void *d_out_grads, void *d_weight_grads,
                                          float *d_weight_grads_f32) {
  if (!p) return fail(PLB_ERR_INVALID_PARAMS, "null params");
  if (int rc = checkConvRequest(*p, true, nullptr, 0, nullptr, 0, nullptr, 0)) return rc;
  if (p->input_type != PLB_HALF)
    // float operands need scratch for their bfloat16 pieces
    return fail(PLB_ERR_UNSUPPORTED, "plb_conv_wu_static_scratch takes half operands; use plb_conv_wu for this layer");
  PLB_CUDA(cudaSetDevice(device));
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  WuShape s;
  if (int rc = wuShape(*p, &s)) return rc;
  const int co = int(p->out_chans_per_group), ci = int(p->in_chans_per_group);
  const int taps = s.KH * s.KW;
  const size_t w_elems = size_t(taps) * co * ci;
  if (p->groups == 0 || w_elems == 0) return PLB_OK;
  if (w_elems * sizeof(float) > kStaticScratchBytes)
    return fail(PLB_ERR_UNSUPPORTED,
                "weight gradient of " + std::to_string(w_elems * sizeof(float)) +
                    " bytes per group exceeds the " + std::to_string(kStaticScratchBytes) +
                    "-byte static scratch of plb_conv_wu_static_scratch; use plb_conv_wu");
  {
    size_t n_in, n_w, n_out;
    convElementCounts(*p, &n_in, &n_w, &n_out);
    if (n_in == 0 || n_out == 0) n_in = n_out = 0;
    const void *result = d_weight_grads ? d_weight_grads : static_cast<const void *>(d_weight_grads_f32);
    if (int rc = checkConvRequest(*p, true, d_acts, n_in, d_out_grads, n_out, result, n_w)) return rc;
  }
  // This entry point runs none of plb_conv_wu's preparatory passes (they need
  // scratch memory of their own): say so instead of failing inside the launch.
  if (ci % 8 != 0 || co % 8 != 0)
    return fail(PLB_ERR_UNSUPPORTED,
                "plb_conv_wu_static_scratch needs channel counts per group that are multiples of 8 "
                "(plb_conv_wu pads other counts in scratch memory); use plb_conv_wu");
  StaticScratch scratch;
  if (int rc = staticScratchFor(device, &scratch)) return rc;
  if (int rc = configureWuKernel(device)) return rc;
  const size_t es = 2;
  if (p->batch == 0 || s.OHc <= 0 || s.OWc <= 0 || s.He <= 0 || s.We <= 0) {
    const size_t n = size_t(p->groups) * w_elems;
    if (d_weight_grads) PLB_CUDA(cudaMemsetAsync(d_weight_grads, 0, n * es, stream));
    if (d_weight_grads_f32) PLB_CUDA(cudaMemsetAsync(d_weight_grads_f32, 0, n * sizeof(float), stream));
    PLB_CUDA(cudaStreamSynchronize(stream));
    return PLB_OK;
  }
  WuArgs a{};
  planWu(wuProblem(*p, s, oneGroup(*p), 1), scratch.sm_count, opt ? opt->split_k : 0,
         opt ? opt->plan_flags : 0, &a, nullptr);
  // as many K splits as the fixed scratch can hold
  const int max_split = int(kStaticScratchBytes / (w_elems * sizeof(float)));
  a.ksplit = std::max(1, std::min(a.ksplit, max_split));
  a.partial = scratch.partial;
  a.status = scratch.status;
  // the array keeps whatever the previous call left: the status word must start
  // at zero; the partial sums need no clearing, every CTA overwrites its slice
  PLB_CUDA(cudaMemsetAsync(scratch.status, 0, sizeof(int), stream));

  if (int rc = launchWuPerGroup(stream, *p, s, a, d_acts, d_out_grads, d_weight_grads, d_weight_grads_f32,
                        nullptr))
    return rc;
  // report a kernel that gave up on a bounded wait; this also makes the call
  // complete before it returns, so a second call cannot overlap the first
  PLB_CUDA(cudaStreamSynchronize(stream));
  int status = 0;
  PLB_CUDA(cudaMemcpy(&status, scratch.status, sizeof(int), cudaMemcpyDeviceToHost));
  if (status != 0)
    return fail(PLB_ERR_KERNEL, "weight update kernel reported status " + std::to_string(status));
  return PLB_OK;
}
