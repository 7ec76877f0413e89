// Implicit-GEMM contraction kernel for sm_100a.
//
// One kernel serves poplin::matMul and the forward / backward-data passes of
// poplin::convolution (the roles of the reference's ConvPartial1x1Out and
// ConvPartialnx1 codelets, lib/poplin/codelets/ConvPartial1x1Out.cpp:100-180,
// lib/poplin/codelets/ConvPartialnx1.cpp:115-245, together with the partial
// reduction and the cast to the output type that follow them,
// lib/poplin/Convolution.cpp:2762-2816):
//
//   out[pixel, co] = alpha * sum_{tap, ci} act[pixel + offset(tap), ci] * w[tap, co, ci]
//                    (+ beta * addend[pixel, co]) (+ bias[co])
//
// Data layout in HBM: activations NHWC (channels innermost), weights
// [tap][Co][Ci]; a matrix product is the 1x1 case with pixels = rows of A.
//
// Structure: a persistent CTA per SM walks output tiles of 128 pixels x BN
// channels.
//   warps 0..P-1  TMA producers.  One thread each; K step g is issued by
//                 producer g mod P (one 4-D box of the activations and one box
//                 of the weights per step, 128-byte swizzle, zero fill outside
//                 the tensor, which is what implements the padding).  Issuing a
//                 tensor copy costs a thread a few hundred cycles, so a single
//                 producer cannot keep the tensor core fed on narrow tiles.
//   warp 3        issues tcgen05.mma with fp32 accumulators in tensor memory.
//   warp 2        for short tiles not a producer but a second issuer: issuing an
//                 MMA costs its thread about 28 cycles and every tile a few hundred
//                 more in barrier waits and commits, which on a tile of 16
//                 instructions exceeds the 46 cycles the tensor core needs per
//                 instruction.  The two issuers take alternate tiles (and so
//                 always the same accumulator each).  (Not a warp of its own: with
//                 21 warps one of the SM's four register files serves six of them,
//                 which leaves 80 registers per thread; 20 warps leave 96, and the
//                 epilogue needs more than 80.)
//   warps 4..19   epilogue, two groups of eight warps: drain a finished
//                 accumulator (tcgen05.ld), scale / add / cast, stage 32 rows
//                 x 128 bytes per pair of warps in shared memory and hand them
//                 to a TMA store (coalesced, clipped to the tensor by the
//                 hardware); plain vector stores are the fallback when the
//                 output cannot be described to TMA.  The per-warp chain
//                 load -> convert -> stage -> store is latency bound, so the
//                 epilogue's throughput comes from the number of warps.
// Two accumulators alternate so the epilogue of one tile overlaps the main loop
// of the next; accumulator g is always drained by epilogue group g, so a group
// has two tile periods for its tile.
#pragma once

#include "sm100_prims.cuh"

#ifndef PLB_IGEMM_PRODUCERS
#define PLB_IGEMM_PRODUCERS 3
#endif

namespace plb {

constexpr int kTileM = 128;        // pixels (rows) per tile = TMEM lanes
constexpr int kStageKBytes = 128;  // bytes of K per pipeline stage row (one swizzle span)
constexpr int kIgemmThreads = 640;
constexpr int kIgemmProducers = PLB_IGEMM_PRODUCERS;
constexpr int kIgemmMmaWarp = 3;
constexpr int kIgemmMmaWarp2 = 2;  // second MMA issuer (short tiles), else the third producer
constexpr int kEpiStagingBytes = 8 * 4096;  // 8 pairs of epilogue warps x (32 rows x 128 B)
static_assert(kIgemmProducers > kIgemmMmaWarp2 && kIgemmProducers <= 3, "producer warps are warps 0..2");

// Launches that write disjoint parts of one result and read nothing of one another
// (the phases of a strided layer's input gradient) run side by side where SMs are
// free: the first (kChainLead, or any kernel that waits for its predecessor before
// it lets dependents start) orders the others behind everything earlier in the
// stream; the followers do not wait for their predecessor before they read, but
// before they end, so that the completion of the last is the completion of all.
enum IgemmChain : int { kChainNone = 0, kChainLead = 1, kChainFollow = 2 };

struct IgemmArgs {
  // ---- M side: output pixels, tiled by a (w, h, n) box of 128 pixels ------
  int box_w, box_h, box_n;
  int tiles_w, tiles_h, tiles_n;
  int out_w, out_h, out_n;  // extents of the output (matrix product: rows, 1, 1)
  int h_outer;              // rows of a tile are ordered (w, n, h) instead of (w, h, n)
  // Halo mode: one stage holds a strip of box_h + (taps_h-1)*dil_h input rows and
  // serves all taps_h vertical taps (row r starts halo_step_bytes * r further on).
  int halo_step_bytes;
  int a_stage_bytes;        // bytes of activations per stage
  int stage_tx_bytes;       // bytes one CTA's copies bring into a stage
  int a_blocks;             // transposed A: blocks of 64 output rows that exist (1 or 2)
  int b_tiles_per_stage;    // streamed weight tiles per stage (taps_h with a halo strip, else 1)
  // ---- groups ---------------------------------------------------------------
  // Independent contractions of one shape in one launch (channel groups of a
  // convolution, a batch of matrix products).  With more than one, the tensor
  // maps of the activations and the output carry the group as their second
  // dimension (so that a group's channels end where the next group's begin), and
  // group g uses the weight tiles [g * taps, (g + 1) * taps).
  int groups;
  FastDiv fd_groups;
  long long out_group_stride, addend_group_stride;  // elements
  // ---- N side ---------------------------------------------------------------
  int n_tiles;  // tiles of BN output channels
  int n_total;  // valid output channels (of one group)
  int n_mma;    // columns of one instruction: BN, or fewer when one narrow tile covers all
  int b_box_bytes;  // bytes one CTA loads of a streamed or resident weight tile
  // ---- K side ---------------------------------------------------------------
  int taps_h, taps_w;  // filter extent (1 x 1 for a matrix product)
  int k_chunks;        // stages per tap = ceil(bytes of K per tap / 128)
  int k_last;          // instructions (32 bytes of K each) of a tap's last chunk: 1..4
  int pad_h, pad_w;    // tap (r, s) reads input pixel (oh*stride_h + r*dil_h - pad_h, ...)
  int dil_h, dil_w;
  int stride_h, stride_w;  // output pixel oh starts at input row oh*stride_h (TMA traversal stride)
  int flip_h, flip_w;  // tap (r, s) uses the weights stored at (R-1-r, ...) / (..., S-1-s)
  // Tap (r, s) of the (flipped) filter is tile (first_h + r * step_h) * pitch_h +
  // first_w + s * step_w of the taps_stored tiles of a group: a sub-lattice of a
  // stored filter needs no gathering.
  int tap_first_h, tap_step_h, tap_pitch_h, tap_first_w, tap_step_w, taps_stored;
  int group_m;    // tile rasterisation: M tiles per band
  // division by group_m * n_tiles, group_m, tiles_w and (h_outer ? tiles_n : tiles_h)
  FastDiv fd_band, fd_gm, fd_tw, fd_inner;
  int num_stages;  // pipeline depth (<= kIgemmMaxStages)
  // Split-K: split_k CTAs share one output tile, each taking a contiguous range
  // of the tile's pipeline steps and leaving raw fp32 sums in its own slice of
  // a scratch tensor (`out`, split_stride elements apart), which a second
  // kernel adds in split order before the scale / add / cast.  The role of the
  // reference's inChanSplit / kernelSplit partitions and the reduction that
  // follows them (lib/poplin/ConvPlan.hpp:28-77, lib/poplin/ConvReduce.cpp:316-362).
  int split_k;
  FastDiv fd_split;
  long long split_stride;
  int dual_issue;  // two MMA-issuing threads take alternate tiles
  // Steps of a CTA's first unit that idle warps issue, and how many of its steps they
  // pull towards L2 before (streamed weights; the rule is in launchIgemm).
  int first_loads, first_prefetches;
  int chain;       // IgemmChain
  uint32_t idesc_formats;  // operand format bits of the instruction descriptor (8-bit operands: 1 = E5M2)
  // ---- epilogue ---------------------------------------------------------------
  void *out;
  long long ldc;  // elements between consecutive output pixels (along w)
  long long out_stride_h, out_stride_n;  // elements between output rows / images
  const void *addend;
  long long ld_addend;
  const float *bias;
  float alpha, beta;
  int out_is_f32;
  int use_tma_store;        // tm_out is valid: stage through shared memory + TMA store
  int sub_w, sub_h;         // pixel box of one epilogue warp's 32 rows: (sub_w, sub_h, 32/(sub_w*sub_h))
  int *nonfinite;  // set to 1 if a sum is not finite (null: not asked for)
  int *status;
  // Optional timeline (only written by builds with -DPLB_TRACE): CTA 0 stores
  // clock64() stamps, 4096 slots per role (producer 0, MMA issuer, epilogue).
  long long *trace;
};

#ifdef PLB_TRACE
#define PLB_TRACE_STAMP(role, slot)                                            \
  do {                                                                         \
    if (args.trace != nullptr && blockIdx.x == 0 && (slot) < 4096)             \
      args.trace[(role)*4096 + (slot)] = clock64();                            \
  } while (0)
#else
#define PLB_TRACE_STAMP(role, slot) do { } while (0)
#endif

constexpr int kIgemmMaxStages = 8;
constexpr int kIgemmBarrierBytes = 384;
constexpr int kIgemmSmemLimit = 227 * 1024;

// Shared memory: [stages][resident weights][epilogue staging][barriers], after
// up to 1023 bytes of alignment slack.  A stage holds the 128 x 128-byte
// activation tile and, unless the weights are resident, the BN x 128-byte
// weight tile of one K step.
// With a CTA pair (k2Cta) each CTA holds half of the weight tile's rows.
template <int BN, bool kResB, bool k2Cta = false>
struct IgemmSmem {
  static constexpr int kABytes = kTileM * kStageKBytes;  // without a halo
  static constexpr int kBBytes = (BN / (k2Cta ? 2 : 1)) * kStageKBytes;
  static constexpr int kFixedBytes = kEpiStagingBytes + kIgemmBarrierBytes + 1024;
  // b_tiles: streamed weight tiles per stage (1, or with a halo strip one per
  // vertical filter tap)
  __host__ __device__ static constexpr int stageBytes(int a_stage_bytes, int b_tiles) {
    return a_stage_bytes + (kResB ? 0 : b_tiles * kBBytes);
  }
  // deepest pipeline that fits beside `resident` bytes of weights
  static constexpr int stagesFor(int a_stage_bytes, int b_tiles, int resident) {
    const int n =
        (kIgemmSmemLimit - kFixedBytes - resident) / stageBytes(a_stage_bytes, b_tiles);
    return n > kIgemmMaxStages ? kIgemmMaxStages : n;
  }
  static constexpr int totalBytes(int a_stage_bytes, int b_tiles, int stages, int resident) {
    return stages * stageBytes(a_stage_bytes, b_tiles) + resident + kFixedBytes;
  }
};

// kFp8: operands are E4M3 bytes (kind::f8f6f4, 128 elements per stage row,
//       K = 32 per instruction); otherwise fp16 (64 per row, K = 16).
// kBMn: the B operand is stored K-by-N with N contiguous (a row-major right-hand
//       matrix); it is loaded as 64-column blocks and fed to the tensor core as
//       an MN-major operand.  fp16 only.
// kAMn: the same for the left operand of a matrix product, stored K-by-M (a
//       transposed A): two blocks of 64 rows per stage.  fp16, no halo.
// kResB: weight-stationary.  All K steps' weight tiles are loaded once per CTA
//       and stay in shared memory; the pipeline then streams activations only.
//       Used when there is a single N tile and the weights fit (small filters
//       with few channels), where re-fetching them per pixel tile would cost
//       as much shared-memory fill bandwidth as the activations themselves.
//       With several groups the grid is a multiple of their number, so that all
//       units of a CTA belong to one group.
// kHalo: one activation strip per (horizontal tap, channel chunk) feeds all
//       vertical taps: the strip of tap row r is the same shared memory shifted
//       by whole 8-row groups, which the descriptor's start address can express.
//       Cuts the activation traffic of a KxK filter K-fold.  Streamed weights
//       (no kResB) then travel as taps_h tiles per stage.
// kGroups: several groups (args.groups), and a last K chunk of fewer than four
//       instructions.  Without it neither is looked at: the tests for them cost a
//       product of eight K steps 0.9 of 4.5 us.
// k2Cta: the kernel is launched in clusters of two CTAs that share one
//       tcgen05.mma of 256 rows (cta_group::2): the CTA of rank r works on M
//       tile 2 * pair + r, loads its own activations and rows
//       [r * BN/2, (r+1) * BN/2) of the weight tile, and drains its own
//       accumulator.  Rank 0 issues the MMAs; its "full" barriers count the
//       bytes of both CTAs' copies, its "accumulator free" barriers the
//       epilogue threads of both, and its commits release the stages and
//       publish the accumulators in both CTAs.  Halving the weight rows per
//       CTA halves their shared-memory fill and operand fetch per FLOP, and
//       the instruction is twice as large, which matters because a
//       128-row instruction is bound by operand fetch, not by arithmetic.
template <int BN, bool kFp8, bool kAMn, bool kBMn, bool kResB, bool kHalo, bool k2Cta, bool kGroups>
__global__ void __launch_bounds__(kIgemmThreads, 1)
igemm_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
             const __grid_constant__ CUtensorMap tm_out, const IgemmArgs args) {
  using S = IgemmSmem<BN, kResB, k2Cta>;
  static_assert(!k2Cta || !kBMn || BN >= 128, "a CTA needs a whole 64-column block of MN-major B");
  // Copies are issued by warps that walk together, one lane of which copies, so that their operands
  // stay in uniform registers (one thread in a branch of its own moves them there one by one): what
  // they are made from is the same in all lanes, as the compiler sees it.  64 products 256 x 64 x 256
  // 5.5 -> 5.1 us, one 56 x 56 image 5.3 -> 5.0, ragged 197 x 770 x 1003 10.2 -> 9.8.  CTA pairs keep one thread a
  // role: their register budget is used up (3x3 of 128 channels, 256 images of 28 x 28, 45 -> 51 us).
  constexpr bool kWalk = !k2Cta;
  const uint32_t cta_rank = k2Cta ? cluster_cta_rank() : 0u;
  const bool leader = cta_rank == 0;
  constexpr int kMaxStages = kIgemmMaxStages;
  const int kStages = args.num_stages;
  const int P = args.dual_issue ? kIgemmMmaWarp2 : kIgemmProducers;
  constexpr uint32_t kTmemCols = 2 * BN;  // two accumulators
  static_assert(kTmemCols >= 32 && kTmemCols <= 512 && (kTmemCols & (kTmemCols - 1)) == 0, "");
  static_assert(!(kFp8 && (kAMn || kBMn)), "MN-major operands are implemented for fp16 only");
  static_assert(!kAMn || (!kHalo && !kResB), "a transposed A is a plain matrix product");

  extern __shared__ uint8_t smem_raw[];
  if (threadIdx.x == 0) PLB_TRACE_STAMP(2, 4000);
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  // K steps: every (r, s, kc); pipeline steps: in halo mode one per (s, kc)
  const int k_iters = args.taps_h * args.taps_w * args.k_chunks;
  const int p_iters = kHalo ? args.taps_w * args.k_chunks : k_iters;
  const int stage_bytes = S::stageBytes(args.a_stage_bytes, args.b_tiles_per_stage);
  const uint32_t resb_base = smem_base + kStages * stage_bytes;
  const uint32_t staging_base = resb_base + (kResB ? k_iters * S::kBBytes : 0);
  const uint32_t bar_base = staging_base + kEpiStagingBytes;
  // barrier words: full[8], empty[8], tmem_full[2], tmem_empty[2], drain, resident-B
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kMaxStages + s); };
  auto tmem_full_bar = [&](int a) { return bar_base + 8u * (2 * kMaxStages + a); };
  auto tmem_empty_bar = [&](int a) { return bar_base + 8u * (2 * kMaxStages + 2 + a); };
  const uint32_t drain_bar = bar_base + 8u * (2 * kMaxStages + 4);
  const uint32_t drain_bar2 = bar_base + 8u * (2 * kMaxStages + 8);
  const uint32_t resb_bar = bar_base + 8u * (2 * kMaxStages + 5);
  const uint32_t tmem_slot = bar_base + 8u * (2 * kMaxStages + 6);
  uint8_t *bar_gen = smem_raw + (bar_base - smem_u32(smem_raw));
  volatile uint32_t *tmem_slot_ptr =
      reinterpret_cast<volatile uint32_t *>(bar_gen + 8 * (2 * kMaxStages + 6));
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bar_gen + 8 * (2 * kMaxStages + 7));

  const int warp = kWalk ? __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0) : int(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;

  // Set-up is spread over the warps: the lanes of warp 0 initialise the barrier
  // words (one each), a thread of warp 1 asks for the tensor maps, warp 3
  // allocates tensor memory.
  if (warp == 0) {
    // barrier slots: full[8], empty[8], tmem_full[2], tmem_empty[2], drain, resident-B;
    // slot 24: the second issuer's drain
    if (lane == 22) mbar_init(bar_base + 8u * (2 * kMaxStages + 8), 1u);
    if (lane < 2 * kMaxStages + 6) {
      // tmem_empty counts a group's epilogue threads (of both CTAs of a pair)
      const bool acc_free = lane == 2 * kMaxStages + 2 || lane == 2 * kMaxStages + 3;
      mbar_init(bar_base + 8u * lane, acc_free ? (k2Cta ? 512u : 256u) : 1u);
    }
    if (lane == 0) *abort_flag = 0;
    mbar_fence_init();
    if (lane == 0) PLB_TRACE_STAMP(2, 4010);
  } else if (threadIdx.x == 32) {
    tma_prefetch_desc(&tm_a);
    tma_prefetch_desc(&tm_b);
    if (args.use_tma_store) tma_prefetch_desc(&tm_out);
  }
  if (warp == kIgemmMmaWarp) {
    if constexpr (k2Cta) {
      tmem_alloc_pair(tmem_slot, kTmemCols);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, kTmemCols);
      tmem_relinquish();
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0) PLB_TRACE_STAMP(2, 4011);
  // the other CTA's copies and arrivals must find initialised barriers
  // (published by fence.mbarrier_init above)
  if constexpr (k2Cta) cluster_sync_relaxed();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot_ptr;
  // Everything above touched only this SM (barriers, tensor memory): with a
  // programmatic launch it overlaps the tail of the previous kernel in the
  // stream.  Each role goes on preparing what it can without reading or writing
  // global memory (tile coordinates, descriptors, L2 prefetches of the first
  // operands, which have no architectural effect) and calls pdl_wait() itself
  // right before its first access.
  if (threadIdx.x == 0) PLB_TRACE_STAMP(2, 4001);
  if (args.chain == kChainLead) pdl_wait();
  pdl_launch_dependents();
  auto wait_predecessor = [&]() {
    if (args.chain != kChainFollow) pdl_wait();
  };

  // Work units: output tiles, or with a CTA pair, pairs of M tiles (the odd
  // last one is padded: its copies read zeros and its stores are clipped).
  const int m_tiles = args.tiles_w * args.tiles_h * args.tiles_n;
  const int m_units = k2Cta ? (m_tiles + 1) / 2 : m_tiles;
  const int total_tiles = m_units * args.n_tiles * (kGroups ? args.groups : 1);
  // a unit of work is an output tile, or with split-K one of its K ranges
  // (the splits of a tile are consecutive units, i.e. run on different CTAs)
  const int total_units = total_tiles * args.split_k;
  const int first_unit = k2Cta ? int(blockIdx.x >> 1) : int(blockIdx.x);
  const int unit_stride = k2Cta ? int(gridDim.x >> 1) : int(gridDim.x);
  // barriers of the CTA that issues the MMAs, as cluster addresses
  auto lead_bar = [&](uint32_t bar) { return k2Cta ? map_to_cta(bar, 0) : bar; };
  constexpr int kElemsPerStage = kFp8 ? 128 : 64;

  // Tile coordinates are needed once per tile by every producer and epilogue
  // thread; a chain of hardware integer divisions there costs more than a
  // thousand cycles per tile (measured: it paced the producers of short tiles).
  // The divisors are fixed for the launch: divide by multiplication instead.
  // (the multipliers come with the launch arguments: computing them here would
  // put four 64-bit divisions into every thread's prologue)
  const FastDiv fd_band = args.fd_band, fd_gm = args.fd_gm, fd_tw = args.fd_tw, fd_inner = args.fd_inner;

  // unit -> (tile, group, range [it_begin, it_end) of the tile's pipeline steps).
  // The groups of a tile are consecutive units: CTAs working side by side then
  // read neighbouring channels of the same pixels.
  auto unit_coords = [&](int unit, int &tile, int &group, int &split, int &it_begin, int &it_end) {
    if (args.split_k == 1) {
      tile = unit;
      split = 0;
      it_begin = 0;
      it_end = p_iters;
    } else {
      tile = int(fast_div(uint32_t(unit), args.fd_split));
      split = unit - tile * args.split_k;
      it_begin = int(fast_div(uint32_t(p_iters * split), args.fd_split));
      it_end = int(fast_div(uint32_t(p_iters * (split + 1)), args.fd_split));
    }
    group = 0;
    if (kGroups) {
      const int t = int(fast_div(uint32_t(tile), args.fd_groups));
      group = tile - t * args.groups;
      tile = t;
    }
  };
  // tile index -> (m tile, n tile): bands of group_m M tiles, M fastest inside a band
  auto tile_coords = [&](int tile, int &m_idx, int &n_idx) {
    const int band_tiles = args.group_m * args.n_tiles;
    const int band = int(fast_div(uint32_t(tile), fd_band));
    const int within = tile - band * band_tiles;
    const int m0 = band * args.group_m;
    const int gm = min(args.group_m, m_units - m0);
    // (only the last band can be narrower)
    const int q = gm == args.group_m ? int(fast_div(uint32_t(within), fd_gm)) : within / gm;
    m_idx = m0 + within - q * gm;
    n_idx = q;
    if constexpr (k2Cta) m_idx = 2 * m_idx + int(cta_rank);
  };

  // M tile index -> first pixel of the tile; tile row -> pixel inside the tile
  auto tile_origin = [&](int m_idx, int &w0, int &h0, int &n0) {
    const int rest = int(fast_div(uint32_t(m_idx), fd_tw));
    const int tw = m_idx - rest * args.tiles_w;
    const int outer = int(fast_div(uint32_t(rest), fd_inner));
    const int inner = rest - outer * (args.h_outer ? args.tiles_n : args.tiles_h);
    int th, tn;
    if (args.h_outer) {
      tn = inner;
      th = outer;
    } else {
      th = inner;
      tn = outer;
    }
    w0 = tw * args.box_w;
    h0 = th * args.box_h;
    n0 = tn * args.box_n;
  };
  auto row_pixel = [&](int row, int &rw, int &rh, int &rn) {
    rw = row % args.box_w;
    const int rest = row / args.box_w;
    if (args.h_outer) {
      rn = rest % args.box_n;
      rh = rest / args.box_n;
    } else {
      rh = rest % args.box_h;
      rn = rest / args.box_h;
    }
  };

  // B tile of K step (r, s, kc) -> shared memory at `dst`; with kPrefetch the
  // same box is only pulled towards L2.  All lanes of a warp call, the one with `on` copies.
  auto load_b = [&](uint32_t on, uint32_t dst, uint32_t bar, int group, int r, int s, int kc, int n_col, bool prefetch) {
    const int b_tap = ((args.flip_h ? args.taps_h - 1 - r : r) * args.tap_step_h + args.tap_first_h) * args.tap_pitch_h +
                      (args.flip_w ? args.taps_w - 1 - s : s) * args.tap_step_w + args.tap_first_w +
                      (kGroups ? group * args.taps_stored : 0);
    // a CTA of a pair loads its half of the tile's N rows / columns
    constexpr int kMyN = k2Cta ? BN / 2 : BN;
    const int my_col = n_col + (kBMn ? int(cta_rank) * kMyN : k2Cta ? int(cta_rank) * (args.n_mma / 2) : 0);
    if constexpr (kBMn) {
      // K rows x 64 columns per block; blocks of 64 columns are 64 rows apart
#pragma unroll
      for (int j = 0; j < kMyN / 64; ++j) {
        if (!on) {
        } else if (prefetch)
          tma_prefetch_l2_3d(&tm_b, my_col + j * 64, kc * 64, b_tap);
        else if constexpr (k2Cta)
          tma_load_3d_pair(dst + j * (64 * kStageKBytes), &tm_b, bar, my_col + j * 64, kc * 64,
                           b_tap);
        else
          tma_load_3d(dst + j * (64 * kStageKBytes), &tm_b, bar, my_col + j * 64, kc * 64, b_tap);
      }
    } else {
      if (!on) {
      } else if (prefetch)
        tma_prefetch_l2_3d(&tm_b, kc * kElemsPerStage, my_col, b_tap);
      else if constexpr (k2Cta)
        tma_load_3d_pair(dst, &tm_b, bar, kc * kElemsPerStage, my_col, b_tap);
      else
        tma_load_3d(dst, &tm_b, bar, kc * kElemsPerStage, my_col, b_tap);
    }
  };
  // pipeline step index inside a tile -> (filter row, filter column, channel chunk)
  auto step_coords = [&](int it, int &r, int &s, int &kc) {
    kc = it % args.k_chunks;
    const int t = it / args.k_chunks;
    s = t % args.taps_w;
    r = t / args.taps_w;
  };
  // the barriers that count copied bytes are those of the MMA-issuing CTA,
  // which alone announces the byte count (both CTAs' shares)
  constexpr uint32_t kPairFactor = k2Cta ? 2u : 1u;

  // One pipeline step: the activation box and, unless the weights are
  // resident, the weight tile(s) of step (r, s, kc) -> stage memory at a_dst
  // (or, before the predecessor kernel is known to have finished, only
  // towards L2).
  auto issue_step = [&](uint32_t on, bool prefetch, uint32_t a_dst, uint32_t full, int group, int r, int s, int kc,
                        int w_base, int h_base, int n0, int n_col) {
    if constexpr (kAMn) {
      // [k][m] rows of one group: two boxes of 64 K rows x 64 output rows
        for (int j = 0; j < args.a_blocks; ++j) {
        if (!on) {
        } else if (prefetch)
          tma_prefetch_l2_3d(&tm_a, w_base + j * 64, kc * 64, group);
        else if constexpr (k2Cta)
          tma_load_3d_pair(a_dst + j * (64 * kStageKBytes), &tm_a, full, w_base + j * 64, kc * 64, group);
        else
          tma_load_3d(a_dst + j * (64 * kStageKBytes), &tm_a, full, w_base + j * 64, kc * 64, group);
      }
    } else {
      const int cw = w_base + s * args.dil_w, ch = h_base + r * args.dil_h;
      const int c2 = args.h_outer ? n0 : ch, c3 = args.h_outer ? ch : n0;
      const int ck = kc * kElemsPerStage;
      if (!on) {
      } else if (kGroups) {
        if (prefetch)
          tma_prefetch_l2_5d(&tm_a, ck, group, cw, c2, c3);
        else if constexpr (k2Cta)
          tma_load_5d_pair(a_dst, &tm_a, full, ck, group, cw, c2, c3);
        else
          tma_load_5d(a_dst, &tm_a, full, ck, group, cw, c2, c3);
      } else if (prefetch) {
        tma_prefetch_l2_4d(&tm_a, ck, cw, c2, c3);
      } else if constexpr (k2Cta) {
        tma_load_4d_pair(a_dst, &tm_a, full, ck, cw, c2, c3);
      } else {
        tma_load_4d(a_dst, &tm_a, full, ck, cw, c2, c3);
      }
    }
    if constexpr (!kResB) {
      // with a halo strip the stage carries the weight tiles of every filter row
      const int row_taps = kHalo ? args.taps_h : 1;
      for (int rr = 0; rr < row_taps; ++rr)
        load_b(on, a_dst + args.a_stage_bytes + rr * S::kBBytes, full, group, kHalo ? rr : r, s, kc, n_col,
               prefetch);
    }
  };
  // The pipeline is empty when the kernel starts, and a copy costs its issuing
  // thread a few hundred cycles: the first unit's first steps, one per stage, are
  // issued by as many warps at once, the epilogue warps, which have nothing to do
  // yet.  (With resident weights those load the weights, and the producers start
  // on the activations themselves.)
  int first_steps = 0;
  int f_tile = 0, f_group = 0, f_split = 0, f_begin = 0, f_end = 0;
  if (first_unit < total_units) {
    unit_coords(first_unit, f_tile, f_group, f_split, f_begin, f_end);
    first_steps = min(f_end - f_begin, kStages);
  }
  const int first_loads = min(first_steps, args.first_loads), first_prefetches = min(first_steps, args.first_prefetches);
  // Step f_begin + i of the first unit towards L2 while the predecessor kernel may
  // still be running, and with `load`, once it has finished, into stage i.
  auto first_step = [&](uint32_t on, int i, bool load) {
    int m_idx, n_idx, w0, h0, n0, r, s, kc;
    tile_coords(f_tile, m_idx, n_idx);
    tile_origin(m_idx, w0, h0, n0);
    step_coords(f_begin + i, r, s, kc);
    const uint32_t dst = smem_base + i * stage_bytes, full = lead_bar(full_bar(i));
    const int w_base = w0 * args.stride_w - args.pad_w, h_base = h0 * args.stride_h - args.pad_h;
    if (kResB || i < first_prefetches) issue_step(on, true, dst, full, f_group, r, s, kc, w_base, h_base, n0, n_idx * BN);
    if (!load) return;
    wait_predecessor();
    if (leader && on)
      mbar_expect_tx(full_bar(i), kPairFactor * uint32_t(args.stage_tx_bytes));
    issue_step(on, false, dst, full, f_group, r, s, kc, w_base, h_base, n0, n_idx * BN);
  };

  if (warp < P) {
    // ===================== TMA producers =====================
    const uint32_t on = elect_one() ? 1u : 0u;
    auto wait = [&](uint32_t bar, uint32_t parity) {
      const bool done = mbar_wait(bar, parity, abort_flag);
      return kWalk ? __all_sync(0xffffffffu, done) != 0 : done;
    };
    if (kWalk || on) {
      const int me = warp;
      int stage = me;          // stage of this producer's next K step
      uint32_t phase = 0;
      int turn = 0;            // (global K step) mod P
      bool ok = true;
      [[maybe_unused]] int trace_slot = 0;
      if constexpr (kResB)
        for (int i = me; i < first_steps; i += P) first_step(on, i, false);
      wait_predecessor();
      if (me == 0) PLB_TRACE_STAMP(2, 4002);
      for (int unit = first_unit; unit < total_units && ok; unit += unit_stride) {
        if (me == 0) { PLB_TRACE_STAMP(0, trace_slot); ++trace_slot; }
        int tile, group, split, it_begin, it_end;
        unit_coords(unit, tile, group, split, it_begin, it_end);
        int m_idx, n_idx;
        tile_coords(tile, m_idx, n_idx);
        int w0, h0, n0;
        tile_origin(m_idx, w0, h0, n0);
        if (me == 0) { PLB_TRACE_STAMP(0, trace_slot); ++trace_slot; }
        const int w_base = w0 * args.stride_w - args.pad_w;
        const int h_base = h0 * args.stride_h - args.pad_h;
        const int n_col = n_idx * BN;
        int r = 0, s = 0, kc = 0;
        if (it_begin != 0) step_coords(it_begin, r, s, kc);
        for (int it = it_begin; it < it_end; ++it) {
          // (the first unit's first steps are on their way already)
          const bool issued = !kResB && unit == first_unit && it - it_begin < first_loads;
          if (turn == me && issued) {
            stage += P;
            if (stage >= kStages) {
              stage -= kStages;
              phase ^= 1u;
            }
          } else if (turn == me) {
            if (me == 0) { PLB_TRACE_STAMP(0, trace_slot); ++trace_slot; }
            if (!wait(empty_bar(stage), phase ^ 1u)) {
              atomicCAS(args.status, kStatusOk, kStatusProducerTimeout);
              ok = false;
              break;
            }
            if (me == 0) { PLB_TRACE_STAMP(0, trace_slot); ++trace_slot; }
            const uint32_t a_dst = smem_base + stage * stage_bytes;
            if (leader && on) mbar_expect_tx(full_bar(stage), kPairFactor * uint32_t(args.stage_tx_bytes));
            const uint32_t full = lead_bar(full_bar(stage));
            issue_step(on, false, a_dst, full, group, r, s, kc, w_base, h_base, n0, n_col);
            if (me == 0) { PLB_TRACE_STAMP(0, trace_slot); ++trace_slot; }
            stage += P;
            if (stage >= kStages) {
              stage -= kStages;
              phase ^= 1u;
            }
          }
          if (++turn == P) turn = 0;
          // next pipeline step: kc fastest, then s, then (without a halo) r
          if (++kc == args.k_chunks) {
            kc = 0;
            if (++s == args.taps_w) {
              s = 0;
              ++r;
            }
          }
        }
      }
      if constexpr (k2Cta) {
        // The leader's commits arrive on this CTA's barriers too: it must not leave, and
        // its shared memory not become another block's, before the last of them has.
        // (the producer whose turn it would be: its stage and phase are the next step's)
        if (!leader && ok && turn == me)
          for (int i = 0; i < kStages && ok; ++i) {
            ok = wait(empty_bar(stage), phase ^ 1u);
            if (!ok) atomicCAS(args.status, kStatusOk, kStatusDrainTimeout);
            if (++stage == kStages) {
              stage = 0;
              phase ^= 1u;
            }
          }
      }
      if (me == 0) PLB_TRACE_STAMP(2, 4014);
    }
  } else if (warp <= kIgemmMmaWarp) {
    // ===================== MMA issuer(s) =====================
    // (with a CTA pair only the CTA of rank 0 issues)
    const int mi = warp == kIgemmMmaWarp ? 0 : 1;
    const int n_issuers = args.dual_issue ? 2 : 1;
    if (mi < n_issuers && leader && elect_one()) {
      const uint32_t idesc =
          make_idesc(k2Cta ? 2 * kTileM : kTileM, uint32_t(args.n_mma), 0, 0, kAMn, kBMn) | args.idesc_formats;
      // completion of the MMAs issued so far -> barrier (in both CTAs of a pair)
      auto commit = [&](uint32_t bar) {
        if constexpr (k2Cta)
          umma_commit_pair(bar, uint16_t(3));
        else
          umma_commit(bar);
      };
      const uint64_t a_desc0 = make_smem_desc(smem_base, kAMn ? 64 * kStageKBytes : 16, 1024);
      // B tiles: resident ones start at resb_base, streamed ones follow the
      // activations inside their stage
      const uint64_t b_desc0 =
          kBMn ? make_smem_desc(kResB ? resb_base : smem_base + uint32_t(args.a_stage_bytes),
                                64 * kStageKBytes, 1024)
               : make_smem_desc(kResB ? resb_base : smem_base + uint32_t(args.a_stage_bytes), 16,
                                1024);
      [[maybe_unused]] const uint64_t halo_step16 = uint64_t(uint32_t(args.halo_step_bytes) >> 4);
      // weight tile of the next filter row: resident tiles are indexed (r, s, kc),
      // streamed ones follow one another inside the stage
      [[maybe_unused]] const uint64_t b_row_step16 =
          uint64_t(uint32_t(kResB ? args.taps_w * args.k_chunks : 1) * (S::kBBytes >> 4));
      int stage = 0;
      uint32_t phase = 0;
      uint32_t acc_phases = 0;  // a bit per accumulator (an array would lie in local memory)
      int local_tile = 0;
      bool ok = true;
      [[maybe_unused]] int trace_slot = 0;
      if (kResB && first_unit < total_units) {
        if (!mbar_wait(resb_bar, 0, abort_flag)) {
          atomicCAS(args.status, kStatusOk, kStatusMmaTimeout);
          ok = false;
        }
      }
      for (int unit = first_unit; unit < total_units && ok; unit += unit_stride, ++local_tile) {
        int tile, group, split, it_begin, it_end;
        unit_coords(unit, tile, group, split, it_begin, it_end);
        if (n_issuers == 2 && (local_tile & 1) != mi) {
          // the other issuer's tile: step over its pipeline stages
          stage += it_end - it_begin;
          while (stage >= kStages) {
            stage -= kStages;
            phase ^= 1u;
          }
          continue;
        }
        const int acc = local_tile & 1;
        if (mi == 0) { PLB_TRACE_STAMP(1, trace_slot); ++trace_slot; }
        // wait for the epilogue to have drained this accumulator
        if (!mbar_wait(tmem_empty_bar(acc), ((acc_phases >> acc) & 1u) ^ 1u, abort_flag)) {
          atomicCAS(args.status, kStatusOk, kStatusMmaTimeout);
          ok = false;
          break;
        }
        acc_phases ^= 1u << acc;
        tc_fence_after_sync();
        if (mi == 0) { PLB_TRACE_STAMP(1, trace_slot); ++trace_slot; }
        const uint32_t d_tmem = tmem_base + acc * BN;
        int s_tap = 0, kc = 0;  // halo mode: pipeline step = (s_tap, kc), kc fastest
        if (it_begin != 0) {
          kc = it_begin % args.k_chunks;
          s_tap = it_begin / args.k_chunks;
        }
        for (int it = it_begin; it < it_end; ++it) {
          if (!mbar_wait(full_bar(stage), phase, abort_flag)) {
            atomicCAS(args.status, kStatusOk, kStatusMmaTimeout);
            ok = false;
            break;
          }
          tc_fence_after_sync();
          if (mi == 0) { PLB_TRACE_STAMP(1, trace_slot); ++trace_slot; }
          // Descriptors are advanced by adding to their start-address field
          // (16-byte units, cannot overflow for shared-memory addresses): the
          // issuing thread's own instruction count bounds the MMA rate on
          // narrow tiles.
          const uint32_t stage_off16 = uint32_t(stage * stage_bytes) >> 4;
          uint64_t a_desc = a_desc0 + stage_off16;
          uint64_t b_desc;
          if constexpr (kHalo && kResB)
            b_desc = b_desc0 + uint64_t((s_tap * args.k_chunks + kc) * (S::kBBytes >> 4));
          else if constexpr (kResB)
            b_desc = b_desc0 + uint64_t(it * (S::kBBytes >> 4));
          else
            b_desc = b_desc0 + stage_off16;
          const int row_taps = kHalo ? args.taps_h : 1;
          // one instruction consumes 32 bytes of K: the start address advances inside
          // the swizzle span (K-major) or by 16 rows (MN-major)
          auto mma = [&](int r, int k) {
            const uint64_t a_k = a_desc + uint64_t(kAMn ? k * ((16 * kStageKBytes) >> 4) : k * 2);
            const uint64_t b_k = b_desc + uint64_t(kBMn ? k * ((16 * kStageKBytes) >> 4) : k * 2);
            if constexpr (k2Cta)
              umma_ss_pair<kFp8>(d_tmem, a_k, b_k, idesc, ((it - it_begin) | r | k) != 0 ? 1u : 0u);
            else
              umma_ss<kFp8>(d_tmem, a_k, b_k, idesc, ((it - it_begin) | r | k) != 0 ? 1u : 0u);
          };
          // (the K range past the last channel holds zeros: no instruction for it)
          const int k_steps = kGroups && kc == args.k_chunks - 1 ? args.k_last : 4;
          for (int r = 0; r < row_taps; ++r) {
            if (k_steps == 4) {
#pragma unroll
              for (int k = 0; k < 4; ++k) mma(r, k);
            } else {
              for (int k = 0; k < k_steps; ++k) mma(r, k);
            }
            if constexpr (kHalo) {
              // next filter row: the strip shifted by whole 8-row groups; its
              // resident weight tile is taps_w * k_chunks tiles further on
              a_desc += halo_step16;
              b_desc += b_row_step16;
            }
          }
          commit(empty_bar(stage));  // frees the stage when these MMAs retire
          if (mi == 0) { PLB_TRACE_STAMP(1, trace_slot); ++trace_slot; }
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
          if (++kc == args.k_chunks) {
            kc = 0;
            ++s_tap;
          }
        }
        if (ok) commit(tmem_full_bar(acc));
      }
      // make sure nothing is still executing before TMEM is released
      const uint32_t my_drain = mi == 0 ? drain_bar : drain_bar2;
      if constexpr (k2Cta)
        umma_commit_pair(my_drain, uint16_t(1));
      else
        umma_commit(my_drain);
      const long long start = clock64();
      while (!mbar_try_wait(my_drain, 0)) {
        if (clock64() - start > kWaitCycleLimit) {
          atomicCAS(args.status, kStatusOk, kStatusDrainTimeout);
          break;
        }
      }
      if constexpr (k2Cta) {
        // Likewise the other CTA's epilogue threads arrive here when they have read a tile
        // (the rendezvous below does not order that): each accumulator's last tile is
        // waited for as the next one's first instruction would.
        for (int acc = 0; acc < 2; ++acc)
          if (ok && (n_issuers == 1 || acc == mi) &&
              !mbar_wait(tmem_empty_bar(acc), ((acc_phases >> acc) & 1u) ^ 1u, abort_flag)) {
            atomicCAS(args.status, kStatusOk, kStatusDrainTimeout);
            ok = false;
          }
      }
      if (mi == 0) PLB_TRACE_STAMP(2, 4015);
    }
  } else {
    // ===================== epilogue (warps 4..19) =====================
    // Accumulator g is drained by the eight warps of group g.  A warp can read
    // the 32 TMEM lanes (tile rows) [32*(warp%4), +32); the two warps that share
    // a lane quarter split every block of 64 columns between them (columns
    // [0,32) and [32,64) of the block), each staging and storing its own half.
    const int group = (warp - 4) >> 3;       // drains accumulator `group`
    const int half = ((warp - 4) >> 2) & 1;  // which 32 columns of each 64-column block
    const int quarter = warp & 3;            // TMEM lanes [32*quarter, 32*quarter+32)
    const int row = quarter * 32 + lane;     // tile row handled by this thread
    uint32_t acc_phase = 0;
    int rw, rh, rn;
    row_pixel(row, rw, rh, rn);
    // origin of this warp's 32 rows inside the tile's pixel box
    int qw, qh, qn;
    row_pixel(quarter * 32, qw, qh, qn);
    // fp32 output: one 32-row x 128-byte staging buffer per lane quarter of a
    // group (a second one was measured: it costs a pipeline stage and hides
    // nothing, the chain below is bound by its own instructions, not by the
    // store reading the buffer)
    const uint32_t buf = staging_base + uint32_t(group * 4 + quarter) * 4096u;
    const uint32_t row_addr = buf + uint32_t(lane) * 128u;
    const bool tma_store = args.use_tma_store != 0;
    const bool out_f32 = args.out_is_f32 != 0;
    // fp32 rows fill the 128-byte staged row with 32 columns: the `half == 1`
    // warps then leave the work to their partners
    const bool idle = out_f32 && args.split_k == 1 && half == 1;
    const bool lean = tma_store && !out_f32 && args.bias == nullptr && args.addend == nullptr && args.nonfinite == nullptr;
    const bool stamp = threadIdx.x == 128;
    const int acc = group;
    int local_tile = group;
    const uint32_t acc_free_bar = lead_bar(tmem_empty_bar(acc));
    if constexpr (kResB) {
      // Resident weights: a single N tile, so every tile of this CTA uses the
      // same weights.  The epilogue warps have nothing to do until the first
      // accumulator is complete, so one lane of each issues a share of the
      // copies (a copy costs its issuing thread some hundred cycles, and the
      // first MMA waits for all of them), leaving the producers free to start
      // on the activations at once.
      const uint32_t on = elect_one() ? 1u : 0u;
      if ((kWalk || on) && first_unit < total_units) {
        for (int it = warp - 4; it < k_iters; it += 16) {
          int r, s, kc;
          step_coords(it, r, s, kc);
          load_b(on, 0u, 0u, f_group, r, s, kc, 0, true);
        }
        wait_predecessor();
        if (warp == 4 && leader && on)
          mbar_expect_tx(resb_bar, kPairFactor * uint32_t(k_iters * args.b_box_bytes));
        const uint32_t resb_bar_lead = lead_bar(resb_bar);
        for (int it = warp - 4; it < k_iters; it += 16) {
          int r, s, kc;
          step_coords(it, r, s, kc);
          load_b(on, resb_base + it * S::kBBytes, resb_bar_lead, f_group, r, s, kc, 0, false);
        }
        if (warp == 4) PLB_TRACE_STAMP(2, 4012);
      }
      __syncwarp();
    } else {
      const uint32_t on = elect_one() ? 1u : 0u;
      if ((kWalk || on) && warp - 4 < max(first_loads, first_prefetches)) first_step(on, warp - 4, warp - 4 < first_loads);
      __syncwarp();
    }
    wait_predecessor();
    for (int unit = first_unit + group * unit_stride; unit < total_units;
         unit += 2 * unit_stride, local_tile += 2) {
      int tile, cgroup, split, it_begin, it_end;
      unit_coords(unit, tile, cgroup, split, it_begin, it_end);
      int m_idx, n_idx;
      tile_coords(tile, m_idx, n_idx);
      int w0, h0, n0;
      tile_origin(m_idx, w0, h0, n0);
      const int ow = w0 + rw, oh = h0 + rh, on = n0 + rn;
      const bool row_ok = ow < args.out_w && oh < args.out_h && on < args.out_n;
      // element offset of this row's output pixel; the addend is dense in pixels
      const long long pixel = (static_cast<long long>(on) * args.out_h + oh) * args.out_w + ow;
      const long long out_off = static_cast<long long>(on) * args.out_stride_n +
                                static_cast<long long>(oh) * args.out_stride_h +
                                static_cast<long long>(ow) * args.ldc + (kGroups ? cgroup * args.out_group_stride : 0);
      if (stamp) PLB_TRACE_STAMP(2, local_tile * 4 + 0);
      if (!mbar_wait(tmem_full_bar(acc), acc_phase, abort_flag)) {
        atomicCAS(args.status, kStatusOk, kStatusEpilogueTimeout);
        break;
      }
      acc_phase ^= 1u;
      tc_fence_after_sync();
      if (stamp) PLB_TRACE_STAMP(2, local_tile * 4 + 1);
      const uint32_t t_addr = tmem_base + acc * BN + (static_cast<uint32_t>(quarter * 32) << 16);
      const int col_base = n_idx * BN;
      // columns of the tile that exist, in blocks of 32
      const int cols_end = min(BN, (args.n_total - col_base + 31) & ~31);
      const bool box_ok = w0 + qw < args.out_w && h0 + qh < args.out_h && n0 + qn < args.out_n;
      auto release_accumulator = [&]() {
        tc_fence_before_sync();
        if constexpr (k2Cta)
          mbar_arrive_cluster(acc_free_bar);
        else
          mbar_arrive(acc_free_bar);
      };
      if (idle) {
        release_accumulator();
        continue;
      }

      // this warp's staged rows of 32 columns from `col` on -> output
      auto store_staged = [&](uint32_t src, int col) {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          // a box that starts outside the tensor has nothing to write
          if (box_ok) {
            const int c2 = args.h_outer ? n0 + qn : h0 + qh, c3 = args.h_outer ? h0 + qh : n0 + qn;
            if (kGroups)
              tma_store_5d(&tm_out, src, col, cgroup, w0 + qw, c2, c3);
            else
              tma_store_4d(&tm_out, src, col, w0 + qw, c2, c3);
          }
          tma_store_commit();
        }
      };
      auto note_nonfinite = [&](const uint32_t (&v)[32], int valid) {
        // (rows beyond the output hold whatever the stage's shared memory held before)
        if (args.nonfinite == nullptr || !row_ok) return;
        uint32_t largest = 0u;
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (j < valid) largest = max(largest, v[j] & 0x7fffffffu);
        if (largest >= 0x7f800000u) *args.nonfinite = 1;
      };

      // The accumulator in blocks of 32 columns, in one of three loops:
      //  - the general one: scale / add, then the block is staged in swizzled shared
      //    memory (half: each warp its own 32 rows x 64 bytes, so that no barrier between
      //    warps lies on the chain load -> convert -> stage -> store; fp32: 32 rows x
      //    128 bytes) and leaves with a tensor store, or, where the output cannot be
      //    described to TMA, row by row: lane after lane writing its own row would
      //    touch a sector per element, consecutive lanes take consecutive columns
      //    instead;
      //  - the fp32 sums of a K split: vector stores of each lane's own row (the
      //    scratch rows are padded to whole blocks);
      //  - a half result that only has to be scaled and stored (products without C,
      //    input gradients).
      // As one loop for all of them it needed more than 96 registers: what was spilled
      // (420 sectors a CTA) and the branches around what a product does not have cost
      // 512 x 512 x 512 0.3 of 4.6 us.  The general one comes first, with nothing of the
      // others between its instructions (7x7 layer on 64 images 49.4 us behind them, 48.8).
      const uint32_t wbuf = staging_base + uint32_t(warp - 4) * 2048u;
      const uint32_t wrow = wbuf + uint32_t(lane) * 64u, sw = (uint32_t(lane) >> 1) & 3u;
      const bool whole_rows = out_f32 && args.split_k == 1;  // 128-byte rows, the half == 0 warps only
      const int c_first = whole_rows ? 0 : half * 32, c_step = whole_rows ? 32 : 64;
      if (c_first >= cols_end) release_accumulator();
      if (!lean && args.split_k == 1) {
#pragma unroll 1
      for (int c = c_first; c < cols_end; c += c_step) {
        uint32_t v[32];
        float f[32];
        __syncwarp();
        tmem_ld_32x32(t_addr + c, v);
        tmem_ld_wait_for(v);
        if (c + c_step >= cols_end) release_accumulator();
        const int col0 = col_base + c;
        const int valid = min(32, args.n_total - col0);
        note_nonfinite(v, valid);
        if (args.alpha != 1.f) {
#pragma unroll
          for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]) * args.alpha;
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
        }
        if (args.bias != nullptr) {
          // (the same addresses in every lane: one 16-byte broadcast per four columns;
          // as 32 predicated words the bias cost the 7x7 layer 60 of 180 us)
          const float *bias = args.bias + cgroup * args.n_total + col0;
          if (valid == 32 && (reinterpret_cast<uintptr_t>(bias) & 15) == 0) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              const float4 b4 = *reinterpret_cast<const float4 *>(bias + j);
              f[j] += b4.x;
              f[j + 1] += b4.y;
              f[j + 2] += b4.z;
              f[j + 3] += b4.w;
            }
          } else if (valid % 4 == 0 && (reinterpret_cast<uintptr_t>(bias) & 15) == 0) {
            // (the last, narrower block: apart, so that the whole one has all its loads in
            // flight at once; 1x1 layer of 24 channels on 34 images of 35 x 22 8.1 -> 6.7 us)
#pragma unroll
            for (int j = 0; j < 28; j += 4) {
              if (j >= valid) break;
              const float4 b4 = *reinterpret_cast<const float4 *>(bias + j);
              f[j] += b4.x;
              f[j + 1] += b4.y;
              f[j + 2] += b4.z;
              f[j + 3] += b4.w;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j < valid) f[j] += bias[j];
          }
        }
        if (args.addend != nullptr && row_ok) {
          const long long at = pixel * args.ld_addend + cgroup * args.addend_group_stride + col0;
          if (out_f32) {
            const float *src = static_cast<const float *>(args.addend) + at;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j < valid) f[j] += args.beta * src[j];
          } else {
            const __half *src = static_cast<const __half *>(args.addend) + at;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j < valid) f[j] += args.beta * __half2float(src[j]);
          }
        }
        if (tma_store && lane == 0) tma_store_wait_read<0>();  // the previous store has read the buffer
        __syncwarp();
        if (whole_rows) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            st_shared_v4(row_addr + (uint32_t(j ^ (lane & 7)) << 4), __float_as_uint(f[4 * j]),
                         __float_as_uint(f[4 * j + 1]), __float_as_uint(f[4 * j + 2]),
                         __float_as_uint(f[4 * j + 3]));
        } else {
          // 16-byte pieces XOR-swizzled with bits 1-2 of the row index: the tensor
          // map's 64-byte swizzle, free of bank conflicts
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t pk[4];
            pack_half8(f + 8 * j, pk);
            st_shared_v4(wrow + ((uint32_t(j) ^ sw) << 4), pk[0], pk[1], pk[2], pk[3]);
          }
        }
        if (tma_store) {
          store_staged(whole_rows ? buf : wbuf, col0);
          continue;
        }
        __syncwarp();
        // fp32: a row of 32 columns per instruction; half: two rows of 16 words.
        // Four instructions' words and row offsets first, then their stores: one at
        // a time is a chain of latencies (3.7 of 14.8 us on a 77x293 fp32 output).
        const uint32_t lo = uint32_t(out_off), hi = row_ok ? uint32_t(out_off >> 32) : 0x80000000u;
        const uint8_t *staged = smem_raw + ((whole_rows ? buf : wbuf) - smem_u32(smem_raw));
        const int cc = whole_rows ? lane : 2 * (lane & 15);
        const uint32_t piece = uint32_t(whole_rows ? lane : lane & 15) >> 2, word = (uint32_t(lane) & 3u) << 2;
#pragma unroll 1
        for (int i0 = 0; i0 < (whole_rows ? 32 : 16); i0 += 4) {
          uint32_t bits[4], off_hi[4], off_lo[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int r = whole_rows ? i0 + u : 2 * (i0 + u) + (lane >> 4);
            bits[u] = *reinterpret_cast<const uint32_t *>(
                staged + (whole_rows ? uint32_t(r) * 128u + ((piece ^ (uint32_t(r) & 7u)) << 4)
                                     : uint32_t(r) * 64u + ((piece ^ ((uint32_t(r) >> 1) & 3u)) << 4)) + word);
            off_hi[u] = __shfl_sync(0xffffffffu, hi, r);
            off_lo[u] = __shfl_sync(0xffffffffu, lo, r);
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (int32_t(off_hi[u]) < 0 || cc >= valid) continue;
            const long long off = (long long)(uint64_t(off_hi[u]) << 32 | off_lo[u]) + col0 + cc;
            if (out_f32) {
              static_cast<uint32_t *>(args.out)[off] = bits[u];
            } else {
              uint16_t *dst = static_cast<uint16_t *>(args.out) + off;
              if (cc + 1 < valid && (reinterpret_cast<uintptr_t>(dst) & 3) == 0) {
                *reinterpret_cast<uint32_t *>(dst) = bits[u];
              } else {
                dst[0] = uint16_t(bits[u]);
                if (cc + 1 < valid) dst[1] = uint16_t(bits[u] >> 16);
              }
            }
          }
        }
        __syncwarp();
      }
        continue;
      }
      if (args.split_k > 1) {
        // (this split's slice of the partial sums, whole 32-byte sectors per lane)
        float *const dst = static_cast<float *>(args.out) + split * args.split_stride + out_off + col_base;
#pragma unroll 1
        for (int c = c_first; c < cols_end; c += 64) {
          uint32_t v[32];
          __syncwarp();
          tmem_ld_32x32(t_addr + c, v);
          tmem_ld_wait_for(v);
          if (c + 64 >= cols_end) release_accumulator();
          note_nonfinite(v, min(32, args.n_total - col_base - c));
          if (row_ok)
#pragma unroll
            for (int j = 0; j < 32; j += 8)
              st_global_v8(dst + c + j, v[j], v[j + 1], v[j + 2], v[j + 3], v[j + 4], v[j + 5], v[j + 6], v[j + 7]);
        }
        continue;
      }
      {
#pragma unroll 1
        for (int c = c_first; c < cols_end; c += 64) {
          uint32_t v[32];
          __syncwarp();
          tmem_ld_32x32(t_addr + c, v);
          tmem_ld_wait_for(v);
          if (c + 64 >= cols_end) release_accumulator();
          if (lane == 0) tma_store_wait_read<0>();  // the previous store has read the buffer
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float f[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(v[8 * j + i]) * args.alpha;
            uint32_t pk[4];
            pack_half8(f, pk);
            st_shared_v4(wrow + ((uint32_t(j) ^ sw) << 4), pk[0], pk[1], pk[2], pk[3]);
          }
          store_staged(wbuf, col_base + c);
        }
        continue;
      }
      if (stamp) PLB_TRACE_STAMP(2, local_tile * 4 + 2);
      if (stamp) PLB_TRACE_STAMP(2, local_tile * 4 + 3);
    }
    // this thread's stores must have read their staging buffers before the CTA
    // gives up its shared memory (the writes themselves complete with the grid)
    if (tma_store && lane == 0) tma_store_wait_read<0>();
    if (stamp) PLB_TRACE_STAMP(2, 4016);
  }

  if (threadIdx.x == 0) PLB_TRACE_STAMP(2, 4003);
  if (args.chain == kChainFollow) pdl_wait();
  tc_fence_before_sync();
  // Every tensor copy must have landed before the CTA gives up its shared
  // memory.  In a run without errors the MMA issuer has waited for every
  // stage it consumed, i.e. for all of them; only after an aborted wait can
  // copies still be in flight, and then they are waited for here (bounded).
  // Stage s was last filled by pipeline step g = the largest g < total with
  // g mod kStages == s, in phase (g / kStages) & 1.  With a CTA pair the
  // barriers live in the MMA-issuing CTA, which waits for both CTAs' copies;
  // the other CTA cannot leave before the rendezvous below.
  __syncthreads();
  if (*abort_flag != 0 && threadIdx.x == 0 && leader) {
    int my_tiles = 0;
    long long total_steps = 0;
    for (int unit = first_unit; unit < total_units; unit += unit_stride, ++my_tiles) {
      int tile, group, split, it_begin, it_end;
      unit_coords(unit, tile, group, split, it_begin, it_end);
      total_steps += it_end - it_begin;
    }
    const long long start = clock64();
    auto drain = [&](uint32_t bar, uint32_t parity) {
      while (!mbar_try_wait(bar, parity)) {
        if (clock64() - start > kWaitCycleLimit) {
          atomicCAS(args.status, kStatusOk, kStatusDrainTimeout);
          break;
        }
      }
    };
    if (kResB && my_tiles > 0) drain(resb_bar, 0);
    for (int st = 0; st < kStages; ++st) {
      if (total_steps <= st) continue;
      const long long g = st + ((total_steps - 1 - st) / kStages) * kStages;
      drain(full_bar(st), uint32_t((g / kStages) & 1));
    }
  }
  // Neither CTA of a pair may go away while the other can still touch its
  // barriers, shared memory or tensor memory.  Arrivals that one leaves on the
  // other's barriers have been waited for above; the rendezvous of all threads of
  // the cluster (which is also this CTA's own barrier) orders the rest.
  if constexpr (k2Cta)
    cluster_sync_relaxed();
  else
    __syncthreads();
  if (threadIdx.x == 0) PLB_TRACE_STAMP(2, 4004);
  if (warp == kIgemmMmaWarp) {
    tc_fence_after_sync();
    if constexpr (k2Cta)
      tmem_dealloc_pair(tmem_base, kTmemCols);
    else
      tmem_dealloc(tmem_base, kTmemCols);
  }
#ifdef PLB_TRACE
  if (threadIdx.x == 0) {
    PLB_TRACE_STAMP(2, 4005);
    uint32_t smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    if (args.trace != nullptr && blockIdx.x == 0) args.trace[2 * 4096 + 4006] = smid;
  }
#endif
}

}  // namespace plb
