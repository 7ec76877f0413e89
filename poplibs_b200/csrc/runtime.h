// Internal host-side runtime shared by the C ABI entry points: the context
// (device, stream, kernel status word, scratch memory), error reporting and
// TMA tensor-map construction.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "poplibs_b200.h"

// Grow-only scratch buffers of a context, by use.  Entry points call one
// another (3-D -> 2-D -> flipped -> dilated -> padded channels ...), so every
// pre-pass has a slot of its own.
enum plb_scratch_slot {
  kSlotOperands = 0,    // rearranged operands (transposed, space-to-depth)
  kSlotWuPartials,      // fp32 partial sums of a weight update
  kSlotHostIn,          // staging of the host-buffer entry points
  kSlotHostWeights,
  kSlotHostOut,
  kSlotHostBias,
  kSlotChannelSums,     // partial per-channel sums (normalisation, bias update)
  kSlotBlockDiagonal,   // block-diagonal weights of channel groups contracted together
  kSlotUsedTaps,        // gradient of a truncated / flipped kernel's taps
  kSlotRepacked,        // operands with rows rounded up to 16 bytes / split into bfloat16 pieces
  kSlotFlipped,         // reversed input (input flip)
  kSlotDepthFold,       // depth taps of a 3-D field gathered into the channels
  kSlotFoldedWeights,
  kSlotFoldedGrads,
  kSlotDilated,         // zero-stuffed input (input dilation)
  kSlotSplitK,          // fp32 partial sums of a split-K forward / backward / matrix product
  kSlotCount
};

struct plb_context {
  int device = 0;
  int sm_count = 0;
  cudaStream_t stream = nullptr;
  bool owns_stream = false;
  // Kernel status word (0 = OK): page-locked host memory mapped into the device,
  // written by kernels only when a bounded wait runs out, read by the host
  // without a copy (a copy would queue behind other streams' transfers).
  int *d_status = nullptr;        // device address
  volatile int *h_status = nullptr;  // host address of the same word
  // Arrival counter of kernels whose last block finishes the work of all; zero
  // between launches (the last block clears it).
  unsigned *d_ticket = nullptr;
  uint64_t launches = 0;          // kernels launched through this context
  int plan_flags = 0;             // PLB_PLAN_* bits added to every plan made through this context
  long long *trace = nullptr;     // device timeline buffer for builds with -DPLB_TRACE
  cudaEvent_t timer_start = nullptr, timer_stop = nullptr;
  // grow-only scratch buffers, one per use (plb_scratch_slot)
  static constexpr int kScratchSlots = kSlotCount;
  void *scratch[kScratchSlots] = {};
  size_t scratch_bytes[kScratchSlots] = {};
  bool scratch_refused = false;   // a buffer could not grow, as the stream is being captured
};

#include <nvtx3/nvToolsExt.h>

namespace plb {

// A named range around a public entry point, visible to profilers that hook
// NVTX (the role of POPLIN_TRACEPOINT at the reference's entry points,
// include/poplibs_support/Tracepoint.hpp:69-78).  Header-only: without a
// profiler attached the calls are a null-pointer test each.
struct TraceRange {
  explicit TraceRange(const char *name) { nvtxRangePushA(name); }
  ~TraceRange() { nvtxRangePop(); }
  TraceRange(const TraceRange &) = delete;
  TraceRange &operator=(const TraceRange &) = delete;
};

// Records the message for plb_last_error() and returns `code`.
int fail(int code, const std::string &message);
int cudaFail(cudaError_t err, const char *what);

#define PLB_CUDA(expr)                                         \
  do {                                                         \
    cudaError_t plb_err__ = (expr);                            \
    if (plb_err__ != cudaSuccess) return ::plb::cudaFail(plb_err__, #expr); \
  } while (0)

// Makes the context's device current.
int activate(plb_context *ctx);
// Returns a scratch buffer of at least `bytes` (grows, synchronising first, if needed; not while
// the stream is being captured, which is an error that leaves the capture as it is).
int scratch(plb_context *ctx, int slot, size_t bytes, void **ptr);

// cuTensorMapEncodeTiled with 128-byte swizzle and zero fill outside the
// tensor.  dims[0] is the contiguous dimension; strides_bytes[i] is the byte
// stride of dims[i + 1].
int encodeTensorMap(CUtensorMap *tm, CUtensorMapDataType type, int rank, const void *base,
                    const uint64_t *dims, const uint64_t *strides_bytes, const uint32_t *box,
                    const uint32_t *elem_strides, int swizzle_bytes = 128);

// Launch with programmatic stream serialization: the kernel may become resident
// while its predecessor in the stream drains.  It must execute
// griddepcontrol.wait (in every block that touches global memory, and in at
// least one block whatever its arguments) before it reads or writes.
template <typename... KArgs, typename... Args>
int launchPdl(plb_context *ctx, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, Args... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cfg.attrs = attr;
  cfg.numAttrs = (ctx->plan_flags & PLB_PLAN_NO_PDL) ? 0 : 1;
  PLB_CUDA(cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...));
  PLB_CUDA(cudaGetLastError());
  ctx->launches++;
  return PLB_OK;
}

inline size_t dtypeBytes(int dtype) {
  return dtype == PLB_FLOAT ? 4 : (dtype == PLB_HALF || dtype == PLB_BFLOAT16) ? 2 : 1;
}
// 16-bit floating-point operands (the kind::f16 instruction takes either)
inline bool is16BitFloat(int dtype) { return dtype == PLB_HALF || dtype == PLB_BFLOAT16; }

// ---- operands brought into a form TMA can address (repack.cu) -------------------
enum RepackMode : int {
  kRepackCopy = 0,        // row -> row, zero-filled up to dst_pitch
  kRepackSplitCols = 1,   // float row of c -> one row of 3c bfloat16 (the pieces side by side), zero-filled
  kRepackSplitPlanes = 2, // float [outer][mid] rows -> [outer][3][mid] rows of bfloat16, each zero-filled
};
struct Repack {
  const void *src;
  void *dst;              // 16-byte aligned
  uint64_t rows;
  uint32_t cols;          // elements of a source row
  uint64_t src_pitch;     // elements
  uint32_t dst_pitch;     // elements, a multiple of 16 bytes
  uint32_t elem_bytes;    // of the source
  int mode;
  bool weights;           // pieces (hi, hi, lo), else (hi, lo, hi)
  uint64_t mid;           // kRepackSplitPlanes: rows per plane (0 = all)
  // Rows taken from every step_h'th / step_w'th pixel of [image][full_h][full_w][parts]
  // (`rows` counts the taken ones, [image][sub_h][sub_w][parts]; sub_w 0: all rows).
  struct Lattice {
    uint32_t parts, sub_w, sub_h, full_w, full_h, step_w, step_h;
  } lattice;
};
// Bytes of the destination.
size_t repackBytes(const Repack &r);
// One launch for up to two operands.
int repack(plb_context *ctx, const Repack *jobs, int n);
// Rows of `elems` elements rounded up to whole 16-byte vectors.
inline uint32_t roundToVec(uint64_t elems, size_t elem_bytes) {
  const uint64_t q = 16 / elem_bytes;
  return uint32_t((elems + q - 1) / q * q);
}
// The row pitch of a copied operand: whole 16, 32 or 64 bytes up to there, else whole
// 128-byte lines.  A tensor copy fetches 128-byte pieces of rows; pieces that lie
// across lines, or end beyond the tensor's innermost extent and are filled up with
// zeros, take it up to twice as long as whole lines (3x3 layer of 46 images of
// 35x35, 64 output channels: 17.2 us with 88 input channels, 12.5 with 128).
inline uint32_t roundToRow(uint64_t elems, size_t elem_bytes) {
  const uint64_t bytes = elems * elem_bytes;
  const uint64_t q = bytes <= 16 ? 16 : bytes <= 32 ? 32 : bytes <= 64 ? 64 : 128;
  return uint32_t((bytes + q - 1) / q * q / elem_bytes);
}

// Input flip of the reference's input transform: the convolution of a flipped
// input equals the convolution of the reversed tensor with the input padding and
// truncation of the flipped dimensions swapped.  Returns true and fills `q` if
// `p` flips its input in some dimension.
bool unflippedInputParams(const plb_conv_params &p, plb_conv_params *q);
// Spatial flip of an [n][H][W][pixel] tensor (runtime.cu).
int flipField(plb_context *ctx, const void *src, void *dst, size_t n_images, uint32_t H, uint32_t W,
              size_t pixel_bytes, bool flip_h, bool flip_w);

// First check of every convolution entry point, before any pre-pass is
// launched: the reference's parameter validation, the element types this path
// implements (wu: the weight update takes half only) and that no tensor with
// elements is passed as a null pointer.  `in` / `weights` / `out` follow the
// forward naming; pass the tensors of the pass in that order
// (backward: out grads, weights, in grads; weight update: acts, out grads, any
// of the two gradient outputs).
int checkConvRequest(const plb_conv_params &p, bool wu, const void *in_like, size_t in_elems,
                     const void *second, size_t second_elems, const void *result,
                     size_t result_elems);
// Element counts of the activations, weights and output of `p` (any rank).
void convElementCounts(const plb_conv_params &p, size_t *in, size_t *weights, size_t *out);

// Input dilation of the reference's input transform, as data: the convolution of
// a dilated input equals the ordinary convolution of the zero-stuffed tensor
// dilate(truncate(x)).  A fallback (the inserted zeros are multiplied); the
// backward pass of a strided layer does not come this way (plb_conv_bwd takes
// it in forward terms).  [n][H][W] field (H = 1 for 1-D), tH/tW lower truncation,
// TH/TW kept extent, dH/dW dilation, Hd/Wd dilated extent.
struct DilatedField {
  uint32_t H, W, tH, tW, TH, TW, dH, dW, Hd, Wd;
};
// Returns true and fills `q` (field = dilated extent, no truncation, dilation 1)
// and `f` if `p` (1-D or 2-D) dilates its input.
bool undilatedInputParams(const plb_conv_params &p, plb_conv_params *q, DilatedField *f);
// dst = dilate(truncate(src)) ([n][Hd][Wd]); adjoint: dst ([n][H][W]) = the
// elements of src ([n][Hd][Wd]) on the lattice, zero in the truncated margins.
int dilateField(plb_context *ctx, const void *src, void *dst, size_t n_images, const DilatedField &f,
                size_t pixel_bytes, bool adjoint);

// ---- 3-D fields (conv3d.cu): depth folded into the channels of a 2-D problem ----
int conv3dFwd(plb_context *ctx, const plb_conv_params &p, const plb_conv_options *opt,
              const void *d_in, const void *d_weights, const float *d_bias, void *d_out,
              int transpose_and_flip_weights);
int conv3dBwd(plb_context *ctx, const plb_conv_params &p, const plb_conv_options *opt,
              const void *d_out_grads, const void *d_weights, void *d_in_grads);
int conv3dWu(plb_context *ctx, const plb_conv_params &p, const plb_conv_options *opt,
             const void *d_acts, const void *d_out_grads, void *d_weight_grads,
             float *d_weight_grads_f32);
int conv3dPlan(const plb_conv_params &p, const plb_conv_options *opt, int32_t pass, plb_plan *plan);

// ---- contraction launch (igemm_launch.cu) -----------------------------------

// A fully resolved implicit-GEMM problem: one launch of the igemm kernel.
struct IgemmProblem {
  bool fp8 = false;      // 8-bit operands (else 16-bit)
  bool bf16 = false;     // 16-bit operands are bfloat16 (else half)
  int fmt_a = 0, fmt_b = 0;  // plb_quarter_format of the activations / weights when fp8
  bool b_mn = false;     // right operand stored [tap][K][N], N contiguous
  bool a_mn = false;     // matrix product whose left operand is stored [K][M] (act_dims = (K, M), stride of a K row)
  // Groups: independent contractions of one shape.  The weights of group g are
  // the tiles [g * taps_stored, (g + 1) * taps_stored) of wgt_dims[2].
  int groups = 1;
  uint64_t act_group_stride = 0;                               // bytes
  long long out_group_stride = 0, addend_group_stride = 0;     // elements
  // activations: 4-D tensor (C, W, H, N) with byte strides of W, H, N
  const void *act = nullptr;
  uint64_t act_dims[4] = {1, 1, 1, 1};
  uint64_t act_strides[3] = {16, 16, 16};
  uint32_t act_elem_strides[4] = {1, 1, 1, 1};  // traversal strides (conv stride on W, H)
  // weights: (K, N, taps) K-major or (N, K, taps) MN-major, byte strides of dims 1, 2
  const void *wgt = nullptr;
  uint64_t wgt_dims[3] = {1, 1, 1};
  uint64_t wgt_strides[2] = {16, 16};
  // output
  int out_w = 1, out_h = 1, out_n = 1;  // pixels
  int n_total = 0;                      // output channels
  int k_per_tap = 0;                    // reduction length per tap (elements)
  int taps_h = 1, taps_w = 1, pad_h = 0, pad_w = 0, dil_h = 1, dil_w = 1;
  int flip_h = 0, flip_w = 0;
  // Sub-lattice of a stored filter (0 = dense): tap (r, s) after the flip is tile
  // (tap_first_h + r * tap_step_h) * tap_pitch_h + tap_first_w + s * tap_step_w.
  int tap_first_h = 0, tap_step_h = 1, tap_pitch_h = 0, tap_first_w = 0, tap_step_w = 1, taps_stored = 0;
  int stride_h = 1, stride_w = 1;
  void *out = nullptr;
  long long ldc = 0;  // elements between output pixels along w
  // elements between output rows / images; 0 = dense (out_w * ldc, out_h * out_w * ldc)
  long long out_stride_h = 0, out_stride_n = 0;
  const void *addend = nullptr;
  long long ld_addend = 0;
  const float *bias = nullptr;
  float alpha = 1.f, beta = 0.f;
  int chain = 0;         // IgemmChain (igemm_sm100.cuh); none for a split-K product
  int *nonfinite = nullptr;  // device word set to 1 if a sum is not finite
  bool out_f32 = false;
  int force_tile_n = 0;  // 0 = planner's choice
  int force_split_k = 0; // 0 = planner's choice; n = n CTAs per output tile (clamped to the K steps)
  int plan_flags = 0;    // PLB_PLAN_* bits
};

// Fills the tiling part of `plan` for a problem; returns non-zero if the
// problem cannot be run by the igemm kernel (message recorded).
int planIgemm(const IgemmProblem &p, int sm_count, plb_plan *plan);

// Matrices [batch][rows][cols] -> [batch][cols][dst_pitch].
int transposeBatch(plb_context *ctx, uint32_t elem_bytes, uint64_t batch, uint64_t rows, uint64_t cols, const void *src,
                   void *dst, uint64_t dst_pitch);
// weights_transpose_chans_flip_xy with a row pitch (elements) of the result.
int transposeFlipWeights(plb_context *ctx, uint32_t elem_bytes, uint32_t groups, uint32_t out_chans,
                         uint32_t in_chans, uint64_t kernel_elems, uint32_t dst_pitch, const void *src, void *dst);

int launchIgemm(plb_context *ctx, const IgemmProblem &p, const plb_plan &plan);

}  // namespace plb
