// Batch normalisation after a convolution: the entry points behind poplin's Norms
// API (include/poplin/Norms.hpp:33-334, lib/poplin/Norms.cpp), on device-layout
// activations [pixels][chans] (NHWC: the channels of a pixel are contiguous),
// statistics per channel over all pixels.  The kernels are the per-channel sums
// and maps of channel_ops.cuh: memory bound, the order of additions fixed (the
// reference's reductions are deterministic too), one rounding, in the output type.
#include <cuda_fp16.h>

#include <algorithm>
#include <string>

#include "channel_ops.cuh"

namespace plb {
namespace {

// iStdDev from mean and power: the reference's InverseStdDeviation vertex
// (lib/poplin/codelets/InverseStdDeviation.cpp:33-55), in fp32.
template <typename T>
__global__ void normInvStdDevKernel(const T *__restrict__ mean, const float *__restrict__ power,
                                    int chans, float eps, float scale_var, int stable,
                                    T *__restrict__ inv_std) {
  pdl_launch_dependents();
  pdl_wait();  // inputs may come from the previous kernel in the stream
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= chans) return;
  float var;
  if (stable) {
    var = (power[c] + eps) * scale_var;
  } else {
    const float m = toFloat(mean[c]);
    var = power[c] - m * m;
    if (var < 0.f) var = 0.f;   // rounding can make the estimate negative
    var = (var + eps) * scale_var;
  }
  inv_std[c] = fromFloat<T>(1.0f / sqrtf(var));
}

int checkNorm(int32_t dtype, uint64_t pixels, uint32_t chans) {
  if (dtype != PLB_HALF && dtype != PLB_FLOAT)
    return fail(PLB_ERR_UNSUPPORTED, "normalisation is implemented for half and float activations");
  if (chans == 0 || chans > (1u << 30) || pixels > (uint64_t(1) << 40))
    return fail(PLB_ERR_INVALID_PARAMS, "normalisation: channel or pixel count out of range");
  return PLB_OK;
}

template <int kMode>
int sums(plb_context *ctx, int32_t dtype, const void *x, const void *y, const void *centre, uint64_t pixels,
         uint32_t chans, ChanFinish fin) {
  fin.a_half = fin.b_half = dtype == PLB_HALF;
  if (dtype == PLB_HALF)
    return chanSums<__half, kMode>(ctx, static_cast<const __half *>(x), static_cast<const __half *>(y),
                                   static_cast<const __half *>(centre), pixels, chans, fin);
  return chanSums<float, kMode>(ctx, static_cast<const float *>(x), static_cast<const float *>(y),
                                static_cast<const float *>(centre), pixels, chans, fin);
}

struct MapOperands {
  const void *x = nullptr, *y = nullptr, *p = nullptr, *q = nullptr, *r = nullptr, *s = nullptr;
  const float *pf = nullptr, *qf = nullptr;
  void *out = nullptr, *out2 = nullptr;
};

template <int kMode, typename T>
int mapTyped(plb_context *ctx, const MapOperands &m, uint64_t pixels, uint32_t chans) {
  ChanMapArgs<T> g;
  g.x = static_cast<const T *>(m.x);
  g.y = static_cast<const T *>(m.y);
  g.p = static_cast<const T *>(m.p);
  g.q = static_cast<const T *>(m.q);
  g.r = static_cast<const T *>(m.r);
  g.s = static_cast<const T *>(m.s);
  g.pf = m.pf;
  g.qf = m.qf;
  g.out = static_cast<T *>(m.out);
  g.out2 = static_cast<T *>(m.out2);
  return chanMap<T, kMode>(ctx, g, pixels, chans);
}

template <int kMode>
int map(plb_context *ctx, int32_t dtype, const MapOperands &m, uint64_t pixels, uint32_t chans) {
  return dtype == PLB_HALF ? mapTyped<kMode, __half>(ctx, m, pixels, chans)
                           : mapTyped<kMode, float>(ctx, m, pixels, chans);
}

}  // namespace
}  // namespace plb

using namespace plb;

extern "C" {

int plb_norm_moments(plb_context *ctx, int32_t dtype, const void *d_acts, uint64_t pixels,
                     uint32_t chans, float scale, const void *d_centre, void *d_mean,
                     float *d_power) {
  TraceRange trace_range("plb_norm_moments");
  if (int rc = activate(ctx)) return rc;
  if (int rc = checkNorm(dtype, pixels, chans)) return rc;
  if (!d_acts && pixels) return fail(PLB_ERR_INVALID_PARAMS, "null activations");
  ChanFinish fin{};
  fin.scale = scale;
  fin.b_f32 = d_power;
  // mean of squared deviations from a given centre (the "stable" estimator)
  if (d_centre) return sums<kSumCentredXX>(ctx, dtype, d_acts, nullptr, d_centre, pixels, chans, fin);
  fin.a = d_mean;
  return sums<kSumXAndXX>(ctx, dtype, d_acts, nullptr, nullptr, pixels, chans, fin);
}

int plb_norm_statistics(plb_context *ctx, int32_t dtype, const void *d_acts, uint64_t pixels,
                        uint32_t chans, float eps, float scale_var, void *d_mean, void *d_inv_std,
                        float *d_power) {
  TraceRange trace_range("plb_norm_statistics");
  if (int rc = activate(ctx)) return rc;
  if (int rc = checkNorm(dtype, pixels, chans)) return rc;
  if ((!d_acts && pixels) || !d_mean || !d_inv_std)
    return fail(PLB_ERR_INVALID_PARAMS, "normalisation: null pointer");
  ChanFinish fin{};
  fin.scale = pixels > 0 ? 1.0f / float(pixels) : 1.0f;
  fin.a = d_mean;
  fin.b_f32 = d_power;
  fin.inv_std = d_inv_std;
  fin.eps = eps;
  fin.scale_var = scale_var;
  return sums<kSumXAndXX>(ctx, dtype, d_acts, nullptr, nullptr, pixels, chans, fin);
}

int plb_norm_normalise(plb_context *ctx, int32_t dtype, const void *d_acts, const void *d_mean,
                       const void *d_inv_std, const void *d_gamma, const void *d_beta, uint64_t pixels,
                       uint32_t chans, void *d_whitened, void *d_out) {
  TraceRange trace_range("plb_norm_normalise");
  if (int rc = activate(ctx)) return rc;
  if (int rc = checkNorm(dtype, pixels, chans)) return rc;
  if (!d_mean || !d_inv_std || !d_gamma || !d_beta || ((!d_acts || !d_out) && pixels))
    return fail(PLB_ERR_INVALID_PARAMS, "normalisation: null pointer");
  MapOperands m;
  m.x = d_acts;
  m.p = d_mean;
  m.q = d_inv_std;
  m.r = d_gamma;
  m.s = d_beta;
  m.out = d_out;
  m.out2 = d_whitened;
  return map<kNormalise>(ctx, dtype, m, pixels, chans);
}

int plb_norm_inv_std_dev(plb_context *ctx, int32_t dtype, const void *d_mean, const float *d_power,
                         uint32_t chans, float eps, float scale_var, int stable, void *d_inv_std) {
  if (int rc = activate(ctx)) return rc;
  if (int rc = checkNorm(dtype, 0, chans)) return rc;
  if (!d_power || !d_inv_std || (!stable && !d_mean))
    return fail(PLB_ERR_INVALID_PARAMS, "normalisation: null statistics pointer");
  const dim3 grid(unsigned((chans + 127) / 128));
  if (dtype == PLB_HALF)
    return launchPdl(ctx, normInvStdDevKernel<__half>, grid, dim3(128), 0, static_cast<const __half *>(d_mean),
                     d_power, int(chans), eps, scale_var, stable, static_cast<__half *>(d_inv_std));
  return launchPdl(ctx, normInvStdDevKernel<float>, grid, dim3(128), 0, static_cast<const float *>(d_mean),
                   d_power, int(chans), eps, scale_var, stable, static_cast<float *>(d_inv_std));
}

int plb_norm_whiten(plb_context *ctx, int32_t dtype, const void *d_acts, const void *d_mean,
                    const void *d_inv_std, uint64_t pixels, uint32_t chans, void *d_out) {
  TraceRange trace_range("plb_norm_whiten");
  if (int rc = activate(ctx)) return rc;
  if (int rc = checkNorm(dtype, pixels, chans)) return rc;
  MapOperands m;
  m.x = d_acts;
  m.p = d_mean;
  m.q = d_inv_std;
  m.out = d_out;
  return map<kWhiten>(ctx, dtype, m, pixels, chans);
}

int plb_norm_scale_shift(plb_context *ctx, int32_t dtype, const void *d_acts, const void *d_scale,
                         const void *d_shift, uint64_t pixels, uint32_t chans, void *d_out) {
  TraceRange trace_range("plb_norm_scale_shift");
  if (int rc = activate(ctx)) return rc;
  if (int rc = checkNorm(dtype, pixels, chans)) return rc;
  MapOperands m;
  m.x = d_acts;
  m.p = d_scale;
  m.q = d_shift;
  m.out = d_out;
  return d_shift ? map<kScaleShift>(ctx, dtype, m, pixels, chans) : map<kScale>(ctx, dtype, m, pixels, chans);
}

int plb_norm_param_gradients(plb_context *ctx, int32_t dtype, const void *d_whitened,
                             const void *d_grads, uint64_t pixels, uint32_t chans, float scale,
                             void *d_gamma_delta, void *d_beta_delta, float *d_gamma_delta_f32,
                             float *d_beta_delta_f32) {
  TraceRange trace_range("plb_norm_param_gradients");
  if (int rc = activate(ctx)) return rc;
  if (int rc = checkNorm(dtype, pixels, chans)) return rc;
  if (!d_gamma_delta && !d_beta_delta && !d_gamma_delta_f32 && !d_beta_delta_f32) return PLB_OK;
  ChanFinish fin{};
  fin.scale = scale;
  fin.a = d_gamma_delta;
  fin.b = d_beta_delta;
  fin.a_f32 = d_gamma_delta_f32;
  fin.b_f32 = d_beta_delta_f32;
  return sums<kSumXYAndY>(ctx, dtype, d_whitened, d_grads, nullptr, pixels, chans, fin);
}

int plb_norm_statistics_gradients(plb_context *ctx, int32_t dtype, const void *d_whitened,
                                  const void *d_grads, const void *d_inv_std, const void *d_var_delta,
                                  const void *d_mean_delta, uint64_t pixels, uint32_t chans,
                                  void *d_out) {
  TraceRange trace_range("plb_norm_statistics_gradients");
  if (int rc = activate(ctx)) return rc;
  if (int rc = checkNorm(dtype, pixels, chans)) return rc;
  if (pixels == 0) return PLB_OK;
  if ((d_var_delta == nullptr) != (d_mean_delta == nullptr))
    return fail(PLB_ERR_INVALID_PARAMS, "give both per-channel deltas or neither");
  MapOperands m;
  m.x = d_whitened;
  m.y = d_grads;
  m.r = d_inv_std;
  m.out = d_out;
  if (d_var_delta) {
    // the two per-channel means come from the caller (already reduced over replicas)
    m.p = d_var_delta;
    m.q = d_mean_delta;
    return map<kStatsGrad>(ctx, dtype, m, pixels, chans);
  }
  // -mean(whitened * grads) and -mean(grads) per channel, kept in fp32, then
  // out = (grads + whitened * varDelta + meanDelta) * invStdDev
  // (lib/poplin/Norms.cpp:447-512, without its split of the scale in two
  // factors, which only serves half-precision intermediates)
  void *ws = nullptr;
  if (int rc = scratch(ctx, kSlotUsedTaps, size_t(2) * chans * sizeof(float) + 256, &ws)) return rc;
  float *var_delta = static_cast<float *>(ws), *mean_delta = var_delta + chans;
  if (int rc = plb_norm_param_gradients(ctx, dtype, d_whitened, d_grads, pixels, chans,
                                        -1.0f / float(pixels), nullptr, nullptr, var_delta, mean_delta))
    return rc;
  m.pf = var_delta;
  m.qf = mean_delta;
  return map<kStatsGrad>(ctx, dtype, m, pixels, chans);
}

// ---- biases of a convolution -----------------------------------------------------

int plb_add_bias(plb_context *ctx, int32_t dtype, void *d_acts, const void *d_biases,
                 uint64_t pixels, uint32_t chans) {
  if (int rc = activate(ctx)) return rc;
  if (dtype != PLB_HALF && dtype != PLB_FLOAT) {
    if (pixels == 0 || chans == 0) return PLB_OK;
    return fail(PLB_ERR_INVALID_PARAMS, "bias add needs half or float activations");
  }
  MapOperands m;
  m.x = m.out = d_acts;
  m.p = d_biases;
  return map<kAddChan>(ctx, dtype, m, pixels, chans);
}

int plb_conv_bias_update(plb_context *ctx, int32_t acts_dtype, const void *d_out_grads,
                         uint64_t pixels, uint32_t chans, int32_t bias_dtype, void *d_biases,
                         float scale) {
  if (int rc = activate(ctx)) return rc;
  if ((acts_dtype != PLB_HALF && acts_dtype != PLB_FLOAT) ||
      (bias_dtype != PLB_HALF && bias_dtype != PLB_FLOAT))
    return fail(PLB_ERR_INVALID_PARAMS, "bias update needs half or float gradients and biases");
  if (chans == 0) return PLB_OK;
  ChanFinish fin{};
  fin.scale = scale;
  fin.bias = d_biases;
  fin.bias_half = bias_dtype == PLB_HALF;
  return sums<kSumX>(ctx, acts_dtype, d_out_grads, nullptr, nullptr, pixels, chans, fin);
}

}  // extern "C"
