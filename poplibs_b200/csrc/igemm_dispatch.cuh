// Launch of one instance of the implicit-GEMM kernel.  The instances of each
// column-tile width are compiled in a file of their own (igemm_bn*.cu).
#pragma once

#include <atomic>

#include "igemm_sm100.cuh"
#include "launch_shape.h"
#include "runtime.h"

namespace plb {

// Which instance, and how it is launched.
struct IgemmVariant {
  bool fp8, a_mn, b_mn, resident, halo, pair, groups;
  int grid, grid_multiple, resident_bytes;  // grid_multiple: of the CTAs (pairs of them)
  bool pdl;
};

int launchIgemm64(plb_context *ctx, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &tout,
                  const IgemmArgs &args, const IgemmVariant &v);
int launchIgemm128(plb_context *ctx, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &tout,
                   const IgemmArgs &args, const IgemmVariant &v);
int launchIgemm256(plb_context *ctx, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &tout,
                   const IgemmArgs &args, const IgemmVariant &v);

template <int BN, bool kFp8, bool kAMn, bool kBMn, bool kResB, bool kHalo, bool k2Cta, bool kGroups>
int launchInstance(plb_context *ctx, const CUtensorMap &ta, const CUtensorMap &tb,
                   const CUtensorMap &tout, const IgemmArgs &args, const IgemmVariant &v) {
  if constexpr (k2Cta && kBMn && BN < 128) {
    return fail(PLB_ERR_INVALID_OPTION, "a CTA pair needs tile_n >= 128 for a row-major B");
  } else {
    using S = IgemmSmem<BN, kResB, k2Cta>;
    // (contexts may live on several threads; each would store the same values)
    static std::atomic<bool> configured[64] = {};
    static std::atomic<int> max_clusters[64] = {};
    auto kernel = igemm_kernel<BN, kFp8, kAMn, kBMn, kResB, kHalo, k2Cta, kGroups>;
    const int dev = ctx->device & 63;
    if (!configured[dev]) {
      PLB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kIgemmSmemLimit));
      configured[dev] = true;
    }
    const int smem =
        S::totalBytes(args.a_stage_bytes, args.b_tiles_per_stage, args.num_stages, v.resident_bytes);
    // Launch attributes: programmatic stream serialization (the kernel's set-up
    // may overlap the previous kernel's tail; it waits before touching global
    // memory) and, for CTA pairs, clusters of two.
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(kIgemmThreads);
    cfg.dynamicSmemBytes = size_t(smem);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    unsigned n_attr = 0;
    if (v.pdl) {
      attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
      ++n_attr;
    }
    if constexpr (!k2Cta) {
      cfg.gridDim = dim3(unsigned(v.grid));
    } else {
      // a persistent grid of as many clusters as can be resident at once
      // (pairs of SMs in one GPC), each walking tile pairs
      attr[n_attr].id = cudaLaunchAttributeClusterDimension;
      attr[n_attr].val.clusterDim.x = 2;
      attr[n_attr].val.clusterDim.y = 1;
      attr[n_attr].val.clusterDim.z = 1;
      ++n_attr;
      if (max_clusters[dev] == 0) {
        // queried with the largest shared-memory size, a lower bound for smaller ones
        cudaLaunchConfig_t q = cfg;
        q.gridDim = dim3(unsigned(2 * ctx->sm_count));
        q.dynamicSmemBytes = size_t(kIgemmSmemLimit);
        q.attrs = &attr[n_attr - 1];
        q.numAttrs = 1;
        int n = 0;
        PLB_CUDA(cudaOccupancyMaxActiveClusters(&n, kernel, &q));
        if (n <= 0) return fail(PLB_ERR_CUDA, "no cluster of two CTAs can be resident on this device");
        max_clusters[dev] = n;
      }
      cfg.gridDim = dim3(unsigned(2 * clusterCount(v.grid / 2, max_clusters[dev], v.grid_multiple)));
    }
    cfg.attrs = attr;
    cfg.numAttrs = n_attr;
    PLB_CUDA(cudaLaunchKernelEx(&cfg, kernel, ta, tb, tout, args));
    PLB_CUDA(cudaGetLastError());
    ctx->launches++;
    return PLB_OK;
  }
}

template <int BN>
int launchForTile(plb_context *ctx, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &tout,
                  const IgemmArgs &args, const IgemmVariant &v) {
#define PLB_LAUNCH(FP8, AMN, BMN, RES, HALO, GROUPS)                                                          \
  return v.pair ? launchInstance<BN, FP8, AMN, BMN, RES, HALO, true, GROUPS>(ctx, ta, tb, tout, args, v)      \
                : launchInstance<BN, FP8, AMN, BMN, RES, HALO, false, GROUPS>(ctx, ta, tb, tout, args, v)
#define PLB_LAUNCH_OPERANDS(RES, HALO, GROUPS)                       \
  if (v.fp8) PLB_LAUNCH(true, false, false, RES, HALO, GROUPS);      \
  if (v.b_mn) PLB_LAUNCH(false, false, true, RES, HALO, GROUPS);     \
  PLB_LAUNCH(false, false, false, RES, HALO, GROUPS)
  if (v.a_mn && v.groups) {
    if (v.b_mn) PLB_LAUNCH(false, true, true, false, false, true);
    PLB_LAUNCH(false, true, false, false, false, true);
  }
  if (v.a_mn) {
    if (v.b_mn) PLB_LAUNCH(false, true, true, false, false, false);
    PLB_LAUNCH(false, true, false, false, false, false);
  }
  if (v.groups && v.halo && v.resident) {
    PLB_LAUNCH_OPERANDS(true, true, true);
  }
  if (v.groups && v.resident) {
    PLB_LAUNCH_OPERANDS(true, false, true);
  }
  if (v.groups && v.halo) {
    PLB_LAUNCH_OPERANDS(false, true, true);
  }
  if (v.groups) {
    PLB_LAUNCH_OPERANDS(false, false, true);
  }
  if (v.halo && v.resident) {
    PLB_LAUNCH_OPERANDS(true, true, false);
  }
  if (v.halo) {
    PLB_LAUNCH_OPERANDS(false, true, false);
  }
  if (v.resident) {
    PLB_LAUNCH_OPERANDS(true, false, false);
  }
  PLB_LAUNCH_OPERANDS(false, false, false);
#undef PLB_LAUNCH_OPERANDS
#undef PLB_LAUNCH
}

}  // namespace plb
