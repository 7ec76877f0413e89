// Launch of one instance of the patch kernel; the instances of each operand type are
// compiled in a file of their own (patch_*.cu).
#pragma once

#include <atomic>

#include "patch.cuh"

namespace plb {

template <int kType, bool kBMn, int MT, int NT>
int launchPatchInstance(plb_context *ctx, const PatchVariant &v, const PatchArgs &g) {
  static std::atomic<bool> configured[64] = {};  // (contexts may live on several threads)
  auto kernel = patchKernel<kType, kBMn, MT, NT>;
  std::atomic<bool> &done = configured[ctx->device & 63];
  if (!done) {
    PLB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024));
    done = true;
  }
  return launchPdl(ctx, kernel, dim3(v.grid), dim3(kPatchThreads), v.smem, g);
}

template <int kType, bool kBMn>
int launchPatchShape(plb_context *ctx, const PatchVariant &v, const PatchArgs &g) {
  // (floats, two pieces of each operand in registers, keep to 32 pixels an item)
  if constexpr (kType != PLB_FLOAT)
    switch (v.mt * 8 + v.nt) {
      case 4 * 8 + 1: return launchPatchInstance<kType, kBMn, 4, 1>(ctx, v, g);
      case 4 * 8 + 2: return launchPatchInstance<kType, kBMn, 4, 2>(ctx, v, g);
      case 4 * 8 + 3: return launchPatchInstance<kType, kBMn, 4, 3>(ctx, v, g);
      case 4 * 8 + 4: return launchPatchInstance<kType, kBMn, 4, 4>(ctx, v, g);
      default: break;
    }
  switch (v.mt * 8 + v.nt) {
    case 2 * 8 + 1: return launchPatchInstance<kType, kBMn, 2, 1>(ctx, v, g);
    case 2 * 8 + 2: return launchPatchInstance<kType, kBMn, 2, 2>(ctx, v, g);
    case 2 * 8 + 3: return launchPatchInstance<kType, kBMn, 2, 3>(ctx, v, g);
    case 2 * 8 + 4: return launchPatchInstance<kType, kBMn, 2, 4>(ctx, v, g);
    default: return fail(PLB_ERR_UNSUPPORTED, "no instance of the patch kernel of this shape");
  }
}

template <int kType>
int launchPatchType(plb_context *ctx, const PatchVariant &v, const PatchArgs &g) {
  return v.b_mn ? launchPatchShape<kType, true>(ctx, v, g) : launchPatchShape<kType, false>(ctx, v, g);
}

}  // namespace plb
