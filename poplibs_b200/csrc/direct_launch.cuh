// Launch of one instance of the direct kernel; the instances of each operand type are
// compiled in a file of their own (direct_*.cu).
#pragma once

#include <atomic>

#include "direct.cuh"

namespace plb {

template <int kType, class S, bool kAMn, bool kBMn, bool kVec>
int launchDirectInstance(plb_context *ctx, const DirectVariant &v, const DirectArgs &g) {
  constexpr int kTeamBytes = S::template kSmem<kType, kVec>;
  static std::atomic<bool> configured[64] = {};  // (contexts may live on several threads)
  auto kernel = directKernel<kType, S, kAMn, kBMn, kVec>;
  std::atomic<bool> &done = configured[ctx->device & 63];
  if (!done) {
    PLB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDirectTeams * kTeamBytes));
    done = true;
  }
  return launchPdl(ctx, kernel, dim3(v.blocks), dim3(v.teams * kDirectTeam), size_t(v.teams) * kTeamBytes, g);
}

template <int kType, DirectKind kKind, class S>
int launchDirectShape(plb_context *ctx, const DirectVariant &v, const DirectArgs &g) {
  if (!directHas(kKind, kType, v.vec)) return fail(PLB_ERR_UNSUPPORTED, "no instance of the direct kernel of this shape");
#define PLB_DIRECT(A, B)                                                      \
  return v.vec ? launchDirectInstance<kType, S, A, B, true>(ctx, v, g)        \
               : launchDirectInstance<kType, S, A, B, !directHas(kKind, kType, false)>(ctx, v, g)
  if (v.a_mn) {
    if (v.b_mn) PLB_DIRECT(true, true);
    PLB_DIRECT(true, false);
  }
  if (v.b_mn) PLB_DIRECT(false, true);
  PLB_DIRECT(false, false);
#undef PLB_DIRECT
}

template <int kType>
int launchDirectType(plb_context *ctx, const DirectVariant &v, const DirectArgs &g) {
  switch (v.kind) {
    case kDirectFew: return launchDirectShape<kType, kDirectFew, DirectFew>(ctx, v, g);
    case kDirectSmall: return launchDirectShape<kType, kDirectSmall, DirectSmall>(ctx, v, g);
    case kDirectMid: return launchDirectShape<kType, kDirectMid, DirectMid>(ctx, v, g);
    default: return launchDirectShape<kType, kDirectWide, DirectWide>(ctx, v, g);
  }
}

}  // namespace plb
