// Instances of the patch kernel for half operands.
#include "patch_launch.cuh"

namespace plb {

int launchPatchHalf(plb_context *ctx, const PatchVariant &v, const PatchArgs &g) {
  return launchPatchType<PLB_HALF>(ctx, v, g);
}

}  // namespace plb
