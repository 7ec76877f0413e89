// Instances of the patch kernel for quarter operands.
#include "patch_launch.cuh"

namespace plb {

int launchPatchQuarter(plb_context *ctx, const PatchVariant &v, const PatchArgs &g) {
  return launchPatchType<PLB_QUARTER>(ctx, v, g);
}

}  // namespace plb
