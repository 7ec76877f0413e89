// Instances of the patch kernel for float operands.
#include "patch_launch.cuh"

namespace plb {

int launchPatchFloat(plb_context *ctx, const PatchVariant &v, const PatchArgs &g) {
  return launchPatchType<PLB_FLOAT>(ctx, v, g);
}

}  // namespace plb
