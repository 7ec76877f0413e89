// Instances of the direct kernel for float operands.
#include "direct_launch.cuh"

namespace plb {

int launchDirectFloat(plb_context *ctx, const DirectVariant &v, const DirectArgs &g) {
  return launchDirectType<PLB_FLOAT>(ctx, v, g);
}

}  // namespace plb
