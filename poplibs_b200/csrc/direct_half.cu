// Instances of the direct kernel for half operands.
#include "direct_launch.cuh"

namespace plb {

int launchDirectHalf(plb_context *ctx, const DirectVariant &v, const DirectArgs &g) {
  return launchDirectType<PLB_HALF>(ctx, v, g);
}

}  // namespace plb
