// Instances of the direct kernel for quarter operands.
#include "direct_launch.cuh"

namespace plb {

int launchDirectQuarter(plb_context *ctx, const DirectVariant &v, const DirectArgs &g) {
  return launchDirectType<PLB_QUARTER>(ctx, v, g);
}

}  // namespace plb
