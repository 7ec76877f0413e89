// Instances of the implicit-GEMM kernel with 256-column tiles.
#include "igemm_dispatch.cuh"

namespace plb {

int launchIgemm256(plb_context *ctx, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &tout,
                   const IgemmArgs &args, const IgemmVariant &v) {
  return launchForTile<256>(ctx, ta, tb, tout, args, v);
}

}  // namespace plb
