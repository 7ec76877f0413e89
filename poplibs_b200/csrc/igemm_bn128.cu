// Instances of the implicit-GEMM kernel with 128-column tiles.
#include "igemm_dispatch.cuh"

namespace plb {

int launchIgemm128(plb_context *ctx, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &tout,
                   const IgemmArgs &args, const IgemmVariant &v) {
  return launchForTile<128>(ctx, ta, tb, tout, args, v);
}

}  // namespace plb
