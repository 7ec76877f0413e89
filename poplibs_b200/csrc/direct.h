// Matrix products that read their operands where they lie (direct.cuh, direct.cu).
#pragma once

#include "runtime.h"

namespace plb {

// The product as gemmProblem describes it, on the caller's operands of element type
// `type`.  `copied`: the implicit-GEMM kernel could only read a copy of an operand.
// `slower_too`: whatever that takes.
bool directSuits(int sm_count, const IgemmProblem &p, int type, bool copied, bool slower_too);
int launchDirect(plb_context *ctx, const IgemmProblem &p, int type);

}  // namespace plb
