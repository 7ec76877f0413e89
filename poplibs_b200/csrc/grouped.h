// Narrow channel groups contracted together as dense blocks (grouped.cu).
#pragma once

#include "runtime.h"

namespace plb {

// Groups per dense block (a divisor of `groups`; 1 = keep them apart).
uint32_t groupsTogether(uint32_t groups, uint32_t ci, uint32_t co, int type);
// Device word that a launch with IgemmProblem::nonfinite sets when a sum is not finite.
int *nonfiniteFlag(plb_context *ctx);
// Weights [groups][taps][rows][cols] as [groups/S][taps][S*rows][S*cols] in scratch;
// clears the flag.
int blockDiagonalWeights(plb_context *ctx, int type, const void *src, uint32_t groups, uint32_t S, uint32_t taps,
                         uint32_t rows, uint32_t cols, const void **out);
// Recomputes the outputs of `p` that are not finite if the flag is set.  `p`
// describes the separate groups on the caller's operands (of type `type`).
// Input position i of the problem is element i / in_dil of the operand (none if the
// division leaves a rest).
int repairNonFinite(plb_context *ctx, const IgemmProblem &p, int type, int in_dil_h = 1, int in_dil_w = 1);

}  // namespace plb
