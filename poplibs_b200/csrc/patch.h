// Convolutions of narrow channel groups and small ragged layers from input patches in
// shared memory (patch.cuh, patch.cu).
#pragma once

#include "rows.h"
#include "runtime.h"

namespace plb {

// Problems of one launch: the phases of a strided layer's input gradient, else one.
constexpr int kPatchMaxPhases = 4;

// Whether these problems (same operands, groups and channel counts; `type` is the
// operands' element type, all pointers are the caller's) run on the patch kernel.
// The general route: `contractions` launches, of `together` groups as one, on copies of the
// operands (`copied`); `packed`: it gathers the channels of several taps into one operand row.
// `slower_too`: by the first estimates alone.  Where the kernel for the rows of narrow groups is to
// take the place of the patch kernel, `rows` is its tiling, else its blocks are 0.
bool patchSuits(int sm_count, const IgemmProblem *p, int n, int type, int contractions, int together, bool copied, bool packed,
                bool slower_too, RowsTiling *rows);
// `repair`: outputs whose sum is not finite are formed again without the products
// with padding, as repairNonFinite does.
int launchPatch(plb_context *ctx, const IgemmProblem *p, int n, int type, bool repair);

}  // namespace plb
