// Forward convolutions of few input channels in one launch, straight from the caller's
// tensors (stem.cu).
#pragma once

#include "runtime.h"
#include "small_channel.h"

namespace plb {

// Whether the layer (g: smallChannelShape of it) runs on the stem kernel.
// (`slower_too`: whatever the rearranged form takes)
bool stemSuits(int sm_count, const S2dShape &g, int co, bool out_f32, const void *out, bool slower_too);
int launchStem(plb_context *ctx, const S2dShape &g, int co, bool bf16, const void *x, const void *w, const float *bias,
               void *out);

}  // namespace plb
