// The rearranged form of a convolution whose input has too few channels for a TMA
// row (small_channel.cu), shared by the forward pass and the weight update.
#pragma once

#include <cuda_fp16.h>

#include "runtime.h"

namespace plb {

struct S2dShape {
  int N, H, W, C;       // input
  int s, padH, padW;    // stride (both dims), padding
  int KH, KW;
  int OH, OW;
  int Cp, C2;           // padded channels per original pixel, channels of X2
  int K2h, K2w;         // taps after folding the stride
  int H2, W2;           // extent of X2
};

int smallChannelShape(const plb_conv_params &p, S2dShape *g);
bool stemLayer(int sm_count, int plan_flags, const plb_conv_params &p, const plb_conv_options *opt, const void *d_out, bool slower_too, S2dShape *g);
size_t smallChannelElems(const S2dShape &g);
int smallChannelPrepare(plb_context *ctx, const S2dShape &g, const void *d_in, __half *x2, const void *d_weights,
                        __half *w2, int co);

}  // namespace plb
