// Weight and bias gradients of the U-Net's 3x3x3 convolutions (unet_wgrad.cu).
#pragma once

#include <stdint.h>

namespace nusif {

// one channels-last BF16 source of a layer's input; up: stored at half
// resolution and read by nearest upsampling
struct WgradSrc {
  const void *p;
  int c;  // channels, a multiple of 16; 0: none
  int up;
};

// floats of scratch that wgrad_conv needs for this layer
int64_t wgrad_scratch(int co, int ci, int B, int Z, int Y, int X);

// dw[27][co][ci] = sum over cells of G[cell][o] X[cell + tap][i], db[co] = sum
// of G: G BF16 [cells][co], or FP32 [cells] (co 1, g32) used exactly; X the
// channel concat of s0 and s1, of whose channels the first ci are stored
bool wgrad_conv(const WgradSrc &s0, const WgradSrc &s1, const void *g, const float *g32, int co,
    int ci, int B, int Z, int Y, int X, float *scratch, float *dw, float *db);

}  // namespace nusif
