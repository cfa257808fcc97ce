// Tensor-core (tcgen05) 3x3x3 convolutions of the U-Net (unet_tc.cu).
#pragma once

namespace nusif {

// the volume and channel counts have a tcgen05 kernel: tiles of 128 cells
// cover whole x-rows (x <= 128 dividing 128, y a multiple of 128 / x) or
// 128-cell pieces of longer rows; 16-channel input groups; 16..96 outputs
bool tc_conv_supported(int X, int Y, int Z, int B, int N, int C0, int C1);

// what a convolution stores per cell
enum TcOut {
  TC_BF16,    // [N] BF16
  TC_F32,     // [N] FP32
  TC_ONE,     // channel 0, FP32 (a 1-channel layer whose weights are padded to 16 rows)
  TC_MASKED,  // [N] BF16, zero where the mask [cells][N] (BF16) is not positive
  TC_SPLIT    // FP32, the first 32 channels to out, the other 16 to out2
};

// out[cell] = act(sum over taps and input channels of in[cell + tap][c] *
// w[tap][N][c] + bias), zero padding; the input is the channel concat of two
// channels-last BF16 volumes s0 (C0) and s1 (C1, 0: none); w BF16
// [27][N][C0 + C1]; *err is set when a wait timed out. Where
// tc_conv_marches(N, C0 + C1) is false the output is TC_BF16 or TC_F32 and
// up0 (s0 at half resolution, read by nearest upsampling) is 0.
bool tc_conv_marches(int N, int C);
bool tc_conv(const void *s0, int C0, const void *s1, int C1, int B, int Z, int Y, int X,
    const void *w, int N, const float *bias, int relu, TcOut kind, void *out, int *err,
    int up0 = 0, const void *mask = nullptr, void *out2 = nullptr);

}  // namespace nusif
