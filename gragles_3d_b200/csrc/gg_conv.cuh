// gg_conv.cuh -- launch interface of the convolution passes.
#pragma once

#include <cuda_runtime.h>
#include <cstddef>

namespace gg {

struct ConvArgs {
    int G;
    const int* toff;          // tile offsets (G + 2): n tiles per convolved grain
    const double* in;         // input arena
    const int* in_box;
    const long long* in_off;
    double* out;              // output arena (same boxes as the input)
    const long long* out_off;
    double2* spec;            // half-spectrum scratch
    const long long* spec_off;
    const double2* tw;        // (cos, sin) twiddles for every side n, at tw_off[n]
    const long long* tw_off;
    const double* gtab;       // Gaussian multiplier by S = i2^2+j2^2+k2^2, at g_off[n]
    const long long* g_off;
};

// Largest box side the FP64 convolution takes: a chosen bound, up to which it is tested.  (The
// passes hold lines, not planes: at most 39 KB a warp at this side.)
constexpr int kConvF64MaxSide = 97;
// Five launches; nmax: the largest side among the boxes of the tiles.
void launch_conv_f64(const ConvArgs& a, int nmax, cudaStream_t s);

}  // namespace gg
