// Two-pass FP32 transforms of the y and x axes (two_pass.cu).
#pragma once

#include <cuda_runtime.h>

#include "fmt_engine.h"

namespace deft {

// Whether lines of length n have two-pass kernels.
bool two_pass_length(int n);
// Shared-memory caps of the x kernels for length n (once per engine).
void two_pass_setup(int n);

// In-place transform of nf half-complex fields along y, of sign `sign`
// (unnormalised); tw: the Ny roots exp(-2 pi i t / Ny).
void two_pass_y(float2 *data, const Geom &g, int nf, int sign, const float2 *tw,
                cudaStream_t stream);
// The forward and adjoint convolutions along x (as k_x_conv_fwd, k_x_conv_adj);
// R: device address of the hard-sphere radius.
void two_pass_x_fwd(const float2 *in, float2 *out5, const Geom &g, const float2 *tw,
                    const double *R, cudaStream_t stream);
void two_pass_x_adj(const float2 *in5, float2 *out, const Geom &g, const float2 *tw,
                    const double *R, cudaStream_t stream);

}  // namespace deft
