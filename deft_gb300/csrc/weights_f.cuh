// FP32 helpers of the k-space convolutions.
#pragma once

#include <cuda_runtime.h>

namespace deft {

// Signed frequency of index i of N.
__device__ __forceinline__ int wrapm(int i, int N) { return i > N / 2 ? i - N : i; }

// The analytic weights at |k| (src/ReciprocalOperators.h:94-142,162-235: step w3,
// shell w2, the radial factor wv of the vector shells) in FP32, evaluated on the fly in the convolution kernels
// (scale = dV/V folded in).  Below kR = 0.5 the closed forms lose digits to
// cancellation in FP32, so the Taylor series of the reference's small-kR
// branch is used there, times the smear factor (which is not 1 to FP32
// precision at that threshold; at kR <= 1e-3, where the FP64 branch omits it,
// the two differ by at most 6 (k dr)^2 < 3e-7).
__device__ __forceinline__ void weights_at_f(float k2, float R, float dr, float scale, float &w3,
                                             float &w2, float &wv) {
  const float kk = sqrtf(k2);
  const float kR = kk * R;
  const float kdr = kk * dr;
  const float smear = expf(-6.0f * kdr * kdr) * scale;
  const float fpi = 12.566370614359172954f;
  if (kR > 0.5f) {
    float sn, cs;
    sincosf(kR, &sn, &cs);
    const float ik = 1.0f / kk;
    w3 = smear * fpi * (sn - kR * cs) * ik * ik * ik;
    w2 = smear * fpi * R * sn * ik;
    wv = smear * fpi * ik * ik * (R * cs - sn * ik);
  } else {
    const float x = kR * kR, R3 = R * R * R;
    w3 = smear * (fpi / 3) * R3 * (((-1.0f / 15120) * x + 1.0f / 280) * x - 0.1f) * x + smear * (fpi / 3) * R3;
    w2 = smear * fpi * R * R * ((((-1.0f / 5040) * x + 1.0f / 120) * x - 1.0f / 6) * x + 1.0f);
    wv = smear * fpi * R3 * (((1.0f / 5040 - 1.0f / 720) * x + (1.0f / 24 - 1.0f / 120)) * x -
                             1.0f / 3);
  }
}

}  // namespace deft
