// Fixed-order FP64 and double-float sums over warps and blocks.
#pragma once

#include <cuda_runtime.h>

#include "dfloat.cuh"

namespace deft {

// Sums K doubles over a warp: at each of the first steps a lane keeps half of
// the values it still holds and sends the other half away, so six values
// take eight FP64 additions a lane instead of thirty (a warp-wide addition
// occupies a scheduler's FP64 pipe for 64 cycles).  On return v[0] holds the
// sum of value warp_sum_slot<K>(lane) (-1: padding).
template <int K, int O, typename A>
__device__ __forceinline__ void warp_sum_step(A &v, int lane) {
  if constexpr (O > 0) {
    if constexpr (K == 1) {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
      warp_sum_step<1, O / 2>(v, lane);
    } else {
      constexpr int H = (K + 1) / 2;
      const bool up = lane & O;
#pragma unroll
      for (int i = 0; i < H; i++) {
        const double hi = H + i < K ? v[H + i < K ? H + i : 0] : 0.0;
        const double send = up ? v[i] : hi;
        v[i] = (up ? hi : v[i]) + __shfl_xor_sync(0xffffffffu, send, O);
      }
      warp_sum_step<H, O / 2>(v, lane);
    }
  }
}
template <int K, int O = 16> __device__ __forceinline__ int warp_sum_slot(int lane) {
  if constexpr (K == 1 || O == 0) {
    return 0;
  } else {
    constexpr int H = (K + 1) / 2;
    const int s = warp_sum_slot<H, O / 2>(lane);
    const int t = s + ((lane & O) ? H : 0);
    return s >= 0 && t < K ? t : -1;
  }
}
// Lanes that share a slot's sum differ in the low bits only: one writes it.
template <int K> __host__ __device__ constexpr int warp_sum_same() {
  int k = K, o = 32;
  while (k > 1) {
    k = (k + 1) / 2;
    o /= 2;
  }
  return o;  // lanes per slot
}
template <int K>
__device__ __forceinline__ void warp_sum_store(double (&v)[K], double *dst /* K */) {
  const int lane = threadIdx.x & 31;
  warp_sum_step<K, 16>(v, lane);
  const int slot = warp_sum_slot<K>(lane);
  if (slot >= 0 && lane % warp_sum_same<K>() == 0) dst[slot] = v[0];
}

// Deterministic block reduction of K doubles; thread 0 gets the sums (lane k
// of the first warp adds the warps' sums of value k, in order).
template <int K>
__device__ __forceinline__ void block_reduce(double (&v)[K], double *smem /* 32*K */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  warp_sum_store<K>(v, smem + warp * K);
  __syncthreads();
  if (warp == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    double s = 0;
    if (lane < K)
      for (int w = 0; w < nw; w++) s += smem[w * K + lane];
#pragma unroll
    for (int k = 0; k < K; k++) v[k] = __shfl_sync(0xffffffffu, s, k);
  }
}

// The same for the FP32 kernels' per-thread sums, in double-float (2^-47 a step
// against the terms' own 2^-24): no FP64 addition but the last one.  Three
// values over a warp are about 170 issue slots instead of 10 x 64 cycles of
// FP64 pipe; the Hessian product's last stage at 96^3 (its dot in FP64) spent 2
// of 17 us there, the gradient with two dots 4 of 22.
template <int K>
__device__ __forceinline__ void block_reduce(const float (&x)[K], double (&v)[K],
                                             double *smem /* 32*K */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  dfl *part = reinterpret_cast<dfl *>(smem);
#pragma unroll
  for (int k = 0; k < K; k++) {
    dfl r = df_two_sum(x[k], __shfl_xor_sync(0xffffffffu, x[k], 16));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
      r += dfl(__shfl_xor_sync(0xffffffffu, r.hi, o), __shfl_xor_sync(0xffffffffu, r.lo, o));
    if (lane == 0) part[warp * K + k] = r;
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    dfl s(0.f, 0.f);
    if (lane < K)
      for (int w = 0; w < nw; w++) s += part[w * K + lane];
    const double d = double(s);
#pragma unroll
    for (int k = 0; k < K; k++) v[k] = __shfl_sync(0xffffffffu, d, k);
  }
}

}  // namespace deft
