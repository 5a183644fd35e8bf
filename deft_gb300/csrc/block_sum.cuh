// Fixed-order FP64 sums over warps and blocks.
#pragma once

#include <cuda_runtime.h>

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

}  // namespace deft
