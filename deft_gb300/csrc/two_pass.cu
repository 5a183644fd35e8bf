// Two-pass FP32 transforms of the y and x axes for lengths L = R1 R2: both
// passes run in registers and the elements cross shared memory once.
//
// A block holds B = 256 / R1 columns (adjacent in memory), column fastest
// across the threads:
//   natural holders   thread (j, b), j < R2: elements j + R2 s, s < R1
//   spectral holders  thread (k1, b), k1 < R1: frequencies k1 + R1 k2, k2 < R2
// natural -> spectral: R1-point DFTs over s, the exchange (slot
// (k1 R2 + j) B + b), the twiddles exp(S 2 pi i j k1 / L), R2-point DFTs over j.
// spectral -> natural runs the same steps backwards.  Loads and stores go
// straight between global memory and registers, R1 or R2 of them in flight a
// thread; the shared-memory Stockham kernels these replace staged every tile
// twice and waited at a barrier for each step (96^3: issue slots 60 to 70 %
// idle, stalled on loads, barriers and instruction fetches).
//
// The convolutions keep the spectrum (or the weighted sum) in the spectral
// holders' registers; exchanges alternate between two buffers, one barrier a
// transform.
//
// Measured in FP32 with events (mixed energy and gradient): 96^3 y transforms
// of five fields (two launches) 44 us by the shared-memory passes, 23 here,
// forward convolution 25 and 14.7, adjoint 27 and 14.3.  Against the pencils
// these also replace in FP32: 64^3 forward 17 and 11.5, adjoint 20.7 and 10.2;
// 128^3 24.1 and 20.8, 28.6 and 24.5, y transforms 52.5 and 52.4; 256^3 forward
// 151 and 138, adjoint 210 and 176, y transforms 419 and 312.  What is left is
// latency: five to ten dependent steps a block.
#include "two_pass.h"

#include "fft_smem.cuh"
#include "weights_f.cuh"

namespace deft {

namespace {

template <int SIGN, int R> __device__ __forceinline__ void dft_r(float2 *v) {
  if constexpr (R == 6) dft_pfa<SIGN, float, float2, 2, 3>(v);
  else if constexpr (R == 10) dft_pfa<SIGN, float, float2, 2, 5>(v);
  else if constexpr (R == 12) dft_pfa<SIGN, float, float2, 4, 3>(v);
  else dft_m<SIGN, float, float2, R>(v);
}

template <int R1> constexpr int tp_cols() { return 256 / R1; }
template <int R1, int R2> constexpr int tp_buf() { return R1 * R2 * tp_cols<R1>(); }

// Exchange and second half of natural -> spectral: v (the natural holders'
// R1-point DFTs) to u (X[k1 + R1 k2]).  Ends without a barrier: the buffer is
// free after the next one.
template <int SIGN, int R1, int R2>
__device__ __forceinline__ void tp_to_spectral(const float2 (&v)[R1], float2 (&u)[R2], float2 *xs,
                                               const float2 *__restrict__ tw) {
  constexpr int B = tp_cols<R1>();
  const int t = threadIdx.x, k1 = t / B;
  if (t < R2 * B) {
#pragma unroll
    for (int q = 0; q < R1; q++) xs[q * (R2 * B) + t] = v[q];
  }
  __syncthreads();
  if (t < R1 * B) {
    const float2 *p = xs + k1 * (R2 * B) + (t - k1 * B);
#pragma unroll
    for (int j = 0; j < R2; j++) u[j] = p[j * B];
#pragma unroll
    for (int j = 1; j < R2; j++) u[j] = c_mul(u[j], tw_load<SIGN>(tw, j * k1));
    dft_r<SIGN, R2>(u);
  }
}

// Spectral -> natural: u in, v[s] = y[j + R2 s] out.
template <int SIGN, int R1, int R2>
__device__ __forceinline__ void tp_to_natural(float2 (&u)[R2], float2 (&v)[R1], float2 *xs,
                                              const float2 *__restrict__ tw) {
  constexpr int B = tp_cols<R1>();
  const int t = threadIdx.x, k1 = t / B;
  if (t < R1 * B) {
    dft_r<SIGN, R2>(u);
    float2 *p = xs + k1 * (R2 * B) + (t - k1 * B);
    p[0] = u[0];
#pragma unroll
    for (int j = 1; j < R2; j++) p[j * B] = c_mul(u[j], tw_load<SIGN>(tw, j * k1));
  }
  __syncthreads();
  if (t < R2 * B) {
#pragma unroll
    for (int q = 0; q < R1; q++) v[q] = xs[q * (R2 * B) + t];
    dft_r<SIGN, R1>(v);
  }
}

// grid.x = tiles of B lines (x, kz), grid.y = field.
template <int SIGN, int R1, int R2>
__global__ void __launch_bounds__(256, 4)
    k_y_two_pass(float2 *data, Geom g, const float2 *__restrict__ tw) {
  constexpr int B = tp_cols<R1>();
  __shared__ float2 xs[tp_buf<R1, R2>()];
  const int t = threadIdx.x, j = t / B;
  const int l = blockIdx.x * B + (t - j * B);
  int x, kz;
  fdivmod(l < g.Nx * g.NzH ? l : 0, g.fNzH, x, kz);
  const bool act = l < g.Nx * g.NzH;
  float2 *p = data + (size_t)blockIdx.y * g.NC + (size_t)x * g.Ny * g.NzH + kz + j * g.NzH;
  float2 v[R1], u[R2];
  if (t < R2 * B) {
#pragma unroll
    for (int s = 0; s < R1; s++) v[s] = act ? p[R2 * s * g.NzH] : make_float2(0.f, 0.f);
    dft_r<SIGN, R1>(v);
  }
  tp_to_spectral<SIGN, R1, R2>(v, u, xs, tw);
  if (t < R1 * B && act) {
#pragma unroll
    for (int k2 = 0; k2 < R2; k2++) p[R1 * k2 * g.NzH] = u[k2];
  }
}

// Weights at the R2 frequencies a spectral holder has, in thread-private shared
// slots (as the pencils': in registers they would halve the resident warps).
__device__ __forceinline__ float &tp_wt(float *wts, int q, int a) {
  return wts[(q * 3 + a) * 256 + threadIdx.x];
}
template <int R1, int R2>
__device__ __forceinline__ void tp_weights(float *wts, const Geom &g, int k1, int y, int kz, float R,
                                           float (&kc)[3]) {
  const float yw = (float)wrapm(y, g.Ny), zf = (float)kz;
#pragma unroll
  for (int c = 0; c < 3; c++) kc[c] = g.Bmf[3 * c + 1] * yw + g.Bmf[3 * c + 2] * zf;
#pragma unroll 1
  for (int q = 0; q < R2; q++) {
    const float xw = (float)wrapm(k1 + R1 * q, R1 * R2);
    const float kx = g.Bmf[0] * xw + kc[0], ky = g.Bmf[3] * xw + kc[1], kzz = g.Bmf[6] * xw + kc[2];
    weights_at_f(kx * kx + ky * ky + kzz * kzz, R, (float)g.dr, (float)g.scale, tp_wt(wts, q, 0),
                 tp_wt(wts, q, 1), tp_wt(wts, q, 2));
  }
}
template <int R1, int R2> constexpr size_t tp_conv_smem() {
  return sizeof(float2) * 2 * tp_buf<R1, R2>() + sizeof(float) * 3 * R2 * 256;
}

// Forward convolution along x: the column's spectrum times w3, w2, i k_c wv,
// and the five inverse transforms.
template <int R1, int R2>
__global__ void __launch_bounds__(256, R1 > 12 ? 2 : 3)
    k_x_fwd_two_pass(const float2 *__restrict__ in, float2 *__restrict__ out5, Geom g,
                     const float2 *__restrict__ tw, const double *__restrict__ Rp) {
  constexpr int B = tp_cols<R1>(), L = R1 * R2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2 *xs = reinterpret_cast<float2 *>(smem_raw);
  float *wts = reinterpret_cast<float *>(xs + 2 * tp_buf<R1, R2>());
  const int t = threadIdx.x, j = t / B;
  const int J = g.Ny * g.NzH, col = blockIdx.x * B + (t - j * B);
  const bool act = col < J;
  const size_t at = (size_t)j * J + col;
  const int step = R2 * J;
  float2 v[R1], S[R2];
  if (t < R2 * B) {
#pragma unroll
    for (int s = 0; s < R1; s++) v[s] = act ? in[at + (size_t)s * step] : make_float2(0.f, 0.f);
  }
  int y, kz;
  fdivmod(act ? col : 0, g.fNzH, y, kz);
  float kc[3];
  tp_weights<R1, R2>(wts, g, j, y, kz, (float)*Rp, kc);
  if (t < R2 * B) dft_r<-1, R1>(v);
  tp_to_spectral<-1, R1, R2>(v, S, xs, tw);
#pragma unroll 1
  for (int a = 0; a < 5; a++) {
    const float kca = a == 2 ? kc[0] : a == 3 ? kc[1] : kc[2];
    const float bx = a == 2 ? g.Bmf[0] : a == 3 ? g.Bmf[3] : g.Bmf[6];
    float2 u[R2];
#pragma unroll
    for (int q = 0; q < R2; q++) {
      if (a < 2) {
        const float w = tp_wt(wts, q, a);
        u[q] = make_float2(S[q].x * w, S[q].y * w);
      } else {
        const float xw = (float)wrapm(j + R1 * q, L);
        const float w = (bx * xw + kca) * tp_wt(wts, q, 2);
        u[q] = make_float2(-S[q].y * w, S[q].x * w);  // times i w
      }
    }
    tp_to_natural<+1, R1, R2>(u, v, xs + ((a + 1) & 1) * tp_buf<R1, R2>(), tw);
    if (t < R2 * B && act) {
      float2 *dst = out5 + (size_t)a * g.NC + at;
#pragma unroll
      for (int s = 0; s < R1; s++) dst[(size_t)s * step] = v[s];
    }
  }
}

// Adjoint convolution along x: the five partial spectra times their weights
// (odd ones negated), summed, one inverse transform.  The next field is read
// while one is transformed, which is worth a third of the resident warps:
// two blocks an SM with it 14.3 us at 96^3 (32.7 at 144^3), three without 16.8
// (40.9), three with it, spilling, 18.4 (49.5).
template <int R1, int R2>
__global__ void __launch_bounds__(256, 2)
    k_x_adj_two_pass(const float2 *__restrict__ in5, float2 *__restrict__ out, Geom g,
                     const float2 *__restrict__ tw, const double *__restrict__ Rp) {
  constexpr int B = tp_cols<R1>(), L = R1 * R2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2 *xs = reinterpret_cast<float2 *>(smem_raw);
  float *wts = reinterpret_cast<float *>(xs + 2 * tp_buf<R1, R2>());
  const int t = threadIdx.x, j = t / B;
  const int J = g.Ny * g.NzH, col = blockIdx.x * B + (t - j * B);
  const bool act = col < J, nat = t < R2 * B;
  const size_t at = (size_t)j * J + col;
  const int step = R2 * J;
  float2 nx[R1], S[R2];
#pragma unroll
  for (int s = 0; s < R1; s++)
    nx[s] = nat && act ? in5[at + (size_t)s * step] : make_float2(0.f, 0.f);
#pragma unroll
  for (int q = 0; q < R2; q++) S[q] = make_float2(0.f, 0.f);
  int y, kz;
  fdivmod(act ? col : 0, g.fNzH, y, kz);
  float kc[3];
  tp_weights<R1, R2>(wts, g, j, y, kz, (float)*Rp, kc);
#pragma unroll 1
  for (int a = 0; a < 5; a++) {
    float2 v[R1], u[R2];
#pragma unroll
    for (int s = 0; s < R1; s++) v[s] = nx[s];
    if (a < 4 && nat && act) {
      const float2 *src = in5 + (size_t)(a + 1) * g.NC + at;
#pragma unroll
      for (int s = 0; s < R1; s++) nx[s] = src[(size_t)s * step];
    }
    if (nat) dft_r<-1, R1>(v);
    tp_to_spectral<-1, R1, R2>(v, u, xs + (a & 1) * tp_buf<R1, R2>(), tw);
    const float kca = a == 2 ? kc[0] : a == 3 ? kc[1] : kc[2];
    const float bx = a == 2 ? g.Bmf[0] : a == 3 ? g.Bmf[3] : g.Bmf[6];
    if (t < R1 * B) {
#pragma unroll
      for (int q = 0; q < R2; q++) {
        if (a < 2) {
          const float w = tp_wt(wts, q, a);
          S[q].x += u[q].x * w;
          S[q].y += u[q].y * w;
        } else {
          const float xw = (float)wrapm(j + R1 * q, L);
          const float w = (bx * xw + kca) * tp_wt(wts, q, 2);
          S[q].x += u[q].y * w;  // times -i w
          S[q].y -= u[q].x * w;
        }
      }
    }
  }
  float2 v[R1];
  tp_to_natural<+1, R1, R2>(S, v, xs + tp_buf<R1, R2>(), tw);
  if (nat && act) {
#pragma unroll
    for (int s = 0; s < R1; s++) out[at + (size_t)s * step] = v[s];
  }
}

template <int A, int B> struct Radices {
  static constexpr int R1 = A, R2 = B;
};

// Calls f(Radices<R1, R2>()) for length n (R1 >= R2); false if it has none.
template <typename F> bool with_radices(int n, F &&f) {
  switch (n) {
    case 32: f(Radices<8, 4>()); return true;
    case 64: f(Radices<8, 8>()); return true;
    case 128: f(Radices<16, 8>()); return true;
    case 256: f(Radices<16, 16>()); return true;
    case 36: f(Radices<6, 6>()); return true;
    case 40: f(Radices<8, 5>()); return true;
    case 48: f(Radices<8, 6>()); return true;
    case 50: f(Radices<10, 5>()); return true;
    case 60: f(Radices<10, 6>()); return true;
    case 72: f(Radices<12, 6>()); return true;
    case 80: f(Radices<10, 8>()); return true;
    case 96: f(Radices<12, 8>()); return true;
    case 100: f(Radices<10, 10>()); return true;
    case 120: f(Radices<12, 10>()); return true;
    case 144: f(Radices<12, 12>()); return true;
    case 160: f(Radices<16, 10>()); return true;
    case 192: f(Radices<16, 12>()); return true;
    default: return false;
  }
}

}  // namespace

bool two_pass_length(int n) {
  return with_radices(n, [](auto) {});
}

void two_pass_setup(int n) {
  with_radices(n, [](auto r) {
    constexpr int R1 = decltype(r)::R1, R2 = decltype(r)::R2;
    constexpr int smem = (int)tp_conv_smem<R1, R2>();
    cudaFuncSetAttribute(k_x_fwd_two_pass<R1, R2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(k_x_adj_two_pass<R1, R2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  });
}

void two_pass_y(float2 *data, const Geom &g, int nf, int sign, const float2 *tw,
                cudaStream_t stream) {
  with_radices(g.Ny, [&](auto r) {
    constexpr int R1 = decltype(r)::R1, R2 = decltype(r)::R2, B = tp_cols<R1>();
    const dim3 grid((g.Nx * g.NzH + B - 1) / B, nf);
    if (sign < 0) k_y_two_pass<-1, R1, R2><<<grid, 256, 0, stream>>>(data, g, tw);
    else k_y_two_pass<+1, R1, R2><<<grid, 256, 0, stream>>>(data, g, tw);
  });
}

void two_pass_x_fwd(const float2 *in, float2 *out5, const Geom &g, const float2 *tw,
                    const double *R, cudaStream_t stream) {
  with_radices(g.Nx, [&](auto r) {
    constexpr int R1 = decltype(r)::R1, R2 = decltype(r)::R2, B = tp_cols<R1>();
    constexpr size_t smem = tp_conv_smem<R1, R2>();
    k_x_fwd_two_pass<R1, R2>
        <<<(g.Ny * g.NzH + B - 1) / B, 256, smem, stream>>>(in, out5, g, tw, R);
  });
}

void two_pass_x_adj(const float2 *in5, float2 *out, const Geom &g, const float2 *tw,
                    const double *R, cudaStream_t stream) {
  with_radices(g.Nx, [&](auto r) {
    constexpr int R1 = decltype(r)::R1, R2 = decltype(r)::R2, B = tp_cols<R1>();
    constexpr size_t smem = tp_conv_smem<R1, R2>();
    k_x_adj_two_pass<R1, R2>
        <<<(g.Ny * g.NzH + B - 1) / B, 256, smem, stream>>>(in5, out, g, tw, R);
  });
}

}  // namespace deft
