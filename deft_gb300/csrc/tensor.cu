// Hard-sphere part of the tensor fundamental-measure functionals, FP64:
//
//   HardSpheresWB        src/HardSpheres.cpp:113-135 (White Bear, tensor third term)
//   HardSpheresTarazona  src/HardSpheres.cpp:90-111  (Rosenfeld prefactor)
//
// phi1 and phi2 are those of the vector form; phi3 = f3(n3) times
// TensorThirdTerm (src/HardSpheres.cpp:30-61):
//   n2^3 - 3 n2 |v|^2 + 9 (v.T.v - tr(T^3) / 2)
// with the tensor weighted densities T_ab = ab-shell (x) n
// (src/ReciprocalOperators.h:292-404).  Eleven weighted densities instead of
// five: they are formed and differentiated through the engine's own FP64
// r2c / c2r transforms (fft x dV, ifft x 1/V, the reference's convolution),
// rather than in the fused five-field pipeline: in double-float arithmetic as
// two sets of eleven convolutions (Engine::fan_out, fan_in) around one
// pointwise pass, the weights read from radial tables; in FP32 (the mixed
// form) and FP64 one field at a time.
#include <cmath>
#include <string>

#include "block_sum.cuh"
#include "df_phi.cuh"
#include "tensor.h"
#include "wb_phi.cuh"

namespace deft {
namespace {

constexpr int kThreads = 256;
constexpr int kBlocks = 1024;  // grid-stride kernels; fixed so the sums are reproducible
constexpr double kPi = 3.14159265358979323846;

__device__ __forceinline__ int wrap_index(int i, int N) { return i > N / 2 ? i - N : i; }

__device__ __forceinline__ void k_of(const Geom &g, int i, double k[3]) {
  int t, z, x, y;
  fdivmod(i, g.fNzH, t, z);
  fdivmod(t, g.fNy, x, y);
  const int m[3] = {wrap_index(x, g.Nx), wrap_index(y, g.Ny), z};
  for (int c = 0; c < 3; c++) k[c] = g.Bm[3 * c] * m[0] + g.Bm[3 * c + 1] * m[1] + g.Bm[3 * c + 2] * m[2];
}

// Weight a at k as wr + i wi: 0 step, 1 shell, 2-4 x/y/z vector shell
// (src/ReciprocalOperators.h:94-235), 5-10 tensor shells xx, yy, zz, xy,
// yz, zx (:292-404, 0 at k = 0).
__device__ void weight_at(int a, const double k[3], double R, double dr, double &wr, double &wi) {
  const double k2 = k[0] * k[0] + k[1] * k[1] + k[2] * k[2], kk = sqrt(k2), kR = kk * R;
  wr = 0;
  wi = 0;
  const double smear = exp(-6.0 * k2 * dr * dr);
  if (a < 5) {
    if (kR > 1e-3) {
      double s, c;
      sincos(kR, &s, &c);
      if (a == 0) wr = smear * (4 * kPi) * (s - kR * c) / (k2 * kk);
      else if (a == 1) wr = smear * (4 * kPi) * R * s / kk;
      else wi = smear * (4 * kPi) / k2 * (R * c - s / kk) * k[a - 2];
    } else {
      const double x = kR * kR;
      if (a == 0)
        wr = (4 * kPi / 3) * R * R * R * (x * x * x * (-1.0 / 15120) + x * x * (1.0 / 280) + x * (-1.0 / 10) + 1);
      else if (a == 1)
        wr = (4 * kPi) * (R * R) * (-x * x * x * (1.0 / 120 / 6 / 7) + x * x * (1.0 / 120) - x * (1.0 / 6) + 1);
      else
        wi = (4 * kPi) * R * R * R * (x * x * (1.0 / 5040 - 1.0 / 720) + x * (1.0 / 24 - 1.0 / 120) - 1.0 / 3) *
             k[a - 2];
    }
    return;
  }
  if (!(kR > 0)) return;
  double s, c;
  sincos(kR, &s, &c);
  if (a < 8) {
    const double c2 = k[a - 5] * k[a - 5] / k2;
    wr = smear * (4 * kPi * R * R) *
         (s / kR * (-1.0 / 3 + c2 - 3 * c2 / (kR * kR) + 1 / (kR * kR)) + c / (kR * kR) * (-1 + 3 * c2));
  } else {
    const int p = a - 8, q = (a - 8 + 1) % 3;  // xy, yz, zx
    wr = -smear * (4 * kPi) * k[p] * k[q] / (k2 * k2) * ((3 - kR * kR) * s / kR - 3 * c);
  }
}

// out = W_a F (forward convolution) or acc (+)= conj-adjoint W_a F (odd
// weights negated) for the gradient.
__global__ void k_tensor_weight(int a, Geom g, double R, const double2 *__restrict__ F,
                                double2 *__restrict__ out, int adjoint, int first) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.NC; i += gridDim.x * blockDim.x) {
    double k[3], wr, wi;
    k_of(g, i, k);
    weight_at(a, k, R, g.dr, wr, wi);
    if (adjoint) wi = -wi;
    const double2 f = F[i];
    const double2 t = {wr * f.x - wi * f.y, wr * f.y + wi * f.x};
    if (first || !adjoint) {
      out[i] = t;
    } else {
      const double2 o = out[i];
      out[i] = double2{o.x + t.x, o.y + t.y};
    }
  }
}

// FP64: phi3, phi1, phi2 per kT added to acc and, with d, the eleven partials.
__device__ __forceinline__ void tensor_point(int kind, double R, const double *w, double *acc,
                                             double *d) {
  const double a1 = 1 / (4 * kPi * R * R), a2 = 1 / (4 * kPi * R);
  const double n3 = w[0], n2 = w[1];
  const double v[3] = {w[2], w[3], w[4]};
  const double xx = w[5], yy = w[6], zz = w[7], xy = w[8], yz = w[9], zx = w[10];
  const double v2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
  const double u = 1 / (1 - n3), l = log(1 - n3);
  double f2[3], f3[3];
  hs_coeffs<double>(kind == 1 ? kHsRosenfeld : kHsWhiteBear, n3, u, l, f2, f3);
  const double Tv[3] = {xx * v[0] + xy * v[1] + zx * v[2], xy * v[0] + yy * v[1] + yz * v[2],
                        zx * v[0] + yz * v[1] + zz * v[2]};
  const double T2xx = xx * xx + xy * xy + zx * zx, T2yy = xy * xy + yy * yy + yz * yz,
               T2zz = zx * zx + yz * yz + zz * zz;
  const double T2xy = xx * xy + xy * yy + zx * yz, T2yz = xy * zx + yy * yz + yz * zz,
               T2zx = xx * zx + xy * yz + zx * zz;
  const double vTv = v[0] * Tv[0] + v[1] * Tv[1] + v[2] * Tv[2];
  const double tr3 = xx * T2xx + yy * T2yy + zz * T2zz + 2 * (xy * T2xy + yz * T2yz + zx * T2zx);
  const double t = n2 * n2 * n2 - 3 * n2 * v2 + 9 * (vTv - 0.5 * tr3);
  const double q = n2 * n2 - v2;
  acc[0] += f3[0] * t;
  acc[1] += -a1 * n2 * l;
  acc[2] += a2 * q * u;
  if (!d) return;
  const double g3 = f3[0];
  d[0] = a1 * n2 * u + a2 * q * u * u + f3[1] * t;
  d[1] = -a1 * l + 2 * a2 * n2 * u + g3 * 3 * q;
  for (int c = 0; c < 3; c++) d[2 + c] = -2 * a2 * u * v[c] + g3 * (-6 * n2 * v[c] + 18 * Tv[c]);
  d[5] = g3 * 9 * (v[0] * v[0] - 1.5 * T2xx);
  d[6] = g3 * 9 * (v[1] * v[1] - 1.5 * T2yy);
  d[7] = g3 * 9 * (v[2] * v[2] - 1.5 * T2zz);
  d[8] = g3 * 9 * (2 * v[0] * v[1] - 3 * T2xy);
  d[9] = g3 * 9 * (2 * v[1] * v[2] - 3 * T2yz);
  d[10] = g3 * 9 * (2 * v[2] * v[0] - 3 * T2zx);
}

// Per-block sums of kT phi3, kT phi1, kT phi2.
__device__ __forceinline__ void store_sums(double (&acc)[3], double kT, double *partials) {
  __shared__ double red[32 * 3];
  block_reduce<3>(acc, red);
  if (threadIdx.x == 0)
    for (int k = 0; k < 3; k++) partials[3 * blockIdx.x + k] = kT * acc[k];
}

// phi and its eleven partials at each point, FP64; per-block sums into
// partials[3 * block + term]; part[a] = dV kT dphi/dw_a.
__global__ void __launch_bounds__(kThreads)
    k_tensor_phi(int kind, double R, double kT, double dV, const double *__restrict__ w, int NR,
                 double *__restrict__ part, double *__restrict__ partials) {
  double acc[3] = {0, 0, 0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NR; i += gridDim.x * blockDim.x) {
    double wl[11], d[11];
    for (int a = 0; a < 11; a++) wl[a] = w[(size_t)a * NR + i];
    tensor_point(kind, R, wl, acc, part ? d : nullptr);
    if (part)
      for (int a = 0; a < 11; a++) part[(size_t)a * NR + i] = dV * kT * d[a];
  }
  store_sums(acc, kT, partials);
}

// The FP64 formulas for points outside the double-float range.
__device__ __noinline__ void tensor_point_fp64(int kind, double R, double c, const dfl *w,
                                               double *acc, dfl *d) {
  double wl[11], g[11];
  for (int a = 0; a < 11; a++) wl[a] = to_double(w[a]);
  tensor_point(kind, R, wl, acc, g);
  for (int a = 0; a < 11; a++) d[a] = df_from(c * g[a]);
}

// The same in double-float arithmetic, in place (w becomes the partials where
// grad): about 150 double-float operations a point against 200 of the FP64
// pipe, and no conversions (96 x 80 x 100: 310 -> 55 us).
__global__ void __launch_bounds__(kThreads, 2)
    k_tensor_phi_df(int kind, double R, double kT, double c, DfPhiConst k,
                    const double *__restrict__ n, dfl *__restrict__ w, int NR, int grad,
                    double *__restrict__ partials) {
  double acc[3] = {0, 0, 0}, rare[3] = {0, 0, 0};
#pragma unroll 1
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NR; i += gridDim.x * blockDim.x) {
    dfl x[11];
#pragma unroll
    for (int a = 0; a < 11; a++) x[a] = w[(size_t)a * NR + i];
    const dfl n3 = x[0], n2 = x[1], om = df_one_minus(n3);
    const dfl *v = x + 2;
    const dfl v2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
    if (!df_point_ok(om, n2, v2, n[i] != 0)) {
      dfl xl[11], d[11];
      for (int a = 0; a < 11; a++) xl[a] = x[a];
      tensor_point_fp64(kind, R, c, xl, rare, d);
      if (grad)
        for (int a = 0; a < 11; a++) w[(size_t)a * NR + i] = d[a];
      continue;
    }
    const dfl xx = x[5], yy = x[6], zz = x[7], xy = x[8], yz = x[9], zx = x[10];
    const dfl Tv[3] = {xx * v[0] + xy * v[1] + zx * v[2], xy * v[0] + yy * v[1] + yz * v[2],
                       zx * v[0] + yz * v[1] + zz * v[2]};
    const dfl sxy = xy * xy, syz = yz * yz, szx = zx * zx;
    const dfl T2xx = xx * xx + sxy + szx, T2yy = sxy + yy * yy + syz, T2zz = szx + syz + zz * zz;
    const dfl T2xy = xy * (xx + yy) + zx * yz, T2yz = yz * (yy + zz) + xy * zx,
              T2zx = zx * (xx + zz) + xy * yz;
    const dfl vTv = v[0] * Tv[0] + v[1] * Tv[1] + v[2] * Tv[2];
    const dfl tr3 = xx * T2xx + yy * T2yy + zz * T2zz +
                    df_ldexp(xy * T2xy + yz * T2yz + zx * T2zx, 2.0f);
    const dfl n22 = n2 * n2, q = n22 - v2;
    const dfl t = n2 * (n22 - df_scale(v2, 3.0f)) + df_scale(vTv - df_ldexp(tr3, 0.5f), 9.0f);
    const dfl u = df_rcp(om), u2 = u * u, l = df_log1m(n3, om);
    dfl f3 = u2, df3;
    if (kind == 1) {
      df3 = df_ldexp(u2 * u, 2.0f);
    } else {
      dfl S, dS;
      df_S(n3, om, l, S, dS);
      f3 = S * u2;
      df3 = (dS + df_ldexp(S * u, 2.0f)) * u2;
    }
    const dfl p[3] = {f3 * t, n2 * l, q * u};
#pragma unroll
    for (int m = 0; m < 3; m++) {
      acc[m] += f2d(p[m].hi);
      acc[m] += f2d(p[m].lo);
    }
    if (!grad) continue;
    const dfl f3k = k.k3 * f3, n2u = n2 * u;
    w[i] = k.a1 * n2u + (k.a2 * q) * u2 + (k.k3 * df3) * t;
    w[(size_t)NR + i] = k.a2x2 * n2u - k.a1 * l + df_scale(f3k * q, 3.0f);
    const dfl cv = -(k.a2x2 * u + df_scale(f3k * n2, 6.0f)), f18 = df_scale(f3k, 18.0f);
#pragma unroll
    for (int e = 0; e < 3; e++) w[(size_t)(2 + e) * NR + i] = cv * v[e] + f18 * Tv[e];
    const dfl f9 = df_ldexp(f18, 0.5f);
    w[(size_t)5 * NR + i] = f9 * (v[0] * v[0] - df_scale(T2xx, 1.5f));
    w[(size_t)6 * NR + i] = f9 * (v[1] * v[1] - df_scale(T2yy, 1.5f));
    w[(size_t)7 * NR + i] = f9 * (v[2] * v[2] - df_scale(T2zz, 1.5f));
    w[(size_t)8 * NR + i] = f9 * (df_ldexp(v[0] * v[1], 2.0f) - df_scale(T2xy, 3.0f));
    w[(size_t)9 * NR + i] = f9 * (df_ldexp(v[1] * v[2], 2.0f) - df_scale(T2yz, 3.0f));
    w[(size_t)10 * NR + i] = f9 * (df_ldexp(v[2] * v[0], 2.0f) - df_scale(T2zx, 3.0f));
  }
  acc[0] = fma(acc[0], k.s0, rare[0]);
  acc[1] = fma(acc[1], k.s1, rare[1]);
  acc[2] = fma(acc[2], k.s2, rare[2]);
  store_sums(acc, kT, partials);
}

// Fixed-order sums of the block partials, times dV: a block per term.
__global__ void __launch_bounds__(kThreads)
    k_tensor_sum(const double *__restrict__ partials, int nblk, double dV,
                 double *__restrict__ out) {
  __shared__ double red[32];
  double x[1] = {0};
  for (int b = threadIdx.x; b < nblk; b += kThreads) x[0] += partials[3 * b + blockIdx.x];
  block_reduce<1>(x, red);
  if (threadIdx.x == 0) out[blockIdx.x] = x[0] * dV;
}

// dst += src, masked as constrain() masks a gradient (0 where mask is 0).
__global__ void k_add_masked(const double *__restrict__ src, const double *__restrict__ mask,
                             double *__restrict__ dst, int N) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
    const double v = src[i];
    dst[i] += mask ? (mask[i] == 0 ? 0.0 : mask[i] * v) : v;
  }
}

}  // namespace

int add_masked(Engine *e, const double *src, const double *mask, double *dst) {
  const int N = e->geom().NR;
  k_add_masked<<<kBlocks, kThreads, 0, e->stream()>>>(src, mask, dst, N);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

size_t tensor_scratch_doubles(const Geom &g) {
  // one field at a time: spectrum of n, work spectrum, accumulator, 11 weighted
  // densities and 11 partials; double-float: 11 spectra and 11 fields (the
  // partials take the weighted densities' place).  Block partials and the
  // three sums.
  const size_t one = 6 * (size_t)g.NC + 22 * (size_t)g.NR;
  const size_t df = 22 * (size_t)g.NC + 11 * (size_t)g.NR;
  return (one > df ? one : df) + 3 * kBlocks + 4;
}

int tensor_hs(Engine *e, const FmtSpec &f, const double *n, double *scratch, double *grad,
              double terms3[3], std::string *err) {
  const Geom &g = e->geom();
  cudaStream_t s = e->stream();
  const int NR = g.NR, NC = g.NC;
  double *partials = scratch, *sums = partials + 3 * kBlocks;
  double *fields = sums + 3 + (3 * kBlocks + 3) % 2;  // 16-byte aligned (kBlocks is even)
  auto fail = [&](const char *what) {
    if (err) *err = std::string("tensor functional: ") + what;
    return -1;
  };
  const int kind = f.hs == kHsTarazona ? 1 : 0;
  auto finish = [&]() {
    cudaError_t ce = cudaMemcpyAsync(terms3, sums, 3 * sizeof(double), cudaMemcpyDeviceToHost, s);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
    if (ce == cudaSuccess) ce = cudaGetLastError();
    if (ce == cudaSuccess) return 0;
    if (err) *err = std::string("tensor functional: ") + cudaGetErrorString(ce);
    return -1;
  };
  if (f.precision != kPrecisionMixed && e->df_on()) {
    dfc *spec = reinterpret_cast<dfc *>(fields);
    dfl *w = reinterpret_cast<dfl *>(spec + 11 * (size_t)NC);
    const dfl *step = e->radial(kRadStep, f.R), *shell = e->radial(kRadShell, f.R),
              *vec = e->radial(kRadVShell, f.R), *ta = e->radial(kRadTensorA, f.R),
              *tb = e->radial(kRadTensorB, f.R);
    if (!step || !shell || !vec || !ta || !tb) return fail("weight tables");
    FieldWeights fw;
    fw.add(kWtScalar, step, nullptr, 4 * kPi / 3 * f.R * f.R * f.R * g.scale);
    fw.add(kWtScalar, shell, nullptr, 4 * kPi * f.R * f.R * g.scale);
    for (int c = 0; c < 3; c++) fw.add(kWtVector + c, vec);
    for (int c = 0; c < 3; c++) fw.add(kWtDiag + c, ta, tb);
    for (int c = 0; c < 3; c++) fw.add(kWtXY + c, nullptr, tb);
    if (e->spectrum(n) || e->fan_out(fw, 1, spec, w)) return fail(e->last_error());
    WbRadius wr;
    wb_radius(wr, f.R, kind == 1 ? kHsRosenfeld : kHsWhiteBear);
    const double c = g.dV * f.kT;
    k_tensor_phi_df<<<kBlocks, kThreads, 0, s>>>(kind, f.R, f.kT, c, df_phi_const(wr, c), n, w, NR,
                                                 grad != nullptr, partials);
    k_tensor_sum<<<3, kThreads, 0, s>>>(partials, kBlocks, g.dV, sums);
    if (grad && e->fan_in(fw, -1, w, spec, grad)) return fail(e->last_error());
    return finish();
  }
  double2 *Nk = reinterpret_cast<double2 *>(fields);
  double2 *tmp = Nk + NC, *acc = tmp + NC;
  double *w = reinterpret_cast<double *>(acc + NC);
  double *part = w + 11 * (size_t)NR;
  // the mixed form runs the transforms in FP32 (Phi and its partials FP64)
  const Engine::Arith arith =
      f.precision == kPrecisionMixed ? Engine::kArithFP32 : Engine::kArithDF;
  const int cblocks = (NC + kThreads - 1) / kThreads < 4096 ? (NC + kThreads - 1) / kThreads : 4096;
  if (e->fft(n, Nk, arith)) return fail("fft");
  for (int a = 0; a < 11; a++) {
    k_tensor_weight<<<cblocks, kThreads, 0, s>>>(a, g, f.R, Nk, tmp, 0, 1);
    if (e->ifft(tmp, w + (size_t)a * NR, arith)) return fail("ifft");
  }
  k_tensor_phi<<<kBlocks, kThreads, 0, s>>>(kind, f.R, f.kT, g.dV, w, NR, grad ? part : nullptr,
                                            partials);
  k_tensor_sum<<<3, kThreads, 0, s>>>(partials, kBlocks, g.dV, sums);
  if (grad) {
    for (int a = 0; a < 11; a++) {
      if (e->fft(part + (size_t)a * NR, tmp, arith)) return fail("fft");
      k_tensor_weight<<<cblocks, kThreads, 0, s>>>(a, g, f.R, tmp, acc, 1, a == 0);
    }
    if (e->ifft(acc, grad, arith)) return fail("ifft");
  }
  return finish();
}

}  // namespace deft
