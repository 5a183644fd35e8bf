// Water SAFT association and dispersion terms (src/haskell/WaterSaft.hs:35-104,
// the compiled form src/WaterSaftFast.cpp), with their exact gradient; FP64,
// or with every transform in FP32 in the mixed form (pointwise work FP64):
//
//   F_disp  = int n a1 + int n a2 / kT
//     eta_d = (4 pi R^3 / 3) ifft(exp(-k^2 (2 ls lambda R)^2 / 2) fft n)
//     a1 = -4 (lambda^3 - 1) eps_d eta_d g(eta_eff),  g(x) = (1 - x/2) / (1 - x)^3,
//     eta_eff = (c1 + c2 eta_d + c3 eta_d^2) eta_d     (Gil-Villegas 1997, eq. 36)
//     a2 = K_HS eps_d eta_d (d a1 / d eta_d) / 2,  K_HS = (1 - eta_d)^4 / (1 + 2 eta_d)^2
//   F_assoc = int 4 kT n (ln X - X/2 + 1/2),  X = (sqrt(1 + 8 y) - 1) / (4 y),
//     y = nA Delta, nA = shell_2R(n) / (4 pi (2R)^2), Delta = gSW kappa_a (exp(eps_a/kT) - 1)
//     gSW = gSigmaA + (d a1/d eta_d - lambda / (3 eta_d) d a1/d lambda) / (4 kT)
//
// gSigmaA is the contact-value field of contact.cu (eight convolutions of
// pointwise functions of the weighted densities, over shell_2R(n)).  The
// gradient follows every convolution back: per point the adjoints of the
// pointwise chain (X from y, y from nA and Delta, gSW from gSigmaA and
// eta_d), then the adjoint of gSigmaA's eight convolutions, the Jacobian
// of its source fields in the weighted densities (second derivatives of
// phi), and the adjoint weighted-density, shell_2R and Gaussian convolutions.
// The White Bear, ideal-gas, mu and mask parts come from the fused
// evaluator; this module adds the two SAFT terms.
#include <cmath>
#include <string>

#include "block_sum.cuh"
#include "contact_math.cuh"
#include "df_phi.cuh"
#include "saft.h"

namespace deft {
namespace {

constexpr int kThreads = 256;
constexpr int kBlocks = 1024;  // fixed, so the energy sums are reproducible
using cm::kPi;

__device__ void a1_terms(double eta, double lam, double eps, double o[5]) {
  const double c[3] = {2.25855 - 1.50349 * lam + 0.249434 * lam * lam,
                       -0.669270 + 1.40049 * lam - 0.827739 * lam * lam,
                       10.1576 - 15.0427 * lam + 5.30827 * lam * lam};
  const double cl[3] = {-1.50349 + 2 * 0.249434 * lam, 1.40049 - 2 * 0.827739 * lam,
                        -15.0427 + 2 * 5.30827 * lam};
  const double x = (c[0] + c[1] * eta + c[2] * eta * eta) * eta;
  const double xe = c[0] + 2 * c[1] * eta + 3 * c[2] * eta * eta, xee = 2 * c[1] + 6 * c[2] * eta;
  const double xl = (cl[0] + cl[1] * eta + cl[2] * eta * eta) * eta;
  const double xel = cl[0] + 2 * cl[1] * eta + 3 * cl[2] * eta * eta;
  const double om = 1 - x, om2 = om * om;
  const double g = (1 - x / 2) / (om2 * om), g1 = (2.5 - x) / (om2 * om2),
               g2 = (9 - 3 * x) / (om2 * om2 * om);
  const double L3 = lam * lam * lam - 1, pre = -4 * eps;
  o[0] = pre * L3 * eta * g;                                          // a1
  o[1] = pre * L3 * (g + eta * g1 * xe);                              // d a1 / d eta
  o[2] = pre * eta * (3 * lam * lam * g + L3 * g1 * xl);              // d a1 / d lambda
  o[3] = pre * L3 * (2 * g1 * xe + eta * (g2 * xe * xe + g1 * xee));  // d2 a1 / d eta2
  o[4] = pre * (3 * lam * lam * (g + eta * g1 * xe) +
                L3 * (g1 * xl + eta * (g2 * xl * xe + g1 * xel)));    // d2 a1 / d eta d lambda
}

// The eight source fields of gSigmaA (White Bear partials, computed once
// per point): src + a NR, a < 8.
__global__ void k_saft_sources(double R, const double *__restrict__ w, int NR,
                               double *__restrict__ src) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NR; i += gridDim.x * blockDim.x) {
    const double v[3] = {w[2 * (size_t)NR + i], w[3 * (size_t)NR + i], w[4 * (size_t)NR + i]};
    const cm::Partials p = cm::partials(kHsWhiteBear, R, w[i], w[(size_t)NR + i],
                                        v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
#pragma unroll
    for (int a = 0; a < 8; a++) src[(size_t)a * NR + i] = cm::gsa_source(a, p, v, R);
  }
}

// Per point: the two energy densities (block sums into partials[2 block +
// term]) and, with grad, the adjoints lA (of gSigmaA's numerator), lD (of
// shell_2R n), lE (of the Gaussian convolution) and the explicit derivative.
__global__ void k_saft_point(SaftParams sp, double R, double kT, const double *__restrict__ n,
                             const double *__restrict__ A, const double *__restrict__ D2,
                             const double *__restrict__ Eg, int NR, int grad,
                             double *__restrict__ lA, double *__restrict__ lD,
                             double *__restrict__ lE, double *__restrict__ expl,
                             double *__restrict__ partials) {
  __shared__ double red[2][kThreads / 32];
  const double v43 = 4 * kPi * R * R * R / 3, area2 = 16 * kPi * R * R;
  const double Kf = sp.kappa_a * (exp(sp.eps_a / kT) - 1), lam = sp.lambda_d, eps = sp.eps_d;
  double acc[2] = {0, 0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NR; i += gridDim.x * blockDim.x) {
    const double ni = n[i], eta = v43 * Eg[i];
    double a1[5];
    a1_terms(eta, lam, eps, a1);
    const double om = 1 - eta, q = 1 + 2 * eta;
    const double KHS = om * om * om * om / (q * q);
    const double a2 = 0.5 * eps * KHS * eta * a1[1];
    const double gsig = A[i] / D2[i], nA = D2[i] / area2;
    const double gSW = gsig + (a1[1] - lam / (3 * eta) * a1[2]) / (4 * kT);
    const double Dl = gSW * Kf, y = nA * Dl;
    const double X = (sqrt(1 + 8 * y) - 1) / (4 * y);
    const double lx = log(X);
    acc[0] += 4 * kT * ni * (lx - X / 2 + 0.5);
    acc[1] += ni * a1[0] + ni * a2 / kT;
    if (grad) {
      const double KHS1 = -4 * om * om * om * (2 + eta) / (q * q * q);
      // X solves 2 y X^2 + X - 1 = 0: dX/dy = -2 X^2 / (1 + 4 y X)
      const double ly = 4 * kT * ni * (1 / X - 0.5) * (-2 * X * X / (1 + 4 * y * X));
      const double lnA = ly * Dl, lgSW = ly * nA * Kf;
      lA[i] = lgSW / D2[i];
      lD[i] = -lgSW * A[i] / (D2[i] * D2[i]) + lnA / area2;
      double leta = lgSW / (4 * kT) * (a1[3] - lam * (a1[4] / (3 * eta) - a1[2] / (3 * eta * eta)));
      leta += ni * a1[1] + ni / kT * 0.5 * eps * (KHS1 * eta * a1[1] + KHS * a1[1] + KHS * eta * a1[3]);
      lE[i] = v43 * leta;
      expl[i] = 4 * kT * (lx - X / 2 + 0.5) + a1[0] + a2 / kT;
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int k = 0; k < 2; k++) {
    double x = acc[k];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red[k][warp] = x;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double x = 0;
    for (int k = 0; k < kThreads / 32; k++) x += red[threadIdx.x][k];
    partials[2 * blockIdx.x + threadIdx.x] = x;
  }
}

// Fixed-order sums of the block partials: a block per term.
__global__ void __launch_bounds__(kThreads)
    k_saft_sum(const double *__restrict__ partials, int nblk, double dV,
               double *__restrict__ out) {
  __shared__ double red[32];
  double x[1] = {0};
  for (int b = threadIdx.x; b < nblk; b += kThreads) x[0] += partials[2 * b + blockIdx.x];
  block_reduce<1>(x, red);
  if (threadIdx.x == 0) out[blockIdx.x] = x[0] * dV;
}

// lw[b] = sum_a t_a d(source a)/d(w_b) (t_a = t + a NR): the adjoint of
// gSigmaA's numerator through its source fields into the five weighted
// densities, the partials and their derivatives computed once per point.
__global__ void k_saft_jacs(double R, const double *__restrict__ w,
                            const double *__restrict__ t, int NR, double *__restrict__ lw) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NR; i += gridDim.x * blockDim.x) {
    const double v[3] = {w[2 * (size_t)NR + i], w[3 * (size_t)NR + i], w[4 * (size_t)NR + i]};
    double D[6][3];
    const cm::Partials p = cm::partials(kHsWhiteBear, R, w[i], w[(size_t)NR + i],
                                        v[0] * v[0] + v[1] * v[1] + v[2] * v[2], D);
    double acc[5] = {0, 0, 0, 0, 0};
    for (int a = 0; a < 8; a++) {
      double J[5];
      cm::gsa_jacobian(a, p, D, v, R, J);
      const double ti = t[(size_t)a * NR + i];
      for (int b = 0; b < 5; b++) acc[b] += ti * J[b];
    }
    for (int b = 0; b < 5; b++) lw[(size_t)b * NR + i] = acc[b];
  }
}

__global__ void k_saft_grad(double dV, const double *__restrict__ expl,
                            const double *__restrict__ t, int NR, double *__restrict__ grad) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NR; i += gridDim.x * blockDim.x)
    grad[i] = dV * (expl[i] + t[i]);
}

// ---------------------------------------------------------------------------
// The FP64 form's pointwise passes on fields that stay double-floats between
// the sets of convolutions: gSigmaA's sources and their Jacobian in
// double-float arithmetic (dfloat.cuh; 96^3: 191 -> 26 us and 341 -> 41 us),
// association and dispersion in FP64.

// White Bear's coefficients at a point: u = 1/(1-n3), l = ln(1-n3), f3 and its
// derivatives with their constant 1/(36 pi).
struct DfWb {
  dfl u, u2, l, f3, df3;
};
__device__ __forceinline__ DfWb df_wb(dfl n3, dfl om, dfl *d2f3) {
  const tfl k36(1.0 / (36 * kPi));
  DfWb r;
  r.u = df_rcp(om);
  r.u2 = r.u * r.u;
  r.l = df_log1m(n3, om);
  dfl S, dS;
  df_S(n3, om, r.l, S, dS);
  const dfl Su = S * r.u;
  r.f3 = k36 * (Su * r.u);
  r.df3 = k36 * ((dS + df_ldexp(Su, 2.0f)) * r.u2);
  if (d2f3)
    *d2f3 = k36 * ((df_d2S(n3, om, r.l) + df_ldexp(dS * r.u, 4.0f) + df_scale(Su * r.u, 6.0f)) *
                   r.u2);
  return r;
}

// FP64 formulas for points outside the double-float range.
__device__ __noinline__ void saft_sources_fp64(double R, const dfl *w, dfl *src) {
  const double v[3] = {to_double(w[2]), to_double(w[3]), to_double(w[4])};
  const cm::Partials p = cm::partials(kHsWhiteBear, R, to_double(w[0]), to_double(w[1]),
                                      v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
  for (int a = 0; a < 8; a++) src[a] = df_from(cm::gsa_source(a, p, v, R));
}
__device__ __noinline__ void saft_jacs_fp64(double R, const dfl *w, const dfl *t, dfl *lw) {
  const double v[3] = {to_double(w[2]), to_double(w[3]), to_double(w[4])};
  double D[6][3], acc[5] = {0, 0, 0, 0, 0};
  const cm::Partials p = cm::partials(kHsWhiteBear, R, to_double(w[0]), to_double(w[1]),
                                      v[0] * v[0] + v[1] * v[1] + v[2] * v[2], D);
  for (int a = 0; a < 8; a++) {
    double J[5];
    cm::gsa_jacobian(a, p, D, v, R, J);
    for (int b = 0; b < 5; b++) acc[b] += to_double(t[a]) * J[b];
  }
  for (int b = 0; b < 5; b++) lw[b] = df_from(acc[b]);
}

// Constants of the White Bear sources: c1 = 1/(4 pi R), c0 = c1/R, 2 c0/R.
struct SaftWbConst {
  tfl c1, c0, c02R;
};

// gSigmaA's eight sources with d0 = -l, d1 = n2 u, d1v = -u and so on put in
// (the terms c0 n2 u of d3 and of d1 cancel):
//   s0 = c1 q u^2 + t3 f3' + (2 c0/R) l       s1 = 2 c1 n2 u + 3 q f3 - c0 l
//   s_v = -c0 u v                             s_v' = -(2 c1 u + 6 n2 f3) v
__global__ void __launch_bounds__(kThreads)
    k_saft_sources_df(double R, SaftWbConst k, const double *__restrict__ n,
                      const dfl *__restrict__ w, int NR, dfl *__restrict__ src) {
#pragma unroll 1
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NR; i += gridDim.x * blockDim.x) {
    dfl x[5];
#pragma unroll
    for (int a = 0; a < 5; a++) x[a] = w[(size_t)a * NR + i];
    const dfl n2 = x[1], v2 = x[2] * x[2] + x[3] * x[3] + x[4] * x[4], om = df_one_minus(x[0]);
    if (!df_point_ok(om, n2, v2, n[i] != 0)) {
      dfl xl[5] = {x[0], x[1], x[2], x[3], x[4]}, o[8];
      saft_sources_fp64(R, xl, o);
      for (int a = 0; a < 8; a++) src[(size_t)a * NR + i] = o[a];
      continue;
    }
    const DfWb b = df_wb(x[0], om, nullptr);
    const dfl n22 = n2 * n2, q = n22 - v2, t3 = n2 * (n22 - df_scale(v2, 3.0f));
    src[i] = k.c1 * (q * b.u2) + t3 * b.df3 + k.c02R * b.l;
    src[(size_t)NR + i] =
        df_ldexp(k.c1 * (n2 * b.u), 2.0f) + df_scale(q * b.f3, 3.0f) - k.c0 * b.l;
    const dfl m0 = -(k.c0 * b.u);
    const dfl m1 = -(df_ldexp(k.c1 * b.u, 2.0f) + df_scale(n2 * b.f3, 6.0f));
#pragma unroll
    for (int e = 0; e < 3; e++) {
      src[(size_t)(2 + e) * NR + i] = m0 * x[2 + e];
      src[(size_t)(5 + e) * NR + i] = m1 * x[2 + e];
    }
  }
}

// w becomes lw[b] = sum_a t_a d(source a)/d(w_b) (the derivatives of the
// sources above, t_v . v and t_v' . v formed once).
__global__ void __launch_bounds__(kThreads)
    k_saft_jacs_df(double R, SaftWbConst k, const double *__restrict__ n, dfl *__restrict__ w,
                   const dfl *__restrict__ t, int NR) {
#pragma unroll 1
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NR; i += gridDim.x * blockDim.x) {
    dfl x[5], s[8];
#pragma unroll
    for (int a = 0; a < 5; a++) x[a] = w[(size_t)a * NR + i];
#pragma unroll
    for (int a = 0; a < 8; a++) s[a] = t[(size_t)a * NR + i];
    const dfl n2 = x[1], v2 = x[2] * x[2] + x[3] * x[3] + x[4] * x[4], om = df_one_minus(x[0]);
    if (!df_point_ok(om, n2, v2, n[i] != 0)) {
      dfl xl[5] = {x[0], x[1], x[2], x[3], x[4]}, sl[8], o[5];
      for (int a = 0; a < 8; a++) sl[a] = s[a];
      saft_jacs_fp64(R, xl, sl, o);
      for (int a = 0; a < 5; a++) w[(size_t)a * NR + i] = o[a];
      continue;
    }
    dfl d2f3;
    const DfWb b = df_wb(x[0], om, &d2f3);
    const dfl n22 = n2 * n2, q = n22 - v2, t3 = n2 * (n22 - df_scale(v2, 3.0f));
    const dfl V = s[2] * x[2] + s[3] * x[3] + s[4] * x[4];
    const dfl P = s[5] * x[2] + s[6] * x[3] + s[7] * x[4];
    const dfl qf3 = df_scale(q * b.df3, 3.0f), c1n2u2 = df_ldexp(k.c1 * (n2 * b.u2), 2.0f);
    const dfl m1 = df_ldexp(k.c1 * b.u, 2.0f) + df_scale(n2 * b.f3, 6.0f);
    const dfl m1d = df_ldexp(k.c1 * b.u2, 2.0f) + df_scale(n2 * b.df3, 6.0f);
    w[i] = s[0] * (df_ldexp(k.c1 * (q * (b.u2 * b.u)), 2.0f) + t3 * d2f3 - k.c02R * b.u) +
           s[1] * (c1n2u2 + qf3 + k.c0 * b.u) - (k.c0 * b.u2) * V - m1d * P;
    w[(size_t)NR + i] = s[0] * (c1n2u2 + qf3) + s[1] * m1 - df_scale(b.f3 * P, 6.0f);
    const dfl vv = df_ldexp(
        s[0] * (k.c1 * b.u2 + df_scale(n2 * b.df3, 3.0f)) + df_scale(s[1] * b.f3, 3.0f), -2.0f);
    const dfl c0u = k.c0 * b.u;
#pragma unroll
    for (int e = 0; e < 3; e++)
      w[(size_t)(2 + e) * NR + i] = vv * x[2 + e] - c0u * s[2 + e] - m1 * s[5 + e];
  }
}

// Constants of the association and dispersion pass (host-made).
struct SaftPointConst {
  double c[3], l[3];       // effective packing fraction: coefficients, their lambda derivatives
  double v43;              // 4 pi R^3 / 3
  double preL3, pre3l2;    // -4 eps (lambda^3 - 1), -4 eps 3 lambda^2
  double lam3;             // lambda / 3
  double i4kT, heps, ikT;  // 1/(4 kT), eps/2, 1/kT
  double nAKf;             // kappa (e^(eps_a/kT) - 1) / (16 pi R^2)
  double kT4;              // 4 kT
};
SaftPointConst saft_point_const(const SaftParams &sp, double R, double kT) {
  const double l = sp.lambda_d, eps = sp.eps_d;
  SaftPointConst k;
  k.c[0] = 2.25855 - 1.50349 * l + 0.249434 * l * l;
  k.c[1] = -0.669270 + 1.40049 * l - 0.827739 * l * l;
  k.c[2] = 10.1576 - 15.0427 * l + 5.30827 * l * l;
  k.l[0] = -1.50349 + 2 * 0.249434 * l;
  k.l[1] = 1.40049 - 2 * 0.827739 * l;
  k.l[2] = -15.0427 + 2 * 5.30827 * l;
  k.v43 = 4 * kPi * R * R * R / 3;
  k.preL3 = -4 * eps * (l * l * l - 1);
  k.pre3l2 = -4 * eps * 3 * l * l;
  k.lam3 = l / 3;
  k.i4kT = 1 / (4 * kT);
  k.heps = eps / 2;
  k.ikT = 1 / kT;
  k.nAKf = sp.kappa_a * (exp(sp.eps_a / kT) - 1) / (16 * kPi * R * R);
  k.kT4 = 4 * kT;
  return k;
}

// k_saft_point on double-float fields, FP64 throughout (its explicit
// derivative enters the gradient point by point, where double-float rounding
// would show): the energies and, with grad, the adjoints in place (A becomes
// lA, D2 lD, Eg lE).  X = 2 / (1 + r), r = sqrt(1 + 8 y), is X's defining
// quadratic without its cancellation at small y; then 1/X - 1/2 = r/2, 1 + 4
// y X = r and the derivative of 4 kT (ln X - X/2 + 1/2) in y is -4 kT X^2.  With
// b = (1/eta) d a1/d lambda the dispersion part of gSW is (d a1/d eta - lambda
// b/3) / (4 kT), free of 1/eta, and it is what D2's adjoint keeps after
// gSigmaA's own.  About 100 FP64-pipe operations a point (rcp_fast, sqrt_fast,
// log_tab) against 320; 96^3: 570 -> 217 us
__global__ void __launch_bounds__(kThreads)
    k_saft_point_df(SaftPointConst k, const double *__restrict__ n, dfl *__restrict__ A,
                    dfl *__restrict__ D2, dfl *__restrict__ Eg, int NR, int grad,
                    double *__restrict__ expl, double *__restrict__ partials) {
  __shared__ double red[32 * 2];
  double acc[2] = {0, 0};
#pragma unroll 1
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NR; i += gridDim.x * blockDim.x) {
    const double ni = n[i], d2 = to_double(D2[i]), eta = k.v43 * to_double(Eg[i]);
    const double x = fma(fma(k.c[2], eta, k.c[1]), eta, k.c[0]) * eta;
    const double xe = fma(fma(3 * k.c[2], eta, 2 * k.c[1]), eta, k.c[0]);
    const double xee = fma(6 * k.c[2], eta, 2 * k.c[1]);
    const double xl = fma(fma(k.l[2], eta, k.l[1]), eta, k.l[0]) * eta;
    const double xel = fma(fma(3 * k.l[2], eta, 2 * k.l[1]), eta, k.l[0]);
    const double i1 = rcp_fast(1 - x), i2 = i1 * i1, i3 = i2 * i1, i4 = i2 * i2;
    const double g = fma(-0.5, x, 1.0) * i3, g1 = (2.5 - x) * i4, g2 = fma(-3.0, x, 9.0) * (i4 * i1);
    const double g1xe = g1 * xe, a1 = k.preL3 * (eta * g), a1e = k.preL3 * fma(eta, g1xe, g);
    const double a1ee = k.preL3 * fma(eta, fma(g2 * xe, xe, g1 * xee), 2 * g1xe);
    const double b = fma(k.pre3l2, g, k.preL3 * (g1 * xl));
    const double be = fma(k.pre3l2, g1xe, k.preL3 * fma(g2 * xe, xl, g1 * xel));
    const double om = 1 - eta, iq = rcp_fast(fma(2.0, eta, 1.0));
    const double om2 = om * om, iq2 = iq * iq, KHS = om2 * om2 * iq2;
    const double KHS1 = -4 * (om2 * om) * ((2 + eta) * (iq2 * iq));
    const double a2 = k.heps * (KHS * (eta * a1e));
    const double disp = k.i4kT * fma(-k.lam3, b, a1e);
    const double y = k.nAKf * d2 * fma(to_double(A[i]), rcp_fast(d2), disp);
    const double rt = sqrt_fast(fma(8.0, y, 1.0)), ir = rcp_fast(1 + rt), X = 2 * ir;
    // ln X - X/2 + 1/2, with (1 - X)/2 = (r - 1) / (2 (r + 1))
    const double fa = k.kT4 * fma(0.5 * (rt - 1), ir, log_tab(X));
    const double fd = fma(k.ikT, a2, a1);
    acc[0] = fma(ni, fa, acc[0]);
    acc[1] = fma(ni, fd, acc[1]);
    if (grad) {
      const double lA = -ni * (k.kT4 * k.nAKf) * (X * X);
      A[i] = df_from(lA);
      D2[i] = df_from(lA * disp);
      const double hk = fma(KHS1, eta * a1e, KHS * fma(eta, a1ee, a1e));
      Eg[i] = df_from(k.v43 * fma(lA * d2, k.i4kT * fma(-k.lam3, be, a1ee),
                                  ni * fma(k.ikT * k.heps, hk, a1e)));
      expl[i] = fa + fd;
    }
  }
  block_reduce<2>(acc, red);
  if (threadIdx.x < 2) partials[2 * blockIdx.x + threadIdx.x] = threadIdx.x == 0 ? acc[0] : acc[1];
}

int blocks_for(int n) {
  int b = (n + kThreads - 1) / kThreads;
  return b > 4096 ? 4096 : (b < 1 ? 1 : b);
}

}  // namespace

size_t saft_scratch_doubles(const Geom &g) {
  // one field at a time: w (5), A, D2, Eg, the eight source / adjoint fields t,
  // lA, lD, lE, expl, lw (5) real fields, two spectra; double-float: w, D2, Eg,
  // t, A, expl (the adjoints take their places) and eight spectra.  Block
  // partials and sums.
  const size_t one = 25 * (size_t)g.NR + 4 * (size_t)g.NC;
  const size_t df = 17 * (size_t)g.NR + 16 * (size_t)g.NC;
  return (one > df ? one : df) + 2 * kBlocks + 4;
}

int saft_terms(Engine *e, const FmtSpec &f, const SaftParams &sp, const double *n,
               double *scratch, double *grad, double terms2[2], std::string *err) {
  const Geom &g = e->geom();
  cudaStream_t s = e->stream();
  const int NR = g.NR, NC = g.NC, rb = blocks_for(NR), cb = blocks_for(NC);
  double *partials = scratch, *sums = partials + 2 * kBlocks, *fields = sums + 2;
  const double R = f.R, gs = 2 * sp.length_scaling * sp.lambda_d * R;
  auto fail = [&](const char *what) {
    if (err) *err = std::string("water SAFT: ") + what;
    return -1;
  };
  auto finish = [&]() {
    cudaError_t ce = cudaMemcpyAsync(terms2, sums, 2 * sizeof(double), cudaMemcpyDeviceToHost, s);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
    if (ce == cudaSuccess) ce = cudaGetLastError();
    if (ce == cudaSuccess) return 0;
    if (err) *err = std::string("water SAFT: ") + cudaGetErrorString(ce);
    return -1;
  };
  if (f.precision != kPrecisionMixed && e->df_on()) {
    // four sets of convolutions around three pointwise passes
    dfc *spec = reinterpret_cast<dfc *>(fields);
    dfl *F = reinterpret_cast<dfl *>(spec + 8 * (size_t)NC);  // w, D2 / lD, Eg / lE
    dfl *t = F + 7 * (size_t)NR, *A = t + 8 * (size_t)NR;
    dfl *D2 = F + 5 * (size_t)NR, *Eg = D2 + NR;
    double *expl = reinterpret_cast<double *>(A + NR);
    const dfl *step = e->radial(kRadStep, R), *shell = e->radial(kRadShell, R),
              *vec = e->radial(kRadVShell, R), *sp1 = e->radial(kRadShellPrime, R),
              *vp = e->radial(kRadVShellPrime, R), *sh2 = e->radial(kRadShell2R, R),
              *gau = e->radial(kRadGauss, gs);
    if (!step || !shell || !vec || !sp1 || !vp || !sh2 || !gau) return fail("weight tables");
    FieldWeights from_n, gsa;  // n's convolutions; gSigmaA's eight
    from_n.add(kWtScalar, step, nullptr, 4 * kPi / 3 * R * R * R * g.scale);
    from_n.add(kWtScalar, shell, nullptr, 4 * kPi * R * R * g.scale);
    for (int c = 0; c < 3; c++) from_n.add(kWtVector + c, vec);
    from_n.add(kWtScalar, sh2, nullptr, 16 * kPi * R * R * g.scale);
    from_n.add(kWtScalar, gau, nullptr, g.scale);
    gsa.add(kWtScalar, shell, nullptr, 4 * kPi * R * R * g.scale);
    gsa.add(kWtScalar, sp1, nullptr, 8 * kPi * R * g.scale);
    for (int c = 0; c < 3; c++) gsa.add(kWtVector + c, vec);
    for (int c = 0; c < 3; c++) gsa.add(kWtVector + c, vp);
    const double c1 = 1 / (4 * kPi * R);
    const SaftWbConst kw = {tfl(c1), tfl(c1 / R), tfl(2 * c1 / (R * R))};
    if (e->spectrum(n) || e->fan_out(from_n, 1, spec, F)) return fail(e->last_error());
    k_saft_sources_df<<<rb, kThreads, 0, s>>>(R, kw, n, F, NR, t);
    if (e->fan_in(gsa, 1, t, spec, A)) return fail(e->last_error());
    k_saft_point_df<<<kBlocks, kThreads, 0, s>>>(saft_point_const(sp, R, f.kT), n, A, D2, Eg, NR,
                                                 grad != nullptr, expl, partials);
    k_saft_sum<<<2, kThreads, 0, s>>>(partials, kBlocks, g.dV, sums);
    if (grad) {
      if (e->spectrum(A) || e->fan_out(gsa, -1, spec, t)) return fail(e->last_error());
      k_saft_jacs_df<<<rb, kThreads, 0, s>>>(R, kw, n, F, t, NR);
      double *gr = reinterpret_cast<double *>(t);
      if (e->fan_in(from_n, -1, F, spec, gr)) return fail(e->last_error());
      k_saft_grad<<<rb, kThreads, 0, s>>>(g.dV, expl, gr, NR, grad);
    }
    return finish();
  }
  double *w = fields, *A = w + 5 * (size_t)NR, *D2 = A + NR, *Eg = D2 + NR, *t = Eg + NR;
  double *lA = t + 8 * (size_t)NR, *lD = lA + NR, *lE = lD + NR, *expl = lE + NR, *lw = expl + NR;
  double2 *spec = reinterpret_cast<double2 *>(lw + 5 * (size_t)NR + NR % 2), *acc = spec + NC;
  // the mixed form runs every transform in FP32 (pointwise work stays FP64)
  const Engine::Arith arith =
      f.precision == kPrecisionMixed ? Engine::kArithFP32 : Engine::kArithDF;
  FmtSpec fw = f;
  fw.hs = kHsWhiteBear;
  if (e->weighted(fw, n, w, arith)) return fail("weighted densities");
  k_saft_sources<<<rb, kThreads, 0, s>>>(R, w, NR, t);
  for (int a = 0; a < 8; a++) {
    if (e->fft(t + (size_t)a * NR, spec, arith)) return fail("fft");
    cm::k_weight_apply<<<cb, kThreads, 0, s>>>(a, g, R, 0.0, spec, acc, 0, a == 0);
  }
  if (e->ifft(acc, A, arith)) return fail("ifft");
  if (e->fft(n, spec, arith)) return fail("fft");
  cm::k_weight_apply<<<cb, kThreads, 0, s>>>(8, g, R, 0.0, spec, acc, 0, 1);
  if (e->ifft(acc, D2, arith)) return fail("ifft");
  cm::k_weight_apply<<<cb, kThreads, 0, s>>>(10, g, R, gs, spec, acc, 0, 1);
  if (e->ifft(acc, Eg, arith)) return fail("ifft");
  k_saft_point<<<kBlocks, kThreads, 0, s>>>(sp, R, f.kT, n, A, D2, Eg, NR, grad != nullptr, lA, lD,
                                            lE, expl, partials);
  k_saft_sum<<<2, kThreads, 0, s>>>(partials, kBlocks, g.dV, sums);
  if (grad) {
    // adjoint of gSigmaA's eight convolutions, through the source Jacobian
    double2 *specA = acc;  // spectrum of lA, kept while the eight adjoints are formed
    if (e->fft(lA, specA, arith)) return fail("fft");
    for (int a = 0; a < 8; a++) {
      cm::k_weight_apply<<<cb, kThreads, 0, s>>>(a, g, R, 0.0, specA, spec, 1, 1);
      if (e->ifft(spec, t + (size_t)a * NR, arith)) return fail("ifft");
    }
    k_saft_jacs<<<rb, kThreads, 0, s>>>(R, w, t, NR, lw);
    // weighted-density adjoints (step, shell, vector shells), shell_2R, Gaussian
    for (int b = 0; b < 5; b++) {
      if (e->fft(lw + (size_t)b * NR, spec, arith)) return fail("fft");
      cm::k_weight_apply<<<cb, kThreads, 0, s>>>(11 + b, g, R, 0.0, spec, acc, 1, b == 0);
    }
    if (e->fft(lD, spec, arith)) return fail("fft");
    cm::k_weight_apply<<<cb, kThreads, 0, s>>>(8, g, R, 0.0, spec, acc, 1, 0);
    if (e->fft(lE, spec, arith)) return fail("fft");
    cm::k_weight_apply<<<cb, kThreads, 0, s>>>(10, g, R, gs, spec, acc, 1, 0);
    if (e->ifft(acc, t, arith)) return fail("ifft");
    k_saft_grad<<<rb, kThreads, 0, s>>>(g.dV, expl, t, NR, grad);
  }
  return finish();
}

}  // namespace deft
