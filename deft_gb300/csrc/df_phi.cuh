// Phi and its partials at one point for the FP64 form, whose weighted
// densities arrive as the transforms' double-floats and whose partials leave
// as such.  In FP64 the point costs about 140 operations of GB300's narrow
// FP64 pipe (conversions in and out, a logarithm, two reciprocals, 60
// multiply-adds): 741 us of the 1408 us evaluation at 128^3.  In
// double-float arithmetic (dfloat.cuh, logtab.cuh) it costs about 600 FP32
// instructions, one FP64 operation's time for 64 of them.  The Phi kernel
// (with its ten z transforms): 333 -> 193 us at 77^3, 5928 -> 3222 at 256^3,
// mark II 1000 -> 351 at 128^3.  Rounding: each
// partial carries about 2^-46 of its largest term, the size of the rounding
// the transforms on either side leave in it, and unlike theirs white over the
// points, so that the convolution that follows averages it out; constants
// that are not exact are three words long (tfl), since their rounding would
// not be white.  Gradient error against 64-bit arithmetic (relative 2-norm,
// rms of 40 inputs), with Phi in FP64 and the transforms of that time / now: White
// Bear 77^3 fcc 2.06e-14 / 1.63e-14, 128^3 2.42e-14 / 2.24e-14, mark II 128^3
// 2.46e-14 / 1.75e-14.
//
// Points the double-float range or the small-density branch of the terms does
// not cover (1 - n3 outside (2^-20, 2^20), very large weighted densities, a
// dilute fluid whose cubic terms would underflow) take the FP64 formulas of
// wb_phi.cuh, out of line.
#pragma once

#include "logtab.cuh"
#include "wb_phi.cuh"

namespace deft {

// Constants of a launch (host-made).
struct DfPhiConst {
  tfl a1, a2x2;        // c / (4 pi R^2), 2 c / (4 pi R)
  tfl a2;              // c / (4 pi R)
  tfl k3;              // c times the third term's constant (1/(36 pi) or 1/(24 pi))
  double s0, s1, s2;   // factors of the sums of f3' t3, n2 l and q f2
};
inline DfPhiConst df_phi_const(const WbRadius &wr, double c) {
  const double k = wr.kind == kHsWhiteBear ? 1.0 / (36 * 3.14159265358979323846)
                                           : 1.0 / (24 * 3.14159265358979323846);
  DfPhiConst d;
  d.a1 = tfl(c * wr.inv_4piR2);
  d.a2 = tfl(c * wr.inv_4piR);
  d.a2x2 = tfl(2 * c * wr.inv_4piR);
  d.k3 = tfl(c * k);
  d.s0 = k;
  d.s1 = -wr.inv_4piR2;
  d.s2 = wr.inv_4piR;
  return d;
}

// S and S' (wb_phi.cuh) for |e| < 1/32 by their series: five terms in
// double-float, five in FP32 (each below 2^-24 of the sum).
__device__ __forceinline__ void df_S_series(dfl e, dfl &S, dfl &dS) {
  auto c = [](int j) { return 2.0 / (double(j) * (j + 1) * (j + 2)); };
  const float ef = e.hi;
  float s = 0.f, d = 0.f;
#pragma unroll
  for (int j = 10; j > 5; j--) {
    s = fmaf(s, ef, (float)c(j));
    d = fmaf(d, ef, (float)(j * c(j)));
  }
  dfl s2 = df_scale(e, s), d2 = df_scale(e, d);
#pragma unroll
  for (int j = 5; j > 0; j--) {
    s2 = (dfl(c(j)) + s2) * e;
    d2 = dfl(j * c(j)) + d2;
    if (j > 1) d2 = d2 * e;
  }
  S = dfl(1.5f, 0.f) - s2;
  dS = -d2;
}

// P2, P3 of mark II and their first derivatives (wb_phi.cuh); l = ln(1 - e).
// With A = sum_k>=2 e^(k-2)/(k (k+1)): P2 = 1 + 2/3 e^2 A, P3' = 4/3 A - 2/3.
__device__ __forceinline__ void df_m2(dfl e, dfl om, dfl l, dfl &P2, dfl &dP2, dfl &P3,
                                      dfl &dP3) {
  if (fabsf(e.hi) < 0.0625f) {
    const float ef = e.hi;
    float a = 0.f, d = 0.f, b = 0.f;  // tails in FP32: the terms e^5 and beyond
#pragma unroll
    for (int j = 11; j >= 5; j--) {
      a = fmaf(a, ef, (float)(1.0 / ((j + 2) * (j + 3))));
      d = fmaf(d, ef, (float)(1.0 / (j + 3)));
      b = fmaf(b, ef, (float)(1.0 / (double(j + 2) * (j + 3) * (j + 4))));
    }
    dfl A(a, 0.f), D(d, 0.f), B(b, 0.f);
#pragma unroll
    for (int j = 4; j >= 0; j--) {
      A = dfl(1.0 / ((j + 2) * (j + 3))) + A * e;
      D = dfl(1.0 / (j + 3)) + D * e;
      B = dfl(1.0 / (double(j + 2) * (j + 3) * (j + 4))) + B * e;
    }
    const dfl e2 = e * e, k23 = dfl(2.0 / 3), k43 = dfl(4.0 / 3);
    P2 = dfl(1) + k23 * (e2 * A);
    dP2 = k23 * (e * D);
    P3 = dfl(1) + k43 * (e2 * B) - dfl(4.0 / 9) * e;
    dP3 = k43 * A - k23;
  } else {
    // P2 = 1 + 2/3 (1 - e/2 + B), B = (1-e) ln(1-e) / e: the constants that
    // are not exact multiply what is left after the cancellation
    const dfl ie = df_rcp(e), B = om * l * ie;
    const tfl k23(2.0 / 3), k19(1.0 / 9);
    P2 = dfl(1) + k23 * ((dfl(1) - df_ldexp(e, 0.5f)) + B);
    dP2 = -(k23 * (((e + l) * ie) * ie + dfl(0.5f, 0.f)));
    // Q = N/e, N = 6 - 9e + 6e^2 + 6C, C = (1-e) B; P3 = 1 - Q/9
    const dfl C = om * B;
    const dfl Q = (dfl(6) - df_scale(e, 9.0f) + df_scale(e * e + C, 6.0f)) * ie;
    const dfl dC = -(df_ldexp(om * l, 2.0f) + om + C) * ie;
    const dfl dN = df_scale(e, 12.0f) - dfl(9) + df_scale(dC, 6.0f);
    P3 = dfl(1) - k19 * Q;
    dP3 = k19 * ((Q - dN) * ie);
  }
}

// Whether the double-float formulas cover a point: 1 - n3 well inside (0, inf)
// and the powers of n2, v inside FP32's range.
__device__ __forceinline__ bool df_point_ok(dfl om, dfl n2, dfl v2, bool fluid) {
  const float a = fabsf(n2.hi);
  return om.hi > 0x1p-20f && om.hi < 0x1p20f && a < 1e9f && v2.hi < 1e18f &&
         (a > 1e-9f || !fluid);
}
__device__ __forceinline__ dfl df_one_minus(dfl x) {
  const dfl t = df_two_sum(1.0f, -x.hi);
  return df_fast_two_sum(t.hi, t.lo - x.lo);
}

// S'' (wb_phi.cuh) with S and S' as df_S gives them.
__device__ __forceinline__ dfl df_d2S(dfl n3, dfl om, dfl l) {
  if (fabsf(n3.hi) < 0.03125f) {
    auto c = [](int j) { return 2.0 * (j - 1) / (double(j + 1) * (j + 2)); };  // j (j-1) c_j
    const float ef = n3.hi;
    float d = 0.f;
#pragma unroll
    for (int j = 11; j > 6; j--) d = fmaf(d, ef, (float)c(j));
    dfl s = df_scale(n3, d);
#pragma unroll
    for (int j = 6; j >= 2; j--) {
      s = dfl(c(j)) + s;
      if (j > 2) s = s * n3;
    }
    return -s;
  }
  const dfl ol = om * l, g = n3 + om * ol, dg = n3 - df_ldexp(ol, 2.0f);
  const dfl ie = df_rcp(n3), ie2 = ie * ie, d2g = dfl(3) + df_ldexp(l, 2.0f);
  return (d2g - df_ldexp(dg * ie, 4.0f) + df_scale(g * ie2, 6.0f)) * ie2;
}

// The third term's f3 without its constant (White Bear: S u^2, Rosenfeld: u^2)
// and its derivative.
__device__ __forceinline__ void df_S(dfl n3, dfl om, dfl l, dfl &S, dfl &dS) {
  if (fabsf(n3.hi) < 0.03125f) {
    df_S_series(n3, S, dS);
  } else {
    const dfl ol = om * l, g = n3 + om * ol, dg = n3 - df_ldexp(ol, 2.0f);
    const dfl ie = df_rcp(n3), gi = g * ie, ie2 = ie * ie;
    S = gi * ie;
    dS = (dg - df_ldexp(gi, 2.0f)) * ie2;
  }
}

// The FP64 formulas: p[3] = the sums' terms, d = c times the partials.
static __device__ __noinline__ void df_phi_fp64(const WbRadius &r, const DfPhiConst &k, double c,
                                         const dfl *w, double *p, dfl *d) {
  double phi[3], g[5];
  wb_phi<double>(r, to_double(w[0]), to_double(w[1]), to_double(w[2]), to_double(w[3]),
                 to_double(w[4]), phi, g);
  p[0] = phi[0] / k.s0;
  p[1] = phi[1] / k.s1;
  p[2] = phi[2] / k.s2;
  for (int i = 0; i < 5; i++) d[i] = df_from(c * g[i]);
}

// w = (n3, n2, vx, vy, vz): adds f3 t3, n2 l and q f2 (without their
// constants) to acc and gives d = c dphi/dw.  fluid: the point's density is
// not zero, so that a vanishing n2 is a dilute fluid and not the inside of a
// wall.
__device__ __forceinline__ void df_phi_point(const WbRadius &r, const DfPhiConst &k, double c,
                                             const dfl (&w)[5], bool fluid, double (&acc)[6],
                                             dfl (&d)[5]) {
  const dfl n3 = w[0], n2 = w[1];
  const dfl v2 = w[2] * w[2] + w[3] * w[3] + w[4] * w[4];
  const dfl om = df_one_minus(n3);
  if (!df_point_ok(om, n2, v2, fluid)) {
    dfl wl[5] = {w[0], w[1], w[2], w[3], w[4]}, dl[5];
    double p[3];
    df_phi_fp64(r, k, c, wl, p, dl);
#pragma unroll
    for (int i = 0; i < 3; i++) acc[i] += p[i];
#pragma unroll
    for (int i = 0; i < 5; i++) d[i] = dl[i];
    return;
  }
  const dfl u = df_rcp(om), u2 = u * u, l = df_log1m(n3, om);
  const dfl n22 = n2 * n2, q = n22 - v2, t3 = n2 * (n22 - df_scale(v2, 3.0f));
  dfl f2 = u, df2 = u2, f3, df3;
  if (r.kind == kHsRosenfeld) {
    f3 = u2;
    df3 = df_ldexp(u2 * u, 2.0f);
  } else if (r.kind == kHsWhiteBear) {
    dfl S, dS;
    df_S(n3, om, l, S, dS);
    f3 = S * u2;
    df3 = (dS + df_ldexp(S * u, 2.0f)) * u2;
  } else {
    dfl P2, dP2, P3, dP3;
    df_m2(n3, om, l, P2, dP2, P3, dP3);
    f2 = P2 * u;
    df2 = (dP2 + f2) * u;
    f3 = P3 * u2;
    df3 = (dP3 + df_ldexp(P3 * u, 2.0f)) * u2;
  }
  const dfl p0 = f3 * t3, p1 = n2 * l, p2 = q * f2;
  acc[0] += f2d(p0.hi);
  acc[1] += f2d(p1.hi);
  acc[2] += f2d(p2.hi);
  acc[0] += f2d(p0.lo);
  acc[1] += f2d(p1.lo);
  acc[2] += f2d(p2.lo);
  const dfl f3k = k.k3 * f3;
  d[0] = k.a1 * (n2 * u) + (k.a2 * q) * df2 + (k.k3 * df3) * t3;
  d[1] = k.a2x2 * (n2 * f2) - k.a1 * l + df_scale(f3k * q, 3.0f);
  const dfl cv = -(k.a2x2 * f2 + df_scale(f3k * n2, 6.0f));
#pragma unroll
  for (int i = 0; i < 3; i++) d[2 + i] = cv * w[2 + i];
}

}  // namespace deft
