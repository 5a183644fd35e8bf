// Double-float arithmetic for the FP64 form's transforms on sm_103a.
//
// GB300 issues FP32 at about 64 times its FP64 rate, so the FP64 form's FFT
// butterflies and twiddle products run on pairs of FP32 numbers: a value is
// hi + lo with |lo| <= ulp(hi) / 2, about 48 significant bits (unit
// roundoff 2^-48 ~ 3.6e-15).  The building blocks are the error-free
// transformations of Knuth (TwoSum: a + b = s + e exactly, six FP32
// operations), Dekker's FastTwoSum (for |a| >= |b|, three operations) and
// the FMA form of Dekker's TwoProduct (a b = p + e exactly with
// e = fma(a, b, -p)); the sum and product of two double-floats follow the
// "sloppy" addition and the product of Dekker (1971) as analysed by Joldes,
// Muller and Popescu (ACM TOMS 44, 2017): relative error of the sum bounded
// by about 2^-46 of |a| + |b| (an FFT's error is judged against the norm of
// its input, so cancellation does not matter), of the product by about
// 2^-45.  Data enter and leave in FP64 (df_from, to_double); the FP64 form's
// Phi takes the weighted densities as they are (df_phi.cuh), its logarithm
// of the density, local terms and sums are FP64.
//
// Range: FP32's exponent (|x| below 3.4e38, lo underflows below about
// 1e-38 * 2^24), ample for densities, weighted densities and gradients.
#pragma once

#include <cuda_runtime.h>

namespace deft {

// FP32 -> FP64, exact.  The conversion instructions run on the FP64 pipe (two
// lanes a clock and SM, as its arithmetic): widening a normal number with
// integer operations leaves that pipe to the arithmetic that needs it.
__device__ __forceinline__ double f2d(float f) {
  const unsigned b = __float_as_uint(f), m = b & 0x7fffffffu;
  if (m - 0x00800000u < 0x7f000000u)
    return __hiloint2double((int)((b & 0x80000000u) | ((m >> 3) + 0x38000000u)), (int)(b << 29));
  return m == 0 ? __hiloint2double((int)b, 0) : (double)f;
}

struct dfl {
  float hi, lo;
  dfl() = default;
  __host__ __device__ constexpr dfl(float h, float l) : hi(h), lo(l) {}
  // exact for integers up to 2^24, as for any float
  __host__ __device__ constexpr dfl(int v) : hi((float)v), lo(0.f) {}
  // the nearest double-float to d (two roundings, error below 2^-48 |d|)
  __host__ __device__ constexpr dfl(double d)
      : hi((float)d), lo((float)(d - (double)(float)d)) {}
  __host__ __device__ explicit operator double() const {
#ifdef __CUDA_ARCH__
    return f2d(hi) + f2d(lo);
#else
    return (double)hi + (double)lo;
#endif
  }
};

// The nearest double-float to a double, by integer operations for
// 2^-74 <= |d| < 2^127 (and 0): hi is the mantissa rounded to 24 bits (half
// up, by a carry), lo the signed remainder of 29 bits times its power of two.
__device__ __forceinline__ dfl df_from(double d) {
  const unsigned lo = (unsigned)__double2loint(d), hi = (unsigned)__double2hiint(d);
  const unsigned e = hi & 0x7ff00000u, sign = hi & 0x80000000u;
  if (e - (949u << 20) <= (200u << 20)) {
    const unsigned rl = lo + 0x10000000u;
    const unsigned rh = (hi & 0x7fffffffu) + (rl < lo ? 1u : 0u);
    const float h = __uint_as_float((__funnelshift_r(rl, rh, 29) - (384u << 23)) | sign);
    const float unit = __uint_as_float((((e >> 20) - 948u) << 23) | sign);
    return dfl(h, (float)((int)(lo << 3) >> 3) * unit);
  }
  if (((hi & 0x7fffffffu) | lo) == 0) return dfl(__uint_as_float(sign), 0.f);
  const float h = (float)d;
  return dfl(h, (float)(d - (double)h));
}
// The nearest float to a double of magnitude 2^-74 .. 2^127 (others through
// the conversion instruction).
__device__ __forceinline__ float d2f_small(double d) {
  const unsigned lo = (unsigned)__double2loint(d), hi = (unsigned)__double2hiint(d);
  const unsigned e = hi & 0x7ff00000u, sign = hi & 0x80000000u;
  if (e - (949u << 20) <= (200u << 20)) {
    const unsigned rl = lo + 0x10000000u;
    const unsigned rh = (hi & 0x7fffffffu) + (rl < lo ? 1u : 0u);
    return __uint_as_float((__funnelshift_r(rl, rh, 29) - (384u << 23)) | sign);
  }
  if (((hi & 0x7fffffffu) | lo) == 0) return __uint_as_float(sign);
  return (float)d;
}
// A real of the transforms' type from FP64 data (or from FP32: widening or a
// copy), and the way back; none of the common cases runs on the FP64 pipe.
template <typename T> __device__ __forceinline__ T real_from(double d) { return T(d); }
template <> __device__ __forceinline__ dfl real_from<dfl>(double d) { return df_from(d); }
template <> __device__ __forceinline__ float real_from<float>(double d) { return d2f_small(d); }
template <typename T> __device__ __forceinline__ T real_from(dfl d) { return T(d); }
template <typename T> __device__ __forceinline__ T real_from(float f) { return T(f); }
template <> __device__ __forceinline__ double real_from<double>(float f) { return f2d(f); }

// Knuth's TwoSum: s + e == a + b exactly.
__device__ __forceinline__ dfl df_two_sum(float a, float b) {
  const float s = a + b;
  const float bb = s - a;
  return dfl(s, (a - (s - bb)) + (b - bb));
}
// Dekker's FastTwoSum (|a| >= |b| or a == 0): s + e == a + b exactly.
__device__ __forceinline__ dfl df_fast_two_sum(float a, float b) {
  const float s = a + b;
  return dfl(s, b - (s - a));
}
__device__ __forceinline__ dfl operator+(dfl a, dfl b) {
  const dfl s = df_two_sum(a.hi, b.hi);
  return df_fast_two_sum(s.hi, s.lo + (a.lo + b.lo));
}
__device__ __forceinline__ dfl operator-(dfl a) { return dfl(-a.hi, -a.lo); }
__device__ __forceinline__ dfl operator-(dfl a, dfl b) { return a + (-b); }
// Dekker's product with the FMA TwoProduct for hi * hi; the cross terms
// enter the error word.  The rounded product is taken with __fmul_rn so the
// compiler cannot contract it into the following addition.
__device__ __forceinline__ dfl operator*(dfl a, dfl b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, e));
  return df_fast_two_sum(p, e);
}
__device__ __forceinline__ dfl &operator+=(dfl &a, dfl b) { return a = a + b; }
__device__ __forceinline__ dfl &operator-=(dfl &a, dfl b) { return a = a - b; }
__device__ __forceinline__ dfl &operator*=(dfl &a, dfl b) { return a = a * b; }
__device__ __forceinline__ bool operator==(dfl a, dfl b) { return a.hi == b.hi && a.lo == b.lo; }
__device__ __forceinline__ bool operator<(dfl a, dfl b) {
  return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo);
}
// Quotient by one correction step (the long division of Dekker 1971):
// q1 = a.hi / b.hi in FP32, the remainder r = a - q1 b in double-float,
// q = q1 + r.hi / b.hi; relative error about 2^-44.
__device__ __forceinline__ dfl operator/(dfl a, dfl b) {
  const float rb = 1.0f / b.hi;
  const float q1 = a.hi * rb;
  const dfl r = a - dfl(q1, 0.f) * b;
  const float q2 = r.hi * rb;
  const dfl q = df_fast_two_sum(q1, q2);
  // a second correction for the last bits
  const dfl r2 = a - q * b;
  return q + dfl(r2.hi * rb, 0.f);
}
__host__ __device__ __forceinline__ double to_double(dfl a) { return double(a); }
// a b for a float b (exact up to the final rounding, about 2^-47).
__device__ __forceinline__ dfl df_scale(dfl a, float b) {
  const float p = __fmul_rn(a.hi, b);
  return df_fast_two_sum(p, fmaf(a.lo, b, fmaf(a.hi, b, -p)));
}
// A constant as three floats (72 bits), for products whose rounding should
// be the product's alone: a constant's own rounding to a double-float would
// be the same at every point, and a transform sums it up.
struct tfl {
  float a, b, c;
  tfl() = default;
  __host__ __device__ constexpr tfl(float x, float y, float z) : a(x), b(y), c(z) {}
  __host__ __device__ explicit constexpr tfl(double d)
      : a((float)d), b((float)(d - (double)(float)d)),
        c((float)((d - (double)(float)d) - (double)(float)(d - (double)(float)d))) {}
};
__device__ __forceinline__ dfl operator*(tfl k, dfl x) {
  const float p = __fmul_rn(x.hi, k.a);
  float e = fmaf(x.hi, k.a, -p);
  e = fmaf(x.lo, k.b, fmaf(x.hi, k.c, e));
  return df_fast_two_sum(p, fmaf(x.hi, k.b, fmaf(x.lo, k.a, e)));
}
// a times a power of two (exact).
__device__ __forceinline__ dfl df_ldexp(dfl a, float p) { return dfl(a.hi * p, a.lo * p); }
// 1 / b to about 2^-47 for normal b well inside FP32's range: y0 = 1/b.hi to
// FP32, t = 1 - b y0 (|t| <= 2^-22), 1/b = y0 (1 + t + t^2 + ..).
__device__ __forceinline__ dfl df_rcp(dfl b) {
  float y0;
  asm("rcp.approx.f32 %0, %1;" : "=f"(y0) : "f"(b.hi));
  float t = fmaf(-b.hi, y0, 1.0f);
  t = fmaf(-b.lo, y0, t);
  return df_fast_two_sum(y0, y0 * fmaf(t, t, t));
}

// Complex double-float: 16 bytes, the size of a double2, so the FP64 form's
// tiles and spectra keep their shapes.
struct __align__(16) dfc {
  dfl x, y;
};

}  // namespace deft
