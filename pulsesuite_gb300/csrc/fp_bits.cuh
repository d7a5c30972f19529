// FP64 <-> FP32 conversions on the integer pipe.
//
// On GB300 the FP64 pipe (which also executes the F2F conversions between double
// and float) runs at about 1/64 of the FP32 rate, so a per-element (float)x or
// (double)f in an O(Nk^2) kernel costs as much as an FP64 FMA.  These helpers do
// the same IEEE conversions with integer instructions.
#pragma once
#include <cstdint>

namespace sbe {

// round-to-nearest-even of x to FP32: results below the normal range become signed zero (see
// the scaled form below), overflow infinity, NaN stays NaN.  The common case is a funnel shift,
// one 64-bit add for the rounding and a select for zeros; what the branch takes is the last
// value below 2^-126 and everything from 2^127.
__device__ __forceinline__ float f64_to_f32(double x, int e);
__device__ __forceinline__ float f64_to_f32(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned sign = hi & 0x80000000u, a = hi & 0x7FFFFFFFu;
  if (a >= 0x47E00000u || a == 0x380FFFFFu) return f64_to_f32(x, 0);
  const unsigned t = __funnelshift_l(lo, a, 3);   // exponent and 23 bits, modulo 2^32
  const unsigned long long r =
      (((unsigned long long)(t + 0x40000000u) << 32) | (lo << 3)) + (0x7FFFFFFFu + (t & 1u));
  return __uint_as_float(sign | (a < 0x380FFFFFu ? 0u : (unsigned)(r >> 32)));
}

// round-to-nearest-even of x * 2^e to FP32 (e is added to the exponent, so the
// scaling is exact).  Results below the FP32 normal range (|x 2^e| < 2^-126)
// become signed zero; overflow gives infinity; NaN stays NaN.  The 52-bit
// mantissa is rounded to 23 bits with one 64-bit integer add (ties to even); a
// carry out of the mantissa runs into the exponent field.
__device__ __forceinline__ float f64_to_f32(double x, int e) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const unsigned sign = (unsigned)(u >> 32) & 0x80000000u;
  const unsigned long long a = u & 0x7FFFFFFFFFFFFFFFull;
  if (a >= 0x7FF0000000000000ull)   // infinity or NaN
    return __uint_as_float(sign | 0x7F800000u | (a != 0x7FF0000000000000ull ? 0x400000u : 0u));
  const unsigned long long r = (a + 0x0FFFFFFFull + ((a >> 29) & 1ull)) >> 29;
  const int fe = (int)(r >> 23) - (1023 - 127) + e;
  if (fe >= 255) return __uint_as_float(sign | 0x7F800000u);
  if (fe <= 0) return __uint_as_float(sign);
  return __uint_as_float(sign | ((unsigned)fe << 23) | ((unsigned)r & 0x7FFFFFu));
}

// x * 2^e for FP32 by two exact power-of-two multiplies (|e| <= 252, result in
// the normal range)
__device__ __forceinline__ float f32_ldexp(float x, int e) {
  const int e1 = e / 2, e2 = e - e1;
  return x * __int_as_float((127 + e1) << 23) * __int_as_float((127 + e2) << 23);
}

// exact widening of an FP32 value to FP64 (normal values and zeros without a branch)
__device__ __forceinline__ double f32_to_f64(float f) {
  const unsigned u = __float_as_uint(f);
  const unsigned sign = u & 0x80000000u, a = u & 0x7FFFFFFFu;
  if (a - 0x00800000u >= 0x7F000000u && a != 0) {
    unsigned m = u & 0x7FFFFFu;
    if (a >= 0x7F800000u)   // infinity or NaN
      return __hiloint2double((int)(sign | 0x7FF00000u | (m ? 0x80000u : 0u)), 0);
    // FP32 subnormal m 2^-149: normalise the leading bit to bit 23
    const int sh = __clz((int)m) - 8;
    m = (m << sh) & 0x7FFFFFu;
    const unsigned e64 = (unsigned)(1 - 127 + 1023 - sh);
    return __hiloint2double((int)(sign | (e64 << 20) | (m >> 3)), (int)(m << 29));
  }
  return __hiloint2double((int)(sign | (a ? (a >> 3) + 0x38000000u : 0u)), (int)(u << 29));
}

// f * 2^e exactly in FP64 (f finite; the result is assumed to stay normal)
__device__ __forceinline__ double f32_to_f64_scaled(float f, int e) {
  const double d = f32_to_f64(f);
  if (f == 0.f) return d;
  return __hiloint2double(__double2hiint(d) + (e << 20), __double2loint(d));
}

__device__ __forceinline__ float2 f64_to_f32(double2 v) {
  return make_float2(f64_to_f32(v.x), f64_to_f32(v.y));
}

__device__ __forceinline__ float2 f64_to_f32(double2 v, int e) {
  return make_float2(f64_to_f32(v.x, e), f64_to_f32(v.y, e));
}

__device__ __forceinline__ double2 f32_to_f64(float2 v) {
  return make_double2(f32_to_f64(v.x), f32_to_f64(v.y));
}

// 1 / x for normal x of magnitude 2^-1021 to 2^1021, within 0.6 ulp: the hyperpower iteration of
// third order, y (1 + e + e^2) with e = 1 - x y (M. Altman, "An optimum cubically convergent
// iterative method of inverting a linear bounded operator in Hilbert space", Pacific J. Math. 10,
// 1960), whose relative error is e^3.  It starts from PTX's approximate reciprocal, which takes and
// returns 20 mantissa bits: |e| stays below 2^-18.9, e is exact (73 bits of the product less the 20
// that cancel), e^3 < 2^-56.7 or 0.08 ulp.  Three FMAs on the two-wide FP64 pipe.  Zero, subnormal
// and infinite x give NaN.
__device__ __forceinline__ double rcp64(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// x / d from r, the correctly rounded 1 / d: q = x r is within an ulp of the quotient, its remainder
// x - q d is exact in one FMA, and q + (x - q d) r rounds to the quotient as the division does
// (P. W. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM
// J. Res. Dev. 34, 1990).  That holds while d and r are normal and the remainder is (|x| above
// 2^-968); smaller quotients may be off by an ulp, and -0 becomes 0.  Three instructions of the
// two-wide FP64 pipe instead of a dozen.
__device__ __forceinline__ double div_by(double x, double d, double r) {
  const double q = x * r;
  if ((__double2hiint(q) & 0x7FF00000) == 0x7FF00000) return q;   // infinite or NaN
  return fma(fma(-q, d, x), r, q);
}

// infinite or NaN, by the exponent
__device__ __forceinline__ bool not_finite(double x) {
  return (__double2hiint(x) & 0x7FF00000) == 0x7FF00000;
}

__device__ __forceinline__ double nan64() { return __longlong_as_double(0x7FF8000000000000ll); }

// |x| as an ordered integer (the bit pattern of a non-negative double grows with
// its value), for maxima without floating-point instructions
__device__ __forceinline__ unsigned long long absbits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
}

// the unsigned pattern of max(|re|, |im|) rounded to FP32, for atomicMax on
// non-negative floats
__device__ __forceinline__ unsigned bits_to_fmax(unsigned long long b) {
  return __float_as_uint(f64_to_f32(__longlong_as_double((long long)b)));
}

}  // namespace sbe
