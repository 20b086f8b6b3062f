// Reciprocals and roots of single numbers by short chains of FP64 instructions
// (each holds its quarter of a GB300 SM for about 64 clocks, a division about
// 700 and a square root about 770), and tests on the bits (a comparison of
// doubles costs as much as a multiply-add).
//
// Reciprocal and reciprocal root start from FP32 and take one step of
// Householder's iteration of third order (A. S. Householder, The Numerical
// Treatment of a Single Nonlinear Equation, 1970): y (1 + e + e^2) with
// e = 1 - m y for 1/m, y (1 + e/2 + 3/8 e^2) with e = 1 - m y^2 for
// 1/sqrt(m).  Last corrections are Markstein's (P. W. Markstein, Computation of
// elementary functions on the IBM RISC System/6000 processor, IBM J. Res.
// Dev. 34, 1990): a residual by a fused multiply-add, times half the reciprocal.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

// Biased binary exponent: 0 for zero and subnormal numbers, 2047 for infinities
// and NaN.
__device__ __forceinline__ int exponent_field(double v) { return (__double2hiint(v) >> 20) & 0x7FF; }

// positive and finite
__device__ __forceinline__ bool pivot_ok(double d) {
  const long long b = __double_as_longlong(d);
  return b > 0 && b < 0x7FF0000000000000ll;
}
__device__ __forceinline__ bool pivot_ok(float d) {
  const int b = __float_as_int(d);
  return b > 0 && b < 0x7F800000;
}

// sqrt(d) within 2 ulp and 1/sqrt(d) within 1, of a positive, normal, finite d:
// about 300 clocks of dependent FP64 instructions, where sqrt and a division
// take about 1500.
__device__ __forceinline__ void fast_root(double d, double& root, double& inv) {
  const long long b = __double_as_longlong(d);
  const int field = (int)(b >> 52);
  const int k = (field - 1023) >> 1, odd = (field - 1023) & 1;
  const double m = __longlong_as_double((b & 0xFFFFFFFFFFFFFll) | ((long long)(1023 + odd) << 52));  // [1, 4)
  const double y = (double)rsqrtf((float)m);
  const double e = fma(-m * y, y, 1.0);
  const double z = fma(y * e, fma(0.375, e, 0.5), y);
  inv = __longlong_as_double(__double_as_longlong(z) - ((long long)k << 52));
  const double s = d * inv;
  root = fma(fma(-s, s, d) * 0.5, inv, s);
}

// sqrt(d) and 1/sqrt(d) of a positive finite d as sqrt and a division round
// them, in about 700 clocks.
__device__ __forceinline__ void exact_root(double d, double& root, double& inv) {
  if (__double2hiint(d) < 0x06400000) {  // below 2^-923 the residuals fall out of range
    root = sqrt(d);
    inv = 1.0 / root;
    return;
  }
  fast_root(d, root, inv);
  // the correction of the reciprocal misses where the root's mantissa is all ones
  const long long b = __double_as_longlong(root);
  inv = (b & 0xFFFFFFFFFFFFFll) == 0xFFFFFFFFFFFFFll ? 1.0 / root : fma(fma(-root, inv, 1.0), inv, inv);
}

// 1/d within 1 ulp of a positive d of 2^-1021 to 2^1022 (beyond, the result is
// subnormal or infinite): four dependent FP64 instructions from the reciprocal
// of d's mantissa in FP32, both conversions by integer instructions.
__device__ __forceinline__ double fast_inverse(double d) {
  const long long b = __double_as_longlong(d);
  const int field = (int)(b >> 52);  // 2 to 2044
  const double m = __longlong_as_double((b & 0xFFFFFFFFFFFFFll) | 0x3FF0000000000000ll);  // [1, 2)
  const float f = __frcp_rn(__int_as_float(0x3F800000 | (int)((b >> 29) & 0x7FFFFF)));    // (0.5, 1]
  const int fb = __float_as_int(f);
  const double y = __hiloint2double(((fb >> 3) & 0x0FFFFFFF) + 0x38000000, fb << 29);
  const double e = fma(-m, y, 1.0);
  const double z = fma(y, fma(e, e, e), y);
  return __longlong_as_double(__double_as_longlong(z) - ((long long)(field - 1023) << 52));
}
// x / d of a positive finite d within 2 ulp; a division where 1/d leaves the
// normal range (0 times an infinite reciprocal is no zero).
__device__ __forceinline__ double fast_quotient(double x, double d) {
  const int field = __double2hiint(d) >> 20;
  return field < 2 || field > 2044 ? x / d : x * fast_inverse(d);
}
__device__ __forceinline__ float fast_quotient(float x, float d) {
  const int field = __float_as_int(d) >> 23;
  return field < 2 || field > 252 ? x / d : x * (1.0f / d);
}

// (double)x exactly, by integer instructions: the conversion occupies the FP64
// unit like a multiply-add.
__device__ __forceinline__ double widen(float x) {
  const int b = __float_as_int(x);
  if ((b & 0x7F800000) == 0 || (b & 0x7F800000) == 0x7F800000) return (double)x;  // 0, subnormal, infinite, NaN
  return __hiloint2double((b & 0x80000000) | (((b & 0x7FFFFFFF) >> 3) + 0x38000000), b << 29);
}
__device__ __forceinline__ double widen(double x) { return x; }

// The leading 24 bits of v 2^-e (zero when that is below FP32's normal range,
// the largest float above it), by integer instructions.
__device__ __forceinline__ float bits_to_float(double v, int e) {
  const long long b = __double_as_longlong(v);
  const int raw = (int)(b >> 52) & 0x7FF, field = raw - 1023 - e + 127;
  if (raw == 0 || field <= 0) return 0.0f;
  const int mag = field >= 255 ? 0x7F7FFFFF : (field << 23) | ((int)(b >> 29) & 0x7FFFFF);
  return __int_as_float(mag | ((int)(b >> 32) & 0x80000000));
}
