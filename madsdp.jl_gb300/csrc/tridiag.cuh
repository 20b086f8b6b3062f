// Device helpers of the Lanczos iterations: the smallest eigenvalue of a
// symmetric tridiagonal by multisection with the division-free Sturm
// sequence.
//
// With p_0 = 1, p_1 = a_0 - x, p_i = (a_{i-1} - x) p_{i-1} - b_{i-1}^2 p_{i-2},
// x lies below the smallest eigenvalue exactly when every p_i is positive.
// Three FP64 instructions per row (about 64 clocks each on GB300) where the
// quotient form needs a division (about 700).  The matrix is scaled by a power
// of two to a norm of at most 1 and the pair of values is rescaled every
// eighth row, so nothing under- or overflows.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "scalar.cuh"

// v * 2^e for a normal v whose result is normal, or 0
__device__ __forceinline__ double exp_add(double v, int e) {
  return v == 0.0 ? 0.0 : __longlong_as_double(__double_as_longlong(v) + ((long long)e << 52));
}

// Every p_i of the scaled tridiagonal (diagonal a, squared off-diagonal b2,
// b2[i] between rows i - 1 and i) is positive at x.
__device__ __forceinline__ bool sturm_above(int k, const double* a, const double* b2, double x) {
  double p0 = 1.0, p1 = a[0] - x;
  bool pos = __double2hiint(p1) > 0;
  for (int i = 1; i < k; ++i) {
    const double p = fma(a[i] - x, p1, -(b2[i] * p0));
    p0 = p1;
    p1 = p;
    pos = pos && __double2hiint(p) > 0;
    if ((i & 7) == 7) {
      if (__all_sync(0xffffffffu, !pos)) return false;
      if (pos) {
        const int sh = (__double2hiint(p1) >> 20) - 1023;
        p1 = __longlong_as_double(__double_as_longlong(p1) - ((long long)sh << 52));
        p0 = __longlong_as_double(__double_as_longlong(p0) - ((long long)sh << 52));
      } else {
        p0 = p1 = 0.0;  // decided: p stays 0, which is not positive
      }
    }
  }
  return pos;
}
__device__ __forceinline__ bool sturm_above32(int k, const float* a, const float* b2, float x) {
  float p0 = 1.0f, p1 = a[0] - x;
  bool pos = p1 > 0.0f;
  for (int i = 1; i < k; ++i) {
    const float p = fmaf(a[i] - x, p1, -(b2[i] * p0));
    p0 = p1;
    p1 = p;
    pos = pos && p > 0.0f;
    if ((i & 1) == 1 && pos) {
      const int sh = (__float_as_int(p1) >> 23) - 127;
      const float f = __int_as_float((127 - max(min(sh, 126), -126)) << 23);
      p1 *= f;
      p0 *= f;
    }
  }
  return pos;
}

struct TridiagShared {
  double theta;
  int e, first[2][4];
  float lo;
};

// ---- block-wide forms: called by every thread of the block (at least 128)

// Scaled copies of the tridiagonal (a, b), b[i] between rows i - 1 and i:
// sa = a 2^-e, sb = (b 2^-e)^2 with the norm at most 2^e; returns e.  The norm is
// taken in FP32: the caller sees to it that it is below 2^126.
__device__ inline int tridiag_scale(int k, const double* a, const double* b, double* sa, double* sb, float* saf,
                                    float* sbf, TridiagShared& sh) {
  const int t = threadIdx.x;
  if (t < 32) {
    float m = 0.0f;
    for (int i = t; i < k; i += 32)
      m = fmaxf(m, fabsf((float)a[i]) + (i > 0 ? fabsf((float)b[i]) : 0.0f) + (i + 1 < k ? fabsf((float)b[i + 1]) : 0.0f));
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (t == 0) {
      // m 1.001 < 2^e
      const float g = fmaxf(m * 1.001f, 1e-37f);
      sh.e = min((__float_as_int(g) >> 23) - 126, 127);
    }
  }
  __syncthreads();
  const int e = sh.e;
  const double f = __longlong_as_double((long long)(1023 - e) << 52);
  for (int i = t; i < k; i += blockDim.x) {
    const double x = a[i] * f, y = i > 0 ? b[i] * f : 0.0, y2 = y * y;
    sa[i] = x;
    sb[i] = y2;
    saf[i] = (float)x;
    sbf[i] = (float)y2;
  }
  __syncthreads();
  return e;
}

// Smallest eigenvalue of the scaled tridiagonal in FP32 (five rounds of 32
// points, width 2 33^-5).
__device__ inline float tridiag_min32(int k, const float* saf, const float* sbf, TridiagShared& sh) {
  const int t = threadIdx.x;
  if (t < 32) {
    float lo = -1.0f, hi = 1.0f;
    for (int it = 0; it < 5; ++it) {
      const float h = (hi - lo) / 33.0f;
      const unsigned above = __ballot_sync(0xffffffffu, sturm_above32(k, saf, sbf, lo + h * (float)(t + 1)));
      // the first point that is not below the eigenvalue
      const int first = above == 0xffffffffu ? 32 : __ffs(~above) - 1;
      const float l = lo;
      lo = l + h * (float)first;
      if (first < 32) hi = l + h * (float)(first + 1);
    }
    if (t == 0) sh.lo = 0.5f * (lo + hi);
  }
  __syncthreads();
  return sh.lo;
}

// The same in FP64 around an FP32 value: rounds of 128 points on the first
// four warps (one per quarter of the SM) until the bracket is 2 eps |theta| or
// a quarter eps of the norm wide; the whole interval when the FP32 value
// misses.  Returns theta 2^e.  The other warps only wait: FP64 work on them
// would hold up the four.
__device__ inline double tridiag_min64(int k, const double* sa, const double* sb, float th32, int e, TridiagShared& sh) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const double eps = 2.220446049250313e-16;
  if (warp < 4) {
    for (int attempt = 0;; ++attempt) {
      const double lo0 = attempt ? -1.0 : fmax(-1.0, (double)th32 - 8e-6), hi0 = attempt ? 1.0 : fmin(1.0, (double)th32 + 8e-6);
      double lo = lo0, hi = hi0;
      bool lo_moved = false, hi_moved = false;
      for (int it = 0; it < 16; ++it) {
        if (hi - lo <= fmax(2.0 * eps * fmax(fabs(lo), fabs(hi)), 0.25 * eps)) break;
        const double h = (hi - lo) * (1.0 / 129.0);
        const unsigned above = __ballot_sync(0xffffffffu, sturm_above(k, sa, sb, fma(h, (double)(t + 1), lo)));
        if (lane == 0) sh.first[it & 1][warp] = above == 0xffffffffu ? 32 : __ffs(~above) - 1;
        asm volatile("bar.sync 1, 128;" ::: "memory");
        int first = 128;
#pragma unroll
        for (int w = 3; w >= 0; --w)
          if (sh.first[it & 1][w] < 32) first = w * 32 + sh.first[it & 1][w];
        const double l = lo;
        lo = fma(h, (double)first, l);
        lo_moved = lo_moved || first > 0;
        if (first < 128) {
          hi = fma(h, (double)(first + 1), l);
          hi_moved = true;
        }
      }
      // an end that never moved was not tested: once more over the whole interval,
      // after every warp has read the last round's entries of `first`
      if (attempt == 0 && ((!lo_moved && lo0 > -1.0) || (!hi_moved && hi0 < 1.0))) {
        asm volatile("bar.sync 1, 128;" ::: "memory");
        continue;
      }
      if (t == 0) sh.theta = exp_add(0.5 * (lo + hi), e);
      break;
    }
  }
  __syncthreads();
  return sh.theta;
}
