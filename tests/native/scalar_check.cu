// The functions of scalar.cuh against CUDA's sqrt and division, for
// test_gpu_scalar.py.  Thread t of an exponent's row takes a mantissa: the
// smallest ones, the largest ones, powers of two apart, or pseudo-random.
#include "../../madsdp.jl_gb300/csrc/scalar.cuh"

namespace {
__device__ double number(int field, unsigned t, unsigned count) {
  unsigned long long m;
  if (t < 64) m = t;
  else if (t < 128) m = 0xFFFFFFFFFFFFFull - (t - 64);
  else if (t < 180) m = 1ull << (t - 128);
  else if (t < 232) m = 0xFFFFFFFFFFFFFull >> (t - 180);
  else {
    m = ((unsigned long long)field * count + t) * 0x9E3779B97F4A7C15ull;
    m ^= m >> 33; m *= 0xff51afd7ed558ccdull; m ^= m >> 33; m *= 0xc4ceb9fe1a85ec53ull; m ^= m >> 33;
    m &= 0xFFFFFFFFFFFFFull;
  }
  return __longlong_as_double((long long)(((unsigned long long)field << 52) | m));
}
// |x - y| in units of y's last place (both of one sign, finite)
__device__ unsigned long long ulps(double x, double y) {
  const long long d = __double_as_longlong(x) - __double_as_longlong(y);
  return (unsigned long long)(d < 0 ? -d : d);
}
// 1/sqrt(d) rounded once: the reciprocal of a rounded root is off by that root's
// error too, so it gets the residual 1 - d v^2 (formed without rounding d v)
__device__ double inverse_root(double d) {
  const double v = 1.0 / sqrt(d), p = d * v, pe = fma(d, v, -p);
  const double r = fma(-p, v, 1.0) - pe * v;
  return fma(0.5 * r, v, v);
}
// largest distances: 0, 1 fast_root's root and reciprocal, 2, 3 exact_root's,
// 4 fast_inverse, 5 fast_quotient, 6 widen, 7 bits_to_float (truncation, FP32 ulps)
__global__ void k_check(unsigned count, unsigned long long* worst) {
  const int field = blockIdx.x;  // 0: subnormal numbers
  unsigned long long w[6] = {0, 0, 0, 0, 0, 0};
  for (unsigned t = threadIdx.x; t < count; t += blockDim.x) {
    const double d = number(field, t, count);
    if (!(d > 0.0)) continue;
    const double s = sqrt(d), v = 1.0 / s;
    double root, inv;
    exact_root(d, root, inv);
    w[2] = max(w[2], ulps(root, s));
    w[3] = max(w[3], ulps(inv, v));
    if (field > 0) {
      fast_root(d, root, inv);
      w[0] = max(w[0], ulps(root, s));
      w[1] = max(w[1], ulps(inv, inverse_root(d)));
    }
    if (field >= 2 && field <= 2044) w[4] = max(w[4], ulps(fast_inverse(d), 1.0 / d));
    // quotients whose value is normal: x of d's exponent and its neighbours'
    for (int k = -1; k <= 1; ++k) {
      const int xf = field + k;
      if (xf < 1 || xf > 2046) continue;
      const double x = number(xf, count - 1 - t, count);
      w[5] = max(w[5], ulps(fast_quotient(x, d), x / d));
      w[5] = max(w[5], ulps(-fast_quotient(-x, d), x / d));
    }
    if (fast_quotient(0.0, d) != 0.0) w[5] = ~0ull;
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) atomicMax(worst + i, w[i]);
}
// every float
__global__ void k_widen(unsigned long long* worst) {
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < (1ull << 32);
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const float f = __int_as_float((int)(unsigned)i);
    const double a = widen(f), b = (double)f;
    if (f == f && __double_as_longlong(a) != __double_as_longlong(b)) atomicMax(worst + 6, 1ull);
    const int e = exponent_field(b) - 1023;
    // truncation of a float's own value loses nothing where it is normal
    if (f == f && e >= -126 && e <= 127 && bits_to_float(b, 0) != f) atomicMax(worst + 7, 1ull);
    if (f == 0.0f && bits_to_float(b, -1000) != 0.0f) atomicMax(worst + 7, 1ull);
  }
}
}  // namespace

extern "C" int check_scalar(unsigned count, unsigned long long* out) {
  unsigned long long* d = nullptr;
  cudaError_t e = cudaMalloc(&d, 8 * sizeof(*d));
  if (e == cudaSuccess) e = cudaMemset(d, 0, 8 * sizeof(*d));
  if (e == cudaSuccess) {
    k_check<<<2047, 256>>>(count, d);
    k_widen<<<1216, 256>>>(d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d, 8 * sizeof(*d), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
