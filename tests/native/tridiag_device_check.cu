// Device helpers of tridiag.cuh behind a C interface for test_gpu_tridiag.py.
#include "../../madsdp.jl_gb300/csrc/tridiag.cuh"

namespace {
constexpr int kMax = 256;

// smallest eigenvalue of each of `count` tridiagonals of k rows (a, b; b[i]
// between rows i - 1 and i) from the FP32 value plus `shift` (in units of the
// norm): 128 threads a block, one tridiagonal each
__global__ void __launch_bounds__(128) k_min(int k, const double* a, const double* b, const float* shift, double* out) {
  __shared__ double sa[kMax], sb[kMax], as[kMax], bs[kMax];
  __shared__ float saf[kMax], sbf[kMax];
  __shared__ TridiagShared sh;
  for (int i = threadIdx.x; i < k; i += 128) {
    as[i] = a[(int64_t)blockIdx.x * k + i];
    bs[i] = b[(int64_t)blockIdx.x * k + i];
  }
  __syncthreads();
  const int e = tridiag_scale(k, as, bs, sa, sb, saf, sbf, sh);
  const float th = tridiag_min32(k, saf, sbf, sh);
  const double t = tridiag_min64(k, sa, sb, th + shift[blockIdx.x], e, sh);
  if (threadIdx.x == 0) out[blockIdx.x] = t;
}
}  // namespace

extern "C" int check_min64(int count, int k, const double* a, const double* b, const float* shift, double* out) {
  if (k < 1 || k > kMax || count < 1) return -1;
  double *da = nullptr, *db = nullptr, *dout = nullptr;
  float* ds = nullptr;
  const size_t nb = sizeof(double) * count * k;
  cudaError_t e = cudaMalloc(&da, nb);
  if (e == cudaSuccess) e = cudaMalloc(&db, nb);
  if (e == cudaSuccess) e = cudaMalloc(&dout, sizeof(double) * count);
  if (e == cudaSuccess) e = cudaMalloc(&ds, sizeof(float) * count);
  if (e == cudaSuccess) e = cudaMemcpy(da, a, nb, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(db, b, nb, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(ds, shift, sizeof(float) * count, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_min<<<count, 128>>>(k, da, db, ds, dout);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, dout, sizeof(double) * count, cudaMemcpyDeviceToHost);
  cudaFree(da);
  cudaFree(db);
  cudaFree(dout);
  cudaFree(ds);
  return (int)e;
}
