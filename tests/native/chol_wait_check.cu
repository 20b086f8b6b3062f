// The blocked Cholesky with a limit of its own on the panel kernel's waits, for
// test_gpu_chol_waits.py.  Links against libmadsdp_gpu.so.
#include "../../madsdp.jl_gb300/csrc/chol.h"

// A (n x n, column-major, host) is factored in place; *info and *err as the
// device has them afterwards.
extern "C" int check_potrf(int n, double* A, int mixed, int polls, int* info, int* err) {
  char* mem = nullptr;
  double* dA = nullptr;
  const int64_t wb = chol::work_bytes(n);
  const size_t nb = sizeof(double) * n * n;
  cudaError_t e = cudaMalloc(&mem, wb + 256);
  if (e == cudaSuccess) e = cudaMalloc(&dA, nb);
  int* flags = (int*)(mem + wb);
  if (e == cudaSuccess) e = cudaMemset(flags, 0, 2 * sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpy(dA, A, nb, cudaMemcpyHostToDevice);
  chol::Work w;
  if (e == cudaSuccess) e = chol::init(&w, mem, n, flags + 1, nullptr, false);
  if (polls >= 0) w.polls = polls;
  if (e == cudaSuccess) e = chol::potrf(w, n, dA, n, flags, mixed ? tcg::kMixed : tcg::kFp64, nullptr, nullptr);
  int h[2] = {0, 0};
  if (e == cudaSuccess) e = cudaMemcpy(h, flags, sizeof(h), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(A, dA, nb, cudaMemcpyDeviceToHost);
  *info = h[0];
  *err = h[1];
  cudaFree(mem);
  cudaFree(dA);
  return (int)e;
}
