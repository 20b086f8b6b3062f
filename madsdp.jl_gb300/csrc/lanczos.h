// lambda_min of formed symmetric matrices up to order 256 by Lanczos with
// full reorthogonalization, one thread-block cluster per matrix: the
// eigenvalue behind EigenStep's step length (src/step.jl:151-183).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace lanczos {

constexpr int kMaxOrder = 256;

// One matrix: Z (n x n, device), result *out (device).
struct Job {
  int n;
  const double* Z;
  double* out;
};

// All jobs (a device array) in one launch; nmax is the largest order among
// them.
cudaError_t eigmin(const Job* jobs, int count, int nmax, cudaStream_t st);

}  // namespace lanczos
