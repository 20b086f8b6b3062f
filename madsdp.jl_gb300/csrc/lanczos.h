// lambda_min of formed symmetric matrices by Lanczos with full
// reorthogonalization: the eigenvalue behind EigenStep's step length
// (src/step.jl:151-183).  Up to order 256 the whole iteration of one matrix
// runs in one thread-block cluster; above, each step is two launches.
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

// ---- orders above kMaxOrder: steps driven by the host
constexpr int kMaxSteps = 320;

// Device arrays of one iteration: basis Q (n x (kMaxSteps + 1), column 0 the
// normalized start vector), w (n), and the tridiagonal: ab[0 .. kMaxSteps) the
// diagonal, ab[kMaxSteps ..) the squared off-diagonal.
struct Large {
  int n = 0;
  const double* Z = nullptr;
  double *Q = nullptr, *w = nullptr, *ab = nullptr;
};
// Steps [k0, k1) of one matrix on a stream (two launches each).
cudaError_t large_steps(const Large& a, int k0, int k1, cudaStream_t st);

}  // namespace lanczos
