// Cluster Lanczos for the step lengths; see lanczos.h.
#include "lanczos.h"

#include <algorithm>
#include <mutex>

#include "tridiag.cuh"

namespace lanczos {
namespace {

constexpr int kThreads = 512;
constexpr int kSmemMax = 226 * 1024;
constexpr double kEps = 2.220446049250313e-16;

// Shared memory (doubles) of one block of a cluster of cs.
__host__ __device__ inline int64_t smem_doubles(int n, int cs) {
  const int nr = (n + cs - 1) / cs;
  // Z rows, basis rows, q, w, partial sums (two stages), coefficients, the
  // tridiagonal and its scaled copies, the exchange of partial coefficients
  return (int64_t)n * nr + (int64_t)nr * (n | 1) + n + nr + 2 * kThreads + (n + 2) + 5 * (n + 2) +
         (cs > 1 ? 2 * (int64_t)cs * (n + 2) : 0);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void store_remote(const double* p, int rank, double v) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// Every block of the cluster holds a slice of the rows of Z and of the basis
// in shared memory for the whole iteration.  Per step: w = Z q on the slice;
// two passes of classical Gram-Schmidt against the whole basis (the first
// pass's last two coefficients are alpha and beta), whose coefficients are
// summed over the cluster; the second pass also carries w'w, so the new
// norm needs no reduction of its own; the slice of the new q goes to every
// block.  Sums are split over threads as (output, part of the sum) pairs, all
// of the block's threads busy whatever n and the step are, because a FP64
// instruction occupies a quarter of the SM for 64 to 76 clocks and nothing
// overlaps it; all blocks of a cluster form every total in the same order and
// so take the same decisions.
//
// The start vector and the stopping rule are fixed: the smallest Ritz value
// every 4 steps, until it moves by at most 64 eps max(1, |theta|) or the
// Krylov space is exhausted.  The Ritz value is looked at in FP32 first; the
// FP64 values of this check and of the one before are formed only when the
// FP32 ones differ by less than 3e-6 of the norm: they are within 5e-7 of it
// (the rounding of the tridiagonal and of the Sturm sequence, 4 eps, and the
// bracket), so a move of 64 eps cannot be missed.
//
// One block of 256 threads per matrix with Z and the basis in global memory
// and divisions in the Sturm counts took 1.41 ms a launch at n = 100 (two
// matrices, about 28 steps); this takes 0.39 ms, and 1.08 ms for a launch over
// blocks of 120, 60, 30 and 30 (4.96 ms before).
__global__ void __launch_bounds__(kThreads) k_lanczos(const Job* __restrict__ jobs) {
  int cs, rank;
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(cs));
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const Job J = jobs[blockIdx.x / cs];
  const int n = J.n, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int nrm = (n + cs - 1) / cs, r0 = min(n, rank * nrm), nr = min(n, r0 + nrm) - r0, ldq = n | 1;
  extern __shared__ double sm[];
  double* Zs = sm;                              // [n][nr]: Zs[r * nr + i] = Z(r0 + i, r)
  double* Qs = Zs + (int64_t)n * nrm;           // [nr][ldq]
  double* qs = Qs + (int64_t)nrm * ldq;         // [n]
  double* ws = qs + n;                          // [nr]
  double* part = ws + nrm;                      // [kThreads]
  double* part2 = part + kThreads;              // [kThreads]
  double* coef = part2 + kThreads;              // [n + 2]
  double* al = coef + n + 2;                    // [n + 2] each
  double* be = al + n + 2;
  double* sa = be + n + 2;                      // scaled diagonal
  double* sb = sa + n + 2;                      // scaled squared off-diagonal
  float* saf = (float*)(sb + n + 2);            // the same in FP32
  float* sbf = saf + n + 2;
  double* xch = (double*)(sbf + n + 2);         // [2][cs][n + 2], clusters of more than one block
  __shared__ TridiagShared tsh;
  __shared__ double red[8];
  __shared__ int state, stop;

  auto cluster_sync = [&] {
    if (cs == 1) __syncthreads();
    else
      asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
  };
  for (int idx = t; idx < n * nr; idx += kThreads) {
    const int r = idx / nr, i = idx - r * nr;
    Zs[idx] = J.Z[r0 + i + (int64_t)r * n];
  }
  // the start vector, whole on every block
  double v = 0.0;
  if (t < n) {
    uint32_t h = (uint32_t)(t + 1) * 2654435761u;
    h ^= h >> 15; h *= 2246822519u; h ^= h >> 13;
    v = (double)(h & 0xffffff) / 16777216.0 - 0.5 + 0.01;
  }
  if (warp < 8) {
    double s = v * v;
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) red[warp] = s;
  }
  __syncthreads();
  if (t < n) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += red[w];
    v /= sqrt(s);
    qs[t] = v;
    if (t >= r0 && t < r0 + nr) Qs[(t - r0) * ldq] = v;
  }
  if (t == 0) be[0] = 0.0;
  cluster_sync();

  const int U = nr > 64 ? 1 : nr > 32 ? 2 : 4;  // parts of an update: four warps in all
  // parts of a sum split over threads: a power of two, at most 16
  auto parts_of = [](int outputs) {
    int c = 16;
    while (c > 1 && c * outputs > kThreads) c >>= 1;
    return c;
  };
  // part[c * count + o] (c < parts) -> the sum over c, by thread o
  auto combine = [&](int count, int parts) -> double {
    __syncthreads();
    double s = 0.0;
    if (parts > 4) {
      const int g = parts >> 2;  // partial sums of four
      if (t < count * g) {
        const int o = t % count, c = (t / count) * 4;
        part2[t] = (part[c * count + o] + part[(c + 1) * count + o]) +
                   (part[(c + 2) * count + o] + part[(c + 3) * count + o]);
      }
      __syncthreads();
      if (t < count)
        for (int c = 0; c < g; ++c) s += part2[c * count + t];
    } else if (t < count) {
      for (int c = 0; c < parts; ++c) s += part[c * count + t];
    }
    return s;
  };
  double theta = 0.0, theta_prev = INFINITY, znorm = 0.0;
  float theta32_prev = INFINITY;
  bool have_prev = false;  // theta_prev is the FP64 value of the check before
  for (int j = 0; j < n; ++j) {
    // ---- w = Z q on the slice
    double w = 0.0;
    if (nr > 0) {
      const int C = parts_of(nr);
      const int i = t % nr, c = t / nr;
      if (c < C) {
        const int ra = c * n / C, rb = (c + 1) * n / C;
        double s = 0.0;
#pragma unroll 4
        for (int r = ra; r < rb; ++r) s = fma(Zs[r * nr + i], qs[r], s);
        part[c * nr + i] = s;
      }
      w = combine(nr, C);
      if (t < nr) ws[t] = w;
    }
    // ---- two Gram-Schmidt passes against q_0 .. q_j
    const int L = j + 1;
    bool large = false;
    for (int pass = 0; pass < 2; ++pass) {
      const int LL = L + pass;  // the second pass's last output is w'w
      const int C = parts_of(LL);
      __syncthreads();
      {
        const int l = t % LL, c = t / LL;
        if (c < C) {
          const int ia = c * nr / C, ib = (c + 1) * nr / C;
          double s = 0.0;
          if (l < L) {
#pragma unroll 4
            for (int i = ia; i < ib; ++i) s = fma(Qs[i * ldq + l], ws[i], s);
          } else {
            for (int i = ia; i < ib; ++i) s = fma(ws[i], ws[i], s);
          }
          part[c * LL + l] = s;
        }
      }
      double s = combine(LL, C);
      if (cs > 1) {
        double* x = xch + (int64_t)pass * cs * (n + 2);
        if (t < LL)
          for (int r = 0; r < cs; ++r) store_remote(x + (int64_t)rank * (n + 2) + t, r, s);
        cluster_sync();
        if (t < LL) {
          s = 0.0;
          for (int r = 0; r < cs; ++r) s += x[(int64_t)r * (n + 2) + t];
        }
      }
      if (t < LL) coef[t] = s;
      __syncthreads();
      if (t < nr * U) {
        const int i = t % nr, u = t / nr, la = u * L / U, lb = (u + 1) * L / U;
        const double* q = Qs + i * ldq;
        double s1 = 0.0;
#pragma unroll 4
        for (int l = la; l < lb; ++l) s1 = fma(-coef[l], q[l], s1);
        part[t] = s1;
      }
      __syncthreads();
      if (t < nr) {
        double s1 = part[t];
        for (int u = 1; u < U; ++u) s1 += part[u * nr + t];
        w += s1;
        if (pass == 0) ws[t] = w;
      }
      if (pass == 0 && t == 0) al[j] = coef[j];
      if (pass == 1) {
        // a coefficient above 2^-30 |w'| changes the norm
        const int en = (__double2hiint(coef[L]) >> 20) - 1023;
        const int ec = t < L ? ((__double2hiint(coef[t]) >> 20) & 0x7ff) - 1023 : -2000;
        large = __syncthreads_or(2 * ec > en - 60);
      }
    }
    // ---- the norm (the warps that need it), the new basis vector, the state
    // of the iteration (thread 0)
    const int k = j + 1;
    if (warp * 32 < nr || warp == 0) {
      double bn2 = coef[L];
      if (large)
        for (int l = 0; l < L; ++l) bn2 = fma(-coef[l], coef[l], bn2);
      const int field = __double2hiint(bn2) >> 20;  // 0x7ff: infinite or NaN; below 27: 1e-300 or negative
      double bn = 0.0, binv = 0.0;
      if (field > 27 && field < 0x7ff) fast_root(bn2, bn, binv);
      if (t < nr && k < n) {
        const double q = w * binv;
        Qs[t * ldq + k] = q;
        if (cs == 1) qs[t] = q;
        else
          for (int r = 0; r < cs; ++r) store_remote(qs + r0 + t, r, q);
      }
      if (t == 0) {
        const double aj = al[j], bj = j > 0 ? be[j] : 0.0;
        znorm = fmax(znorm, fabs(aj) + bn + fabs(bj));
        be[k] = bn;
        const bool bad = field == 0x7ff || (__double2hiint(aj) & 0x7ff00000) == 0x7ff00000;
        state = bad ? 2 : !(bn > 4.0 * kEps * znorm) ? 1 : 0;
      }
    }
    cluster_sync();
    if (state == 2) {  // infinite or NaN entries: no eigenvalue
      theta = nan("");
      break;
    }
    const bool exhausted = k == n || state == 1;
    if (exhausted || (k >= 4 && (k & 3) == 0)) {
      const int e = tridiag_scale(k, al, be, sa, sb, saf, sbf, tsh);
      const float th32 = tridiag_min32(k, saf, sbf, tsh);  // in units of 2^e
      const float here = ldexpf(th32, e);
      if (exhausted) {
        theta = tridiag_min64(k, sa, sb, th32, e, tsh);
        break;
      }
      if (fabsf(here - theta32_prev) <= 3e-6f * ldexpf(1.0f, e)) {
        theta = tridiag_min64(k, sa, sb, th32, e, tsh);
        if (!have_prev) {
          const double th = theta;
          __syncthreads();
          theta_prev = tridiag_min64(k - 4, sa, sb, ldexpf(theta32_prev, -e), e, tsh);
          theta = th;
        }
        if (t == 0) stop = fabs(theta - theta_prev) <= 64.0 * kEps * fmax(1.0, fabs(theta));
        __syncthreads();
        if (stop) break;
        theta_prev = theta;
        have_prev = true;
      } else {
        have_prev = false;
      }
      theta32_prev = here;
    }
  }
  if (rank == 0 && t == 0) *J.out = theta;
  // no block leaves while another may still reach its shared memory
  if (cs > 1) cluster_sync();
}

}  // namespace

cudaError_t eigmin(const Job* jobs, int count, int nmax, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  if (nmax > kMaxOrder) return cudaErrorInvalidValue;
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(k_lanczos, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
  });
  if (attr != cudaSuccess) return attr;
  // 32 rows a block: the FP64 units of one SM are the bound below (at n = 100
  // a step takes 18000 clocks in one block, most of it their work, and an
  // exchange in the cluster 1200); a full basis and the rows of Z fit at 256
  int cs = 1;
  while (cs < 8 && (nmax + cs - 1) / cs > 32) cs *= 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(count * cs));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = (size_t)(smem_doubles(nmax, cs) * 8);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cs;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_lanczos, jobs);
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace lanczos
