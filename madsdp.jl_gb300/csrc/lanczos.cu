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

__device__ __forceinline__ void store_remote_int(const int* p, int rank, int v) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
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
  __shared__ int state, stop, top_s, tops[8];

  auto cluster_sync = [&] {
    if (cs == 1) __syncthreads();
    else
      asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
  };
  if (t == 0) top_s = 0;
  __syncthreads();
  int top = 0;  // exponent of the largest entry
  for (int idx = t; idx < n * nr; idx += kThreads) {
    const int r = idx / nr, i = idx - r * nr;
    const double z = J.Z[r0 + i + (int64_t)r * n];
    Zs[idx] = z;
    top = max(top, (__double2hiint(z) >> 20) & 0x7FF);
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) atomicMax(&top_s, top);
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
  // Entries outside 2^-100 to 2^100 are scaled to 1: squares and the FP32 norm
  // of the tridiagonal stay in range.  (Infinities and NaN are left to `state`.)
  if (cs > 1) {
    if (t < cs) store_remote_int(tops + rank, t, top_s);
    cluster_sync();
    top = 0;
    for (int r = 0; r < cs; ++r) top = max(top, tops[r]);
  } else {
    top = top_s;
  }
  const bool scaled = top < 0x7FF && (top < 923 || top > 1123);
  const int up = scaled ? min(max(1023 - top, -1022), 1022) : 0;
  const double unit = __longlong_as_double((long long)(1023 + up) << 52);  // 1 of Z's units
  if (scaled) {
    for (int idx = t; idx < n * nr; idx += kThreads) Zs[idx] *= unit;
    __syncthreads();
  }

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
        if (t == 0) stop = fabs(theta - theta_prev) <= 64.0 * kEps * fmax(unit, fabs(theta));
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
  if (rank == 0 && t == 0) *J.out = scaled ? theta * __longlong_as_double((long long)(1023 - up) << 52) : theta;
  // no block leaves while another may still reach its shared memory
  if (cs > 1) cluster_sync();
}

// ---------------------------------------------------------------- orders above 256
// w = Z q, Z symmetric and read by columns: one warp per entry.  Bound by the
// FP64 units (n^2 multiply-adds at 1.6 per clock and SM: 8 us at n = 2000); a
// block per entry with a block-wide sum took 24 us.
constexpr int kMatvecThreads = 128;
__global__ void __launch_bounds__(kMatvecThreads) k_matvec(int n, const double* __restrict__ Z,
                                                          const double* __restrict__ q, double* __restrict__ w) {
  const int lane = threadIdx.x & 31;
  const int j = blockIdx.x * (kMatvecThreads / 32) + (threadIdx.x >> 5);
  if (j >= n) return;
  const double* a = Z + (int64_t)j * n;
  double s = 0.0;
#pragma unroll 8
  for (int i = lane; i < n; i += 32) s = fma(a[i], q[i], s);
#pragma unroll
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) w[j] = s;
}

// Orthogonalization of w against q_0 .. q_j (twice) and the next basis vector,
// in one cluster: every block holds a slice of the rows, the coefficients'
// partial sums go to all blocks through distributed shared memory, and all add
// them in the same order.  The second pass carries w'w, so the new norm
// needs no exchange of its own (as in k_lanczos).  A warp sums four
// coefficients at a time, so that their reduction takes six additions, not
// twenty.  Bound by 4 j n multiply-adds on the FP64 units of 16 SMs, about
// 12 us at n = 2000, j = 70; five launches over the whole GPU took 25 us and
// the gaps between them as much again.
__host__ __device__ inline int64_t large_smem(int n, int cs) {
  const int nr = (n + cs - 1) / cs;
  return 8 * ((int64_t)nr + kThreads + 2 * (kMaxSteps + 2) + 2 * (int64_t)cs * (kMaxSteps + 2));
}
__global__ void __launch_bounds__(kThreads) k_orthogonalize(int n, int j, double* __restrict__ Q,
                                                           const double* __restrict__ w, double* __restrict__ ab) {
  int cs, rank;
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(cs));
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int nrm = (n + cs - 1) / cs, r0 = min(n, rank * nrm), nr = min(n, r0 + nrm) - r0;
  extern __shared__ double sm[];
  double* ws = sm;                       // [nrm]
  double* part = ws + nrm;               // [kThreads]
  double* mine = part + kThreads;        // [kMaxSteps + 2] partial sums of this block
  double* coef = mine + kMaxSteps + 2;   // [kMaxSteps + 2]
  double* xch = coef + kMaxSteps + 2;    // [2][cs][kMaxSteps + 2]
  auto cluster_sync = [&] {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
  };
  for (int i = t; i < nr; i += kThreads) ws[i] = w[r0 + i];
  cluster_sync();  // every block has started before its shared memory is written
  const double* Qr = Q + r0;
  const int L = j + 1;
  bool large = false;
  for (int pass = 0; pass < 2; ++pass) {
    const int LL = L + pass;  // the second pass's last output is w'w
    // ---- partial coefficients, four per warp at a time
    for (int l0 = 4 * warp; l0 < LL; l0 += 4 * (kThreads / 32)) {
      const double* p[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) p[u] = l0 + u < L ? Qr + (int64_t)(l0 + u) * n : ws;  // the last: w itself
      double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
      for (int i = lane; i < nr; i += 32) {
        const double x = ws[i];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = fma(p[u][i], x, v[u]);
      }
      const bool hi = lane & 16, mid = lane & 8;
      const double s0 = (hi ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], 16);
      const double s1 = (hi ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], 16);
      double s = (mid ? s1 : s0) + __shfl_xor_sync(0xffffffffu, mid ? s0 : s1, 8);
#pragma unroll
      for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const int l = l0 + (lane >> 3);
      if ((lane & 7) == 0 && l < LL) mine[l] = s;
    }
    __syncthreads();
    double* x = xch + (int64_t)pass * cs * (kMaxSteps + 2);
    for (int idx = t; idx < LL * cs; idx += kThreads)
      store_remote(x + (int64_t)rank * (kMaxSteps + 2) + idx % LL, idx / LL, mine[idx % LL]);
    cluster_sync();
    for (int l = t; l < LL; l += kThreads) {
      double s = 0.0;
      for (int r = 0; r < cs; ++r) s += x[(int64_t)r * (kMaxSteps + 2) + l];
      coef[l] = s;
    }
    __syncthreads();
    if (pass == 0 && rank == 0 && t == 0) ab[j] = coef[j];
    // ---- w -= Q coef: rows in groups of 128, four parts of the sum each
    for (int i0 = 0; i0 < nr; i0 += 128) {
      const int i = i0 + (t & 127), u = t >> 7;
      double s = 0.0;
      if (i < nr) {
        const double* q = Qr + i;
#pragma unroll 4
        for (int l = u * L / 4; l < (u + 1) * L / 4; ++l) s = fma(-coef[l], q[(int64_t)l * n], s);
      }
      part[t] = s;
      __syncthreads();
      if (t < 128 && i < nr) ws[i] += (part[t] + part[t + 128]) + (part[t + 256] + part[t + 384]);
      __syncthreads();
    }
    if (pass == 1) {
      // a coefficient above 2^-30 |w'| changes the norm
      const int en = (__double2hiint(coef[L]) >> 20) - 1023;
      int ec = -2000;
      for (int l = t; l < L; l += kThreads) ec = max(ec, ((__double2hiint(coef[l]) >> 20) & 0x7ff) - 1023);
      large = __syncthreads_or(2 * ec > en - 60);
    }
  }
  if (t < 128) {
    double bn2 = coef[L];
    if (large)
      for (int l = 0; l < L; ++l) bn2 = fma(-coef[l], coef[l], bn2);
    const int field = __double2hiint(bn2) >> 20;
    double bn = 0.0, binv = 0.0;
    if (field > 0 && field < 0x7ff) fast_root(bn2, bn, binv);
    else bn2 = field == 0x7ff ? bn2 : 0.0;
    for (int i = t; i < nr; i += 128) Q[(int64_t)(j + 1) * n + r0 + i] = ws[i] * binv;
    if (rank == 0 && t == 0) ab[kMaxSteps + j] = bn2;
  }
  cluster_sync();
}

}  // namespace

cudaError_t large_steps(const Large& a, int k0, int k1, cudaStream_t st) {
  if (k1 > kMaxSteps || a.n <= 0) return cudaErrorInvalidValue;
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  static bool wide = false;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(k_orthogonalize, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    wide = cudaFuncSetAttribute(k_orthogonalize, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    cudaGetLastError();
  });
  if (attr != cudaSuccess) return attr;
  const int cs = wide ? 16 : 8;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)cs);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = (size_t)large_smem(a.n, cs);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cs;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cfg.dynamicSmemBytes > (size_t)kSmemMax) return cudaErrorInvalidValue;
  cudaError_t e = cudaSuccess;
  const unsigned grid = (unsigned)((a.n + kMatvecThreads / 32 - 1) / (kMatvecThreads / 32));
  for (int k = k0; k < k1 && e == cudaSuccess; ++k) {
    k_matvec<<<grid, kMatvecThreads, 0, st>>>(a.n, a.Z, a.Q + (int64_t)k * a.n, a.w);
    e = cudaLaunchKernelEx(&cfg, k_orthogonalize, a.n, k, a.Q, (const double*)a.w, a.ab);
    if (e == cudaSuccess) e = cudaGetLastError();
  }
  return e;
}

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
