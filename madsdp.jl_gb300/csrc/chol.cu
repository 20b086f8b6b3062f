// Blocked Cholesky factorization with tensor-core trailing updates; see chol.h.
#include "chol.h"

#include <algorithm>
#include <mutex>

#include "tridiag.cuh"

namespace chol {
namespace {

constexpr int NB = 32;    // block column width (= K of the trailing update)
constexpr int ROWS = 32;  // panel rows per thread block, one per lane

__device__ __forceinline__ void pivot_root(double d, double& root, double& inv) {
  if (__double2hiint(d) < 0x00100000) {  // subnormal
    root = sqrt(d);
    inv = 1.0 / root;
    return;
  }
  fast_root(d, root, inv);
}
__device__ __forceinline__ void pivot_root(float d, float& root, float& inv) {
  root = sqrtf(d);
  inv = 1.0f / root;
}

// Block column k0: factor the diagonal block, solve the panel rows of this
// thread block, write both back and the panel's slices for the update.
// The factored diagonal block goes to `diag` (NB x NB per block column), not
// to A: other thread blocks of the same launch may still be reading it.
//
// Warps 0-3 eliminate the diagonal block (every thread block does so, none
// waits on another), warps 4-7 the same columns from 32 panel rows, one step
// behind; row per lane, column c in warp c % 4 of the group, so each group
// uses all four quarters of the SM: a FP64 instruction holds its quarter for
// about 64 clocks.  Column j of the diagonal block is published unscaled (x)
// and divided by the pivot (x / d): x_c -= x_j (x_cj / d_j) needs the
// reciprocal but no root, and the whole factor is scaled by 1/sqrt(d) at the
// end, all pivots at once.  In each step the owner of the next column updates
// it and publishes its pivot before the rest of the step's work; the warps
// wait for columns by flags in shared memory (bounded), not for each other.
// No FP64 comparisons: they cost as much as a multiply-add.
// Bound by 32 times that chain and the 300 instructions per quarter: 21 to 24 us
// (in stream order).  With the diagonal block in one warp and a root in every
// step the kernel took 40 us, with four warps and block barriers 29 us; with
// block-wide steps, roots and divisions and 64 rows per block 99-123 us.
template <class T, int NS>
__global__ void __launch_bounds__(256) k_panel(int n, int k0, double* __restrict__ A, int64_t lda,
                                              int* __restrict__ info, __nv_bfloat16* __restrict__ sl,
                                              int32_t* __restrict__ ex, int64_t Rpad, double* __restrict__ diag,
                                              int* __restrict__ err, int polls) {
  __shared__ T colx[NB][NB], coll[NB][NB];  // column j: x and x / d, by row
  __shared__ T yv[NB][ROWS];                // column j of the panel, unscaled
  __shared__ T piv[NB], rinv[NB], root[NB];
  __shared__ double xs[ROWS][NB + 1];
  __shared__ int bad_s, stuck_s, failed_s;
  __shared__ volatile int ready_d[NB], ready_y[NB];  // columns published
  // one thread looks whether an earlier block column failed: block 0 of this
  // launch may report a pivot meanwhile, and the block decides as one
  if (threadIdx.x == 0) failed_s = *(volatile int*)info;
  const int kb = min(NB, n - k0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, w = warp & 3;
  const bool dg = warp < 4;
  // panel rows exist only below a full diagonal block (k0 + NB < n)
  const int64_t R = (int64_t)blockIdx.x * ROWS + lane, i = (int64_t)k0 + NB + R;
  const bool own = kb == NB && i < n;
  constexpr int Q = NB / 4;
  T x[Q];  // columns 4 q + w
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int c = 4 * q + w;
    if (dg)
      x[q] = (lane < kb && c <= lane) ? (T)A[(k0 + lane) + (int64_t)(k0 + c) * lda] : (lane == c ? (T)1 : (T)0);
    else
      x[q] = own ? (T)A[i + (int64_t)(k0 + c) * lda] : (T)0;
  }
  if (threadIdx.x == 0) bad_s = stuck_s = 0;
  if (threadIdx.x < NB) ready_d[threadIdx.x] = ready_y[threadIdx.x] = 0;
  // a flag of a warp of this block (all are resident); a wait that runs out is
  // reported at the end, and the warps go on with what is there
  auto wait_for = [&](volatile int* flag) {
    int it = 0;
    while (!*flag && it < polls) ++it;
    if (it == polls && !*flag) stuck_s = 1;
    __threadfence_block();
    __syncwarp();
  };
  auto raise = [&](volatile int* flag) {
    __threadfence_block();
    __syncwarp();
    if (lane == 0) *flag = 1;
  };
  auto publish = [&](int j, T xj) {
    colx[j][lane] = xj;
    T d = __shfl_sync(0xffffffffu, xj, j);
    if (!pivot_ok(d)) {
      if (lane == 0 && bad_s == 0) bad_s = k0 + j + 1;  // columns come in order
      d = (T)1;  // the factor is not used
    }
    coll[j][lane] = fast_quotient(xj, d);
    if (lane == 0) piv[j] = d;
    raise(&ready_d[j]);
  };
  __syncthreads();
  if (failed_s) return;
  if (dg) {
    if (w == 0) publish(0, x[0]);
#pragma unroll
    for (int j = 0; j < NB - 1; ++j) {
      if (w != (j & 3)) wait_for(&ready_d[j]);
      const T xr = colx[j][lane];
      const int qn = (j + 1) >> 2;
      if (w == ((j + 1) & 3)) {
        x[qn] -= xr * coll[j][j + 1];
        publish(j + 1, x[qn]);
      }
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (4 * q + 3 > j + 1 && 4 * q + w > j + 1) x[q] -= xr * coll[j][4 * q + w];
    }
  } else {
#pragma unroll
    for (int p = 0; p < NB; ++p) {
      T yr = (T)0;
      if (p > 0) {
        wait_for(&ready_d[p - 1]);
        if (w != ((p - 1) & 3)) wait_for(&ready_y[p - 1]);
        yr = yv[p - 1][lane];
      }
      const int qp = p >> 2;
      if (w == (p & 3)) {
        if (p > 0) x[qp] -= yr * coll[p - 1][p];
        yv[p][lane] = x[qp];
        raise(&ready_y[p]);
      }
      if (p > 0) {
#pragma unroll
        for (int q = 0; q < Q; ++q)
          if (4 * q + 3 > p && 4 * q + w > p) x[q] -= yr * coll[p - 1][4 * q + w];
      }
    }
  }
  __syncthreads();
  if (stuck_s) {
    // from any block: its rows and slices are missing
    if (threadIdx.x == 0) {
      atomicExch(err, 6);
      atomicCAS(info, 0, k0 + 1);
    }
    return;
  }
  if (bad_s) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(info, 0, bad_s);
    return;
  }
  if (warp == 0) {
    T rt, ri;
    pivot_root(piv[lane], rt, ri);
    root[lane] = rt;
    rinv[lane] = ri;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int c = 4 * q + w;
    if (dg) {
      if (blockIdx.x == 0)
        diag[((int64_t)k0 + c) * NB + lane] =
            lane > c ? (double)(colx[c][lane] * rinv[c]) : (lane == c ? (double)root[c] : 0.0);
    } else {
      const double v = (double)(x[q] * rinv[c]);
      xs[lane][c] = v;
      if (own) A[i + (int64_t)(k0 + c) * lda] = v;
    }
  }
  __syncthreads();
  // row exponents, then slices: eight columns of one row per thread (four
  // neighbouring lanes share a row)
  if (threadIdx.x < 128) {
    const int row = threadIdx.x >> 2, seg = (threadIdx.x & 3) * 8;
    const int64_t Rr = (int64_t)blockIdx.x * ROWS + row;
    double v[8];
    int mx = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      v[c] = xs[row][seg + c];
      mx = max(mx, tcg::exp_field(v[c]));
    }
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    if (kb == NB && k0 + NB + Rr < n) {
      const int e = tcg::row_exp(mx);
      if (seg == 0) ex[Rr] = e;
      tcg::write_slices8<NS>(v, e, sl + Rr * NB + seg, Rpad * NB);
    }
  }
}

// After the last block column (the info check skips a failed factorization):
// the lower triangles of the factored diagonal blocks into A and, when dinv
// is given, their inverses.  One warp per block; lane c solves L x = e_c in
// registers (528 FP64 instructions, about 6 us).
__global__ void __launch_bounds__(32) k_diag_finish(int n, double* __restrict__ A, int64_t lda,
                                                   const double* __restrict__ diag, double* __restrict__ dinv,
                                                   const int* __restrict__ info) {
  if (*info != 0) return;
  __shared__ double Ls[NB][NB];  // Ls[c][r] = L(r, c)
  const int64_t k0 = (int64_t)blockIdx.x * NB;
  const int kb = (int)min((int64_t)NB, (int64_t)n - k0), lane = threadIdx.x;
#pragma unroll 8
  for (int c = 0; c < NB; ++c) {
    const double v = diag[(k0 + c) * NB + lane];
    Ls[c][lane] = v;
    if (lane >= c && lane < kb) A[(k0 + lane) + (k0 + c) * lda] = v;
  }
  if (!dinv) return;
  __syncwarp();
  const double rd = 1.0 / Ls[lane][lane];  // the padding is the identity
  double x[NB];
#pragma unroll
  for (int r = 0; r < NB; ++r) x[r] = r == lane ? 1.0 : 0.0;
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    x[k] *= __shfl_sync(0xffffffffu, rd, k);
#pragma unroll
    for (int r = k + 1; r < NB; ++r) x[r] = fma(-Ls[k][r], x[k], x[r]);
  }
#pragma unroll
  for (int r = 0; r < NB; ++r) dinv[(k0 + lane) * NB + r] = (r < kb && lane < kb) ? x[r] : 0.0;
}

// ---------------------------------------------------------------- triangular solves
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ unsigned long long gtime() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait for a phase of a barrier that a block of the cluster completes.
__device__ __forceinline__ bool cluster_wait(uint32_t bar, uint32_t parity, unsigned long long deadline) {
  for (uint32_t it = 0;; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, "
        "p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((it & 255u) == 255u && gtime() > deadline) return false;
  }
}

constexpr int kSolveThreads = 512;
constexpr int kSolveSmemMax = 220 * 1024;
constexpr unsigned long long kSolveWaitNs = 2000000000ull;

// Shared memory of a block: x (padded), partial sums of its blocks, two
// exchange buffers per warp group, one barrier per block row.
__host__ __device__ inline int64_t solve_smem(int nbk, int cs) {
  const int own = (nbk + cs - 1) / cs;
  return 8 * ((int64_t)nbk * NB + (int64_t)own * NB * NB + 4 * 2 * 4 * NB + nbk);
}

// x <- L^-T L^-1 x in one cluster.  Block rows of 32 go round the cluster's
// blocks.  Forward: as soon as y_b is known its owner writes it to every
// block's shared memory and signals barrier b there; every block subtracts
// L(B, b) y_b from its own later block rows B (a group of four warps per
// block row, eight columns a warp), the owner of b + 1 first.  Backward: the
// same with L(b, B)' (lanes along the rows of L, so that its columns are
// read in order; the sum over the lanes is taken when B's turn comes).  Bound
// by the FP64 pipes of the cluster's SMs (n^2 multiply-adds at 1.6 per clock
// and SM) and, per block row, by one exchange and two 32 x 32 products:
// 385 us at n = 2000 and 25 us at n = 100.  One block of 1024 threads
// alone took 1706 and 46 us.
// Every wait is bounded; a wait that runs out sets *err and the block goes on
// to the closing cluster barrier.
__global__ void __launch_bounds__(kSolveThreads) k_chol_solve(int n, const double* __restrict__ L, int64_t ld,
                                                             const double* __restrict__ dinv, double* __restrict__ x,
                                                             const int* __restrict__ info, int* __restrict__ err) {
  if (*info != 0) return;  // the same for every block of the cluster
  extern __shared__ double sm[];
  int cs, rank;
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(cs));
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int nbk = (n + NB - 1) / NB, own = (nbk + cs - 1) / cs;
  double* xv = sm;                                 // [nbk * NB]
  double* accs = xv + (int64_t)nbk * NB;           // [own][NB][NB]
  double* exch = accs + (int64_t)own * NB * NB;    // [4 groups][2][4][NB]
  unsigned long long* bars = (unsigned long long*)(exch + 4 * 2 * 4 * NB);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cg = warp & 3, grp = warp >> 2;        // eight columns; the group's block rows q = grp, grp + 4, ...
  double* ea = exch + grp * 2 * 4 * NB;
  double* eb = ea + 4 * NB;
  for (int t = threadIdx.x; t < nbk * NB; t += kSolveThreads) xv[t] = t < n ? x[t] : 0.0;
  for (int t = threadIdx.x; t < own * NB * NB; t += kSolveThreads) accs[t] = 0.0;
  for (int t = threadIdx.x; t < nbk; t += kSolveThreads)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bars + t)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
  const unsigned long long deadline = gtime() + kSolveWaitNs;
  bool ok = true;
  auto group_sync = [&] { asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory"); };
  // v (the right-hand side of block row b, in every warp of the group), then
  // x_b = D v (or D' v) to every block of the cluster, and its barrier
  auto finish = [&](int b, const double (&dreg)[8], double v) {
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
      s0 = fma(dreg[c], __shfl_sync(0xffffffffu, v, cg * 8 + c), s0);
      s1 = fma(dreg[c + 1], __shfl_sync(0xffffffffu, v, cg * 8 + c + 1), s1);
    }
    eb[cg * NB + lane] = s0 + s1;
    group_sync();
    const double y = (eb[lane] + eb[NB + lane]) + (eb[2 * NB + lane] + eb[3 * NB + lane]);
    const uint32_t dst = smem_u32(xv + (int64_t)b * NB + lane), bar = smem_u32(bars + b);
    for (int r = cg; r < cs; r += 4)
      asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(cluster_addr(dst, r)), "d"(y) : "memory");
    asm volatile("fence.acq_rel.cluster;" ::: "memory");
    __syncwarp();
    if (lane == 0)
      for (int r = cg; r < cs; r += 4)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr(bar, r))
                     : "memory");
  };
  // ---- forward: L y = x
  for (int b = -1; b < nbk - 1; ++b) {
    // the group's part of the next block row, before y_b is there
    const int nxt = b + 1, q0 = nxt / cs;
    const bool critical = nxt % cs == rank && (q0 & 3) == grp;
    double dreg[8], lreg[8];
    if (critical) {
      const bool rok = nxt * NB + lane < n;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        dreg[c] = dinv[((int64_t)nxt * NB + cg * 8 + c) * NB + lane];
        lreg[c] = (b >= 0 && rok) ? L[(int64_t)nxt * NB + lane + ((int64_t)b * NB + cg * 8 + c) * ld] : 0.0;
      }
    }
    if (b >= 0) ok = ok && cluster_wait(smem_u32(bars + b), 0, deadline);
    const double* yb = xv + (int64_t)(b < 0 ? 0 : b) * NB + cg * 8;
    if (critical) {
      double s0 = accs[(q0 * 4 + cg) * NB + lane], s1 = 0.0;
#pragma unroll
      for (int c = 0; c < 8; c += 2) {
        s0 = fma(lreg[c], yb[c], s0);
        s1 = fma(lreg[c + 1], yb[c + 1], s1);
      }
      ea[cg * NB + lane] = s0 + s1;
      group_sync();
      const double sum = (ea[lane] + ea[NB + lane]) + (ea[2 * NB + lane] + ea[3 * NB + lane]);
      finish(nxt, dreg, xv[(int64_t)nxt * NB + lane] - sum);
      accs[(q0 * 4 + cg) * NB + lane] = 0.0;
    }
    if (b >= 0) {
      for (int q = grp; q < own; q += 4) {
        const int Bq = q * cs + rank;
        if (Bq <= b + 1 || Bq >= nbk) continue;
        const int64_t row = (int64_t)Bq * NB + lane;
        if (row < n) {
          const double* Lr = L + row + ((int64_t)b * NB + cg * 8) * ld;
          double s0 = accs[(q * 4 + cg) * NB + lane], s1 = 0.0;
#pragma unroll
          for (int c = 0; c < 8; c += 2) {
            s0 = fma(Lr[c * ld], yb[c], s0);
            s1 = fma(Lr[(c + 1) * ld], yb[c + 1], s1);
          }
          accs[(q * 4 + cg) * NB + lane] = s0 + s1;
        }
      }
    }
  }
  ok = ok && cluster_wait(smem_u32(bars + nbk - 1), 0, deadline);
  // every y has arrived everywhere before any z overwrites it
  __syncthreads();
  for (int t = threadIdx.x; t < own * NB * NB; t += kSolveThreads) accs[t] = 0.0;
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
  // ---- backward: L' z = y
  for (int b = nbk; b > 0; --b) {
    const int nxt = b - 1, q0 = nxt / cs;
    const bool critical = nxt % cs == rank && (q0 & 3) == grp;
    double dreg[8], lreg[8];
    if (critical) {
      const bool rok = b < nbk && b * NB + lane < n;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        dreg[c] = dinv[((int64_t)nxt * NB + lane) * NB + cg * 8 + c];
        lreg[c] = rok ? L[(int64_t)b * NB + lane + ((int64_t)nxt * NB + cg * 8 + c) * ld] : 0.0;
      }
    }
    if (b < nbk) ok = ok && cluster_wait(smem_u32(bars + b), 1, deadline);
    const double zb = b < nbk ? xv[(int64_t)b * NB + lane] : 0.0;
    if (critical) {
      // the eight columns' sums over the lanes: written out, then column
      // `lane` added up, eight lanes' terms per warp
      double* ac = accs + ((int64_t)q0 * NB + cg * 8) * NB;
#pragma unroll
      for (int c = 0; c < 8; ++c) ac[c * NB + lane] = fma(lreg[c], zb, ac[c * NB + lane]);
      group_sync();
      const double* col = accs + ((int64_t)q0 * NB + lane) * NB;
      double s0 = 0.0, s1 = 0.0;
#pragma unroll
      for (int t = 0; t < 8; t += 2) {
        // rotated by the column so that the lanes read different banks
        s0 += col[cg * 8 + ((t + lane) & 7)];
        s1 += col[cg * 8 + ((t + 1 + lane) & 7)];
      }
      ea[cg * NB + lane] = s0 + s1;
      group_sync();
      const double sum = (ea[lane] + ea[NB + lane]) + (ea[2 * NB + lane] + ea[3 * NB + lane]);
      finish(nxt, dreg, xv[(int64_t)nxt * NB + lane] - sum);
    }
    if (b < nbk) {
      const bool rok = b * NB + lane < n;
      for (int q = grp; q < own; q += 4) {
        const int Bq = q * cs + rank;
        if (Bq >= b - 1) continue;
        if (rok) {
          const double* Lc = L + (int64_t)b * NB + lane + ((int64_t)Bq * NB + cg * 8) * ld;
          double* ac = accs + ((int64_t)q * NB + cg * 8) * NB;
#pragma unroll
          for (int c = 0; c < 8; ++c) ac[c * NB + lane] = fma(Lc[c * ld], zb, ac[c * NB + lane]);
        }
      }
    }
  }
  ok = ok && cluster_wait(smem_u32(bars), 1, deadline);
  if (!ok) atomicExch(err, 5);
  __syncthreads();
  for (int t = rank * kSolveThreads + threadIdx.x; t < n; t += cs * kSolveThreads) x[t] = ok ? xv[t] : nan("");
  // no block leaves while another may still write to its shared memory
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The same in one thread block of 1024 threads, for orders (above 8500) whose
// vectors do not fit the cluster's shared memory: block row by block row, the sums over
// the solved part read NB consecutive entries per column (coalesced), four
// independent accumulators per thread.
__global__ void __launch_bounds__(1024) k_chol_solve_block(int n, const double* __restrict__ L, int64_t ld,
                                                     const double* __restrict__ dinv, double* x,
                                                     const int* __restrict__ info) {
  if (*info != 0) return;
  __shared__ double red[32][33];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int nbk = (n + NB - 1) / NB;
  // forward: L y = x
  for (int b = 0; b < nbk; ++b) {
    const int r0 = b * NB, rows = min(NB, n - r0);
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    if (lane < rows) {
      const double* Lr = L + r0 + lane;
      int c = w;
      for (; c + 96 < r0; c += 128) {
        a0 = fma(Lr[(int64_t)c * ld], x[c], a0);
        a1 = fma(Lr[(int64_t)(c + 32) * ld], x[c + 32], a1);
        a2 = fma(Lr[(int64_t)(c + 64) * ld], x[c + 64], a2);
        a3 = fma(Lr[(int64_t)(c + 96) * ld], x[c + 96], a3);
      }
      for (; c < r0; c += 32) a0 = fma(Lr[(int64_t)c * ld], x[c], a0);
    }
    red[w][lane] = (a0 + a1) + (a2 + a3);
    __syncthreads();
    if (w == 0) {
      double sum = 0.0;
      for (int g = 0; g < 32; ++g) sum += red[g][lane];
      const double v = lane < rows ? x[r0 + lane] - sum : 0.0;
      const double* Di = dinv + (int64_t)b * NB * NB;
      double y = 0.0;
      for (int c = 0; c < NB; ++c) y = fma(Di[lane + c * NB], __shfl_sync(0xffffffffu, v, c), y);
      if (lane < rows) x[r0 + lane] = y;
    }
    __syncthreads();
  }
  // backward: L' z = y
  for (int b = nbk - 1; b >= 0; --b) {
    const int r0 = b * NB, rows = min(NB, n - r0);
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    if (w < rows) {
      const double* Lc = L + (int64_t)(r0 + w) * ld;
      int j = r0 + NB + lane;
      for (; j + 96 < n; j += 128) {
        a0 = fma(Lc[j], x[j], a0);
        a1 = fma(Lc[j + 32], x[j + 32], a1);
        a2 = fma(Lc[j + 64], x[j + 64], a2);
        a3 = fma(Lc[j + 96], x[j + 96], a3);
      }
      for (; j < n; j += 32) a0 = fma(Lc[j], x[j], a0);
    }
    double a = (a0 + a1) + (a2 + a3);
    for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) red[0][w] = a;
    __syncthreads();
    if (w == 0) {
      const double v = lane < rows ? x[r0 + lane] - red[0][lane] : 0.0;
      const double* Di = dinv + (int64_t)b * NB * NB;
      double y = 0.0;
      for (int c = 0; c < NB; ++c) y = fma(Di[c + lane * NB], __shfl_sync(0xffffffffu, v, c), y);
      if (lane < rows) x[r0 + lane] = y;
    }
    __syncthreads();
  }
}

int64_t panel_bytes(int64_t nmax) { return tcg::sliced_bytes(nmax, NB, 7); }

}  // namespace

int64_t work_bytes(int64_t nmax) {
  nmax = std::max<int64_t>(nmax, 1);
  return panel_bytes(nmax) + 2 * (nmax + NB) * NB * 8;
}

cudaError_t init(Work* w, void* mem, int64_t nmax, int* err, cudaStream_t st, bool solves) {
  w->mem = mem;
  w->solves = solves;
  w->nmax = std::max<int64_t>(nmax, 1);
  w->err = err;
  w->diag = (double*)((char*)mem + panel_bytes(w->nmax));
  w->dinv = w->diag + (w->nmax + NB) * NB;
  return tcg::sliced_init(&w->panel, mem, w->nmax, NB, 7, st);
}

cudaError_t solve(const Work& w, int n, const double* L, int64_t ld, double* x, const int* info, cudaStream_t st,
                  int64_t* launches) {
  if (n <= 0) return cudaSuccess;
  if (n > w.nmax || !w.solves) return cudaErrorInvalidValue;
  // 16 blocks (more than the portable 8) from 9 block rows on: the work is
  // FP64-pipe bound, n^2 multiply-adds at 1.6 per clock and SM
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  static bool wide = false;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(k_chol_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, kSolveSmemMax);
    wide = cudaFuncSetAttribute(k_chol_solve, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    cudaGetLastError();
  });
  if (attr != cudaSuccess) return attr;
  const int nbk = (n + NB - 1) / NB;
  int cs = 1;
  while (cs < nbk && cs < (wide ? 16 : 8)) cs *= 2;
  if (solve_smem(nbk, cs) > kSolveSmemMax) {
    k_chol_solve_block<<<1, 1024, 0, st>>>(n, L, ld, w.dinv, x, info);
    if (launches) *launches += 1;
    return cudaGetLastError();
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)cs);
  cfg.blockDim = dim3(kSolveThreads);
  cfg.dynamicSmemBytes = (size_t)solve_smem(nbk, cs);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cs;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_chol_solve, n, L, ld, (const double*)w.dinv, x, info, w.err);
  if (launches) *launches += 1;
  return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t potrf(Work& w, int n, double* A, int64_t lda, int* info, tcg::Mode mode, cudaStream_t st,
                  int64_t* launches) {
  if (n < 0 || n > w.nmax || lda < std::max(n, 1)) return cudaErrorInvalidValue;
  const int ns = tcg::slices_of(mode);
  cudaError_t e = cudaSuccess;
  if (w.panel.ns != ns) {
    e = tcg::sliced_init(&w.panel, w.mem, w.nmax, NB, ns, st, false);
    if (e != cudaSuccess) return e;
  }
  e = cudaMemsetAsync(info, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  for (int k0 = 0; k0 < n; k0 += NB) {
    const int kb = std::min(NB, n - k0);
    const int64_t nr = n - k0 - kb;
    const unsigned grid = (unsigned)std::max<int64_t>(1, (nr + ROWS - 1) / ROWS);
    if (mode == tcg::kMixed)
      k_panel<float, 3><<<grid, 256, 0, st>>>(n, k0, A, lda, info, w.panel.s, w.panel.ex, w.panel.Rpad, w.diag,
                                                 w.err, w.polls);
    else
      k_panel<double, 7><<<grid, 256, 0, st>>>(n, k0, A, lda, info, w.panel.s, w.panel.ex, w.panel.Rpad, w.diag,
                                                 w.err, w.polls);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (launches) *launches += 1;
    if (nr > 0) {
      w.panel.rows = nr;
      tcg::Out o;
      o.C = A + (k0 + kb) + (int64_t)(k0 + kb) * lda;
      o.ldc = lda;
      o.alpha = -1.0;
      o.beta = 1.0;
      o.lower = true;
      o.err = w.err;
      e = tcg::gemm(w.panel, w.panel, mode, o, st, launches);
      if (e != cudaSuccess) return e;
    }
  }
  if (n > 0) {
    k_diag_finish<<<(unsigned)((n + NB - 1) / NB), 32, 0, st>>>(n, A, lda, w.diag, w.solves ? w.dinv : nullptr, info);
    if (launches) *launches += 1;
    e = cudaGetLastError();
  }
  return e;
}

}  // namespace chol

// ---------------------------------------------------------------- C ABI
// DenseCholesky's factorize! (src/schur_solvers.jl:15-19) for one dense
// matrix on the device (include/madsdp_gpu.h).
#include "../../include/madsdp_gpu.h"

extern "C" int msdp_dense_cholesky(int32_t precision, int32_t n, double* A, int64_t lda, int32_t* info,
                                   void* stream) {
  if (n < 0 || !info || (n && !A) || lda < std::max(n, 1)) return MSDP_ERR_INVALID_ARGUMENT;
  if (precision != MSDP_FP64 && precision != MSDP_MIXED) return MSDP_ERR_INVALID_ARGUMENT;
  *info = 0;
  if (n == 0) return MSDP_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t wb = chol::work_bytes(n);
  char* mem = nullptr;
  if (cudaMalloc(&mem, (size_t)(wb + 512)) != cudaSuccess) return MSDP_ERR_OUT_OF_MEMORY;
  int* dinfo = (int*)(mem + wb);
  int* derr = dinfo + 1;
  chol::Work w;
  cudaError_t e = cudaMemsetAsync(derr, 0, sizeof(int), st);
  if (e == cudaSuccess) e = chol::init(&w, mem, n, derr, st, false);
  if (e == cudaSuccess)
    e = chol::potrf(w, n, A, lda, dinfo, precision == MSDP_MIXED ? tcg::kMixed : tcg::kFp64, st, nullptr);
  int h[2] = {0, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, dinfo, 2 * sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFree(mem);
  if (e != cudaSuccess || h[1]) return MSDP_ERR_CUDA;
  *info = h[0];
  return MSDP_OK;
}
