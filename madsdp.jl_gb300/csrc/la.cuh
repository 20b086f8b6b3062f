// CTA-cooperative dense linear algebra for the per-problem IPM kernel.
//
// Every routine is called by all NTHREADS threads of one CTA and ends with a
// __syncthreads(), so results are visible to the whole CTA on return.
// Matrices are column-major with leading dimension n (A(i,j) = A[i + j*n]);
// pointers may address global or shared memory (generic addressing).
// T is the compute type (double for the FP64 path, float for the FP32
// phase of the mixed path).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "scalar.cuh"
#include "tridiag.cuh"

#ifndef NTHREADS
#define NTHREADS 128
#endif
#define NWARPS (NTHREADS / 32)

template <class T> struct Num;
template <> struct Num<double> {
  static __device__ __forceinline__ double eps() { return 2.220446049250313e-16; }
  static __device__ __forceinline__ double sqrt_(double x) { return sqrt(x); }
  static __device__ __forceinline__ double rsqrt_(double x) { return rsqrt(x); }
  static __device__ __forceinline__ bool finite(double x) { return isfinite(x); }
};
template <> struct Num<float> {
  static __device__ __forceinline__ float eps() { return 1.1920928955078125e-7f; }
  static __device__ __forceinline__ float sqrt_(float x) { return sqrtf(x); }
  static __device__ __forceinline__ float rsqrt_(float x) { return rsqrtf(x); }
  static __device__ __forceinline__ bool finite(float x) { return isfinite(x); }
};

// ---------------------------------------------------------------- reductions
template <class T> __device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <class T> __device__ __forceinline__ T warp_max(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Scratch for block reductions (NWARPS doubles + result).
struct RedBuf { double v[NWARPS + 1]; };

__device__ __forceinline__ double block_sum(double v, RedBuf* rb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum(v);
  if (lane == 0) rb->v[warp] = v;
  __syncthreads();
  if (warp == 0) {
    double r = lane < NWARPS ? rb->v[lane] : 0.0;
    r = warp_sum(r);
    if (lane == 0) rb->v[NWARPS] = r;
  }
  __syncthreads();
  double r = rb->v[NWARPS];
  __syncthreads();
  return r;
}

__device__ __forceinline__ double block_max(double v, RedBuf* rb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_max(v);
  if (lane == 0) rb->v[warp] = v;
  __syncthreads();
  if (warp == 0) {
    double r = lane < NWARPS ? rb->v[lane] : -INFINITY;
    r = warp_max(r);
    if (lane == 0) rb->v[NWARPS] = r;
  }
  __syncthreads();
  double r = rb->v[NWARPS];
  __syncthreads();
  return r;
}

// ---------------------------------------------------------------- elementwise
template <class T, class U>
__device__ void cta_convert(int64_t len, T* __restrict__ dst, const U* __restrict__ src) {
  for (int64_t k = threadIdx.x; k < len; k += NTHREADS) dst[k] = (T)src[k];
  __syncthreads();
}
template <class T> __device__ void cta_fill(int64_t len, T* dst, T v) {
  for (int64_t k = threadIdx.x; k < len; k += NTHREADS) dst[k] = v;
  __syncthreads();
}
// A = (A + A') / 2 in place (src/blocks.jl:77-84).  Each unordered pair is
// owned by one thread.
template <class T> __device__ void cta_symmetrize(int n, T* A) {
  const int64_t nn = (int64_t)n * n;
  for (int64_t k = threadIdx.x; k < nn; k += NTHREADS) {
    int i = (int)(k % n), j = (int)(k / n);
    if (i > j) {
      T v = (A[i + (int64_t)j * n] + A[j + (int64_t)i * n]) / (T)2;
      A[i + (int64_t)j * n] = v;
      A[j + (int64_t)i * n] = v;
    }
  }
  __syncthreads();
}
// Upper triangle := lower triangle (after a lower-only symmetric product).
template <class T> __device__ void cta_lower_to_full(int n, T* A) {
  const int64_t nn = (int64_t)n * n;
  for (int64_t k = threadIdx.x; k < nn; k += NTHREADS) {
    const int i = (int)(k % n), j = (int)(k / n);
    if (i < j) A[k] = A[j + (int64_t)i * n];
  }
  __syncthreads();
}
// dst = sym(src) into another buffer.
template <class T, class U> __device__ void cta_sym_copy(int n, T* dst, const U* src) {
  const int64_t nn = (int64_t)n * n;
  for (int64_t k = threadIdx.x; k < nn; k += NTHREADS) {
    int i = (int)(k % n), j = (int)(k / n);
    dst[k] = (T)((src[i + (int64_t)j * n] + src[j + (int64_t)i * n]) / (U)2);
  }
  __syncthreads();
}
template <class T> __device__ void cta_set_identity(int n, T* A, T diag) {
  const int64_t nn = (int64_t)n * n;
  for (int64_t k = threadIdx.x; k < nn; k += NTHREADS) A[k] = ((k % n) == (k / n)) ? diag : (T)0;
  __syncthreads();
}

// (j, k) with j >= k of the idx-th entry of a packed lower triangle (row
// major); the root only has to be near, the loops make it exact.
__device__ __forceinline__ void tri_index(int64_t idx, int& j, int& k) {
  int r = (int)((sqrtf(8.0f * (float)idx + 1.0f) - 1.0f) * 0.5f);
  while ((int64_t)(r + 1) * (r + 2) / 2 <= idx) ++r;
  while ((int64_t)r * (r + 1) / 2 > idx) --r;
  j = r;
  k = (int)(idx - (int64_t)r * (r + 1) / 2);
}

// ---------------------------------------------------------------- GEMM
// C = alpha * op(A) * op(B) + beta * C for n x n matrices.  ta/tb: 0 = as
// stored, 1 = transposed.  loA/loB: the stored operand is lower triangular
// (its upper triangle is zero), which restricts the k range.  C must not
// alias A or B.  Each thread owns R x R output micro-tiles.
template <class T, int R>
__device__ void cta_gemm_r(int n, int ta, int tb, int loA, int loB, T alpha, const T* __restrict__ A,
                           const T* __restrict__ B, T beta, T* __restrict__ C, int loC, int ldc) {
  const int nb = (n + R - 1) / R;
  const int tiles = loC ? nb * (nb + 1) / 2 : nb * nb;
  const bool unit = alpha == (T)1, zero = beta == (T)0;
  for (int t = threadIdx.x; t < tiles; t += NTHREADS) {
    int ti, tj;
    if (loC) {
      tri_index(t, ti, tj);  // only tiles touching the lower triangle
    } else {
      tj = t / nb;
      ti = t - tj * nb;
    }
    const int i0 = ti * R, j0 = tj * R;
    int klo = 0, khi = n;  // k in [klo, khi)
    if (loA) {
      if (!ta) khi = min(khi, i0 + R);  // A(i,k) != 0 -> k <= i
      else klo = max(klo, i0);          // A(k,i) != 0 -> k >= i
    }
    if (loB) {
      if (!tb) klo = max(klo, j0);      // B(k,j) != 0 -> k >= j
      else khi = min(khi, j0 + R);      // B(j,k) != 0 -> k <= j
    }
    T acc[R][R];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < R; ++c) acc[r][c] = (T)0;
    for (int k = klo; k < khi; ++k) {
      T a[R], b[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = i0 + r;
        a[r] = (i < n) ? (ta ? A[k + (int64_t)i * n] : A[i + (int64_t)k * n]) : (T)0;
      }
#pragma unroll
      for (int c = 0; c < R; ++c) {
        const int j = j0 + c;
        b[c] = (j < n) ? (tb ? B[j + (int64_t)k * n] : B[k + (int64_t)j * n]) : (T)0;
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < R; ++c) acc[r][c] = fma(a[r], b[c], acc[r][c]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < R; ++c) {
        const int i = i0 + r, j = j0 + c;
        if (i < n && j < n) {
          const int64_t o = i + (int64_t)j * ldc;
          const T v = unit ? acc[r][c] : alpha * acc[r][c];
          C[o] = zero ? v : fma(alpha, acc[r][c], beta * C[o]);
        }
      }
  }
  __syncthreads();
}

// Tile sizes.  float: 4 x 4 above n = 24 (shared-memory reads bound it).
// double: 2 x 2, because a FP64 multiply-add holds its quarter of the SM for
// 64 clocks and the last round of 4 x 4 tiles leaves many lanes idle (n = 50:
// 169 tiles of 16 on 128 threads take 32 multiply-adds a k, 2 x 2 tiles 20).
template <class T>
__device__ __forceinline__ void cta_gemm_plain(int n, int ta, int tb, int loA, int loB, T alpha, const T* A,
                                               const T* B, T beta, T* C, int loC, int ldc) {
  if (sizeof(T) == 8 || n <= 24) cta_gemm_r<T, 2>(n, ta, tb, loA, loB, alpha, A, B, beta, C, loC, ldc);
  else cta_gemm_r<T, 4>(n, ta, tb, loA, loB, alpha, A, B, beta, C, loC, ldc);
}

// Shared-memory scratch handed to the routines that stage operands
// (nullptr / 0 bytes: operate in global memory).
struct Scratch {
  unsigned char* p;
  int64_t bytes;
};

// GEMM whose operands are first copied into shared memory when they fit
// (operands written earlier by this CTA would otherwise be re-read from L2).
// loC = 1: only the lower triangle of C is needed (a symmetric product);
// tiles strictly above the diagonal are skipped.
template <class T>
__device__ void cta_gemm(int n, int ta, int tb, int loA, int loB, T alpha, const T* A, const T* B, T beta, T* C,
                         Scratch sc, int loC = 0, int ldc = 0) {
  if (ldc == 0) ldc = n;  // column stride of C
  const int64_t nn = (int64_t)n * n;
  const int64_t need = (A == B ? 1 : 2) * nn * (int64_t)sizeof(T);
  if (sc.p != nullptr && need <= sc.bytes) {
    T* sA = (T*)sc.p;
    T* sB = (A == B) ? sA : sA + nn;
    for (int64_t k = threadIdx.x; k < nn; k += NTHREADS) {
      sA[k] = A[k];
      if (A != B) sB[k] = B[k];
    }
    __syncthreads();
    cta_gemm_plain<T>(n, ta, tb, loA, loB, alpha, sA, sB, beta, C, loC, ldc);
  } else {
    cta_gemm_plain<T>(n, ta, tb, loA, loB, alpha, A, B, beta, C, loC, ldc);
  }
}

// ---------------------------------------------------------------- Cholesky
// In-place lower Cholesky of the n x n matrix `a` (leading dimension lda);
// only the lower triangle is read.  Returns false (on every thread) if a
// pivot is not positive and finite, as LAPACK potrf (src/blocks.jl:94-100,
// src/schur_solvers.jl:15-19).  `flag` is a shared int.
//
// Eight columns at a time: warp 0 factors the 8 x 8 diagonal block in
// registers, a thread per row solves the panel below, then 4 x 4 (float) or
// 2 x 2 (double) tiles of the trailing triangle take all eight columns'
// update.  Every entry sees the same operations in the same order as column
// by column (multiply-adds by ascending column, then the multiplication by
// the reciprocal pivot).  Three barriers per eight columns instead of 24, and
// no index divisions over the whole square: the double Schur factorizations
// of a three-iteration slice took 11 million clocks at m = 127, now 2.7.
template <class T> __device__ __forceinline__ void chol_pivot(T d, T& root, T& inv) {
  root = Num<T>::sqrt_(d);
  inv = (T)1 / root;
}
template <> __device__ __forceinline__ void chol_pivot<float>(float d, float& root, float& inv) {
  root = sqrtf(d);
  inv = 1.0f / root;
}
template <> __device__ __forceinline__ void chol_pivot<double>(double d, double& root, double& inv) {
  exact_root(d, root, inv);
}
template <class T>
__device__ __forceinline__ bool pivot_ok(T d) {
  return d > (T)0 && Num<T>::finite(d);
}
// x of lane `src`, for any T of whole 32-bit words
template <class T>
__device__ __forceinline__ T lane_value(T x, int src) {
  static_assert(sizeof(T) % 4 == 0, "whole words");
  unsigned w[sizeof(T) / 4];
  memcpy(w, &x, sizeof(T));
#pragma unroll
  for (int k = 0; k < (int)(sizeof(T) / 4); ++k) w[k] = __shfl_sync(0xffffffffu, w[k], src);
  memcpy(&x, w, sizeof(T));
  return x;
}
template <class T>
__device__ bool cta_potrf(int n, T* a, int lda, int* flag) {
  constexpr int KB = 8, R = sizeof(T) == 8 ? 2 : 4;
  __shared__ T L11[KB][KB], rinv[KB];  // L11[k][c] = L(c, k)
  if (threadIdx.x == 0) *flag = 0;
  __syncthreads();
  for (int k0 = 0; k0 < n; k0 += KB) {
    const int kb = min(KB, n - k0);
    if (threadIdx.x < 32) {
      const int r = threadIdx.x;
      T x[KB];
#pragma unroll
      for (int c = 0; c < KB; ++c)
        x[c] = (r < kb && c <= r) ? a[(k0 + r) + (int64_t)(k0 + c) * lda] : (r == c ? (T)1 : (T)0);
      bool bad = false;
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        T d = lane_value(x[k], k);
        if (!pivot_ok(d)) {
          bad = true;
          d = (T)1;
        }
        T root, inv;
        chol_pivot<T>(d, root, inv);
        const T l = r == k ? root : x[k] * inv;
        x[k] = l;
        if (r < KB) L11[k][r] = l;
        if (r == k) rinv[k] = inv;
#pragma unroll
        for (int c = k + 1; c < KB; ++c) x[c] = fma(-l, lane_value(l, c), x[c]);
      }
      if (bad) *flag = 1;
#pragma unroll
      for (int c = 0; c < KB; ++c)
        if (r < kb && c <= r) a[(k0 + r) + (int64_t)(k0 + c) * lda] = x[c];
    }
    __syncthreads();
    if (*flag) return false;
    const int m0 = k0 + kb, m = n - m0;
    if (m <= 0) break;
    for (int i = m0 + threadIdx.x; i < n; i += NTHREADS) {
      T x[KB];
#pragma unroll
      for (int c = 0; c < KB; ++c) x[c] = a[i + (int64_t)(k0 + c) * lda];
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        x[k] *= rinv[k];
#pragma unroll
        for (int c = k + 1; c < KB; ++c) x[c] = fma(-x[k], L11[k][c], x[c]);
      }
#pragma unroll
      for (int c = 0; c < KB; ++c) a[i + (int64_t)(k0 + c) * lda] = x[c];
    }
    __syncthreads();
    const int nb = (m + R - 1) / R, tiles = nb * (nb + 1) / 2;
    const T* P = a + m0 + (int64_t)k0 * lda;  // panel rows
    for (int t = threadIdx.x; t < tiles; t += NTHREADS) {
      int ti, tj;
      tri_index(t, ti, tj);
      const int i0 = ti * R, j0 = tj * R;
      T acc[R][R];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < R; ++c)
          acc[r][c] = (i0 + r < m && j0 + c <= i0 + r) ? a[(m0 + i0 + r) + (int64_t)(m0 + j0 + c) * lda] : (T)0;
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        T li[R], lj[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          li[r] = i0 + r < m ? P[i0 + r + (int64_t)k * lda] : (T)0;
          lj[r] = j0 + r < m ? P[j0 + r + (int64_t)k * lda] : (T)0;
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = 0; c < R; ++c) acc[r][c] = fma(-li[r], lj[c], acc[r][c]);
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < R; ++c)
          if (i0 + r < m && j0 + c <= i0 + r) a[(m0 + i0 + r) + (int64_t)(m0 + j0 + c) * lda] = acc[r][c];
    }
    __syncthreads();
  }
  return true;
}

// Zero the strict upper triangle and flush the entries below
// eps^2 * max |L_ii| (src/blocks.jl:101-111).  Works on any leading dim.
template <class T>
__device__ void cta_flush_lower(int n, T* L, int lda, RedBuf* rb) {
  double dmax = 0.0;
  for (int i = threadIdx.x; i < n; i += NTHREADS) dmax = fmax(dmax, fabs((double)L[i + (int64_t)i * lda]));
  dmax = block_max(dmax, rb);
  const T tol = (T)((double)Num<T>::eps() * (double)Num<T>::eps() * dmax);
  const int64_t nn = (int64_t)n * n;
  for (int64_t k = threadIdx.x; k < nn; k += NTHREADS) {
    const int i = (int)(k % n), j = (int)(k / n);
    T* p = L + i + (int64_t)j * lda;
    if (i < j) *p = (T)0;
    else if (i > j && fabs(*p) < tol) *p = (T)0;
  }
  __syncthreads();
}

// Inverse of a lower-triangular L (ld = n) into Li (ld = n, lower, upper
// zeroed).  One thread per column; Li may live in shared memory.
template <class T>
__device__ void cta_trtri_lower(int n, const T* __restrict__ L, T* __restrict__ Li) {
  for (int j = threadIdx.x; j < n; j += NTHREADS) {
    T* x = Li + (int64_t)j * n;
    for (int i = 0; i < j; ++i) x[i] = (T)0;
    x[j] = (T)1 / L[j + (int64_t)j * n];
    for (int i = j + 1; i < n; ++i) {
      T s = (T)0;
      for (int k = j; k < i; ++k) s = fma(L[i + (int64_t)k * n], x[k], s);
      x[i] = -s / L[i + (int64_t)i * n];
    }
  }
  __syncthreads();
}

// Solve L L' x = b in place (L lower, ld = n), b of length n.
template <class T, class V>
__device__ void cta_potrs(int n, const T* __restrict__ L, V* x) {
  // forward: L u = b (column oriented)
  for (int k = 0; k < n; ++k) {
    if (threadIdx.x == 0) x[k] = x[k] / (V)L[k + (int64_t)k * n];
    __syncthreads();
    const V xk = x[k];
    for (int i = k + 1 + threadIdx.x; i < n; i += NTHREADS) x[i] -= (V)L[i + (int64_t)k * n] * xk;
    __syncthreads();
  }
  // backward: L' x = u (row of L' = column of L: dot products)
  for (int k = n - 1; k >= 0; --k) {
    // x[k] = (x[k] - sum_{i>k} L(i,k) x[i]) / L(k,k)
    V s = 0;
    for (int i = k + 1 + threadIdx.x; i < n; i += NTHREADS) s += (V)L[i + (int64_t)k * n] * x[i];
    s = warp_sum(s);
    __shared__ V part[NWARPS];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      V t = 0;
      for (int w = 0; w < NWARPS; ++w) t += part[w];
      x[k] = (x[k] - t) / (V)L[k + (int64_t)k * n];
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- Jacobi SVD
// One-sided (Hestenes) Jacobi on the columns of M (n x n, ld n): on return
// M V has mutually orthogonal columns and sigma[k] is the norm of column k.
// The eigenvalues of M'M are sigma^2 with eigenvectors V, which is what
// LowRankOpt.eigen! returns for the NT scaling (src/directions.jl:52-58).
// Every rotation is also applied to the columns of B (n x n): B = I gives
// V itself, B = Lx gives Lx V directly.  Parallel round-robin ordering.
// Returns false if it did not converge in max_sweeps.
//
// The float version: eight lanes per column pair, each standing for V = 1, 2
// or 4 lanes (n <= 16, <= 48, above) of a group of 8 V whose butterfly it
// reproduces: lane gl keeps the partial sums of the virtual lanes gl + 8 v, adds
// them in the order of the butterfly's upper levels and shuffles for the last
// three.  So the results are those of groups of 8 V lanes, bit for bit, but a
// warp has four pairs in flight instead of 4 / V and nine shuffles instead of
// up to fifteen on the critical path of each (a shuffle is about 75 clocks).
template <int V, class T>
__device__ __forceinline__ T virtual_sum(T (&s)[V]) {
  if (V == 4) {
    s[0] += s[2 % V];
    s[1 % V] += s[3 % V];
  }
  if (V >= 2) s[0] += s[1 % V];
  T r = s[0];
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return r;
}
template <int V, bool VECS = true>
__device__ bool cta_jacobi_svd_f32(int n, int ld, float* M, float* B, float* sigma, int max_sweeps, int* sweeps_out) {
  constexpr int G = 8, NG = NTHREADS / G;
  const int gl = threadIdx.x & (G - 1), group = threadIdx.x / G;
  const int N = (n % 2 == 0) ? n : n + 1;
  const float tol = (float)sqrt((double)n) * Num<float>::eps(), big_tol = sqrtf(tol);
  const int slots = (N / 2 + NG - 1) / NG;  // the same for every group: shuffles stay uniform
  bool converged = (n <= 1);
  int sweep = 0;
  for (; sweep < max_sweeps && !converged; ++sweep) {
    int rotated = 0, big = 0;
    for (int r = 0; r < N - 1; ++r) {
      for (int sidx = 0; sidx < slots; ++sidx) {
        const int k = group + sidx * NG;
        int p = -1, q = -1;
        if (k < N / 2) {
          if (k == 0) {
            p = N - 1;
            q = r;
          } else {
            p = r + k < N - 1 ? r + k : r + k - (N - 1);
            q = r - k >= 0 ? r - k : r - k + (N - 1);
          }
          if (p >= n || q >= n) p = q = -1;
        }
        float* mp = M + (int64_t)(p < 0 ? 0 : p) * ld;
        float* mq = M + (int64_t)(p < 0 ? 0 : q) * ld;
        float spp[V], sqq[V], spq[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          spp[v] = sqq[v] = spq[v] = 0.0f;
          if (p >= 0)
            for (int i = gl + G * v; i < n; i += G * V) {
              const float a = mp[i], b = mq[i];
              spp[v] = fmaf(a, a, spp[v]);
              sqq[v] = fmaf(b, b, sqq[v]);
              spq[v] = fmaf(a, b, spq[v]);
            }
        }
        const float app = virtual_sum<V>(spp), aqq = virtual_sum<V>(sqq), apq = virtual_sum<V>(spq);
        const float scale_pq = sqrtf(app) * sqrtf(aqq);
        if (p >= 0 && fabsf(apq) > tol * scale_pq) {
          if (fabsf(apq) > big_tol * scale_pq) big = 1;
          const float zf = (aqq - app) / (2.0f * apq);
          const float t = (zf >= 0.0f ? 1.0f : -1.0f) / (fabsf(zf) + sqrtf(1.0f + zf * zf));
          const float c = rsqrtf(1.0f + t * t), sn = c * t;
          if constexpr (VECS) {
            float* bp = B + (int64_t)p * ld;
            float* bq = B + (int64_t)q * ld;
#pragma unroll 4
            for (int i = gl; i < n; i += G) {
              const float x = mp[i], y = mq[i], u = bp[i], w = bq[i];
              // written out: the choice of the fused product is part of the result
              mp[i] = fmaf(c, x, -__fmul_rn(sn, y));
              mq[i] = fmaf(sn, x, __fmul_rn(c, y));
              bp[i] = fmaf(c, u, -__fmul_rn(sn, w));
              bq[i] = fmaf(sn, u, __fmul_rn(c, w));
            }
          } else {
            constexpr int U = 4;  // rows a lane loads before the first store
            for (int i0 = gl; i0 < n; i0 += G * U) {
              float x[U], y[U];
#pragma unroll
              for (int k4 = 0; k4 < U; ++k4) {
                const int i = min(i0 + G * k4, n - 1);
                x[k4] = mp[i];
                y[k4] = mq[i];
              }
#pragma unroll
              for (int k4 = 0; k4 < U; ++k4) {
                const int i = i0 + G * k4;
                if (i >= n) break;
                mp[i] = fmaf(c, x[k4], -__fmul_rn(sn, y[k4]));
                mq[i] = fmaf(sn, x[k4], __fmul_rn(c, y[k4]));
              }
            }
          }
          rotated = 1;
        }
        __syncwarp();
      }
      __syncthreads();
    }
    rotated = __syncthreads_or(rotated);
    big = __syncthreads_or(big);
    // quadratic convergence: after a sweep whose rotations all had
    // |a_pq| <= sqrt(tol) sqrt(a_pp a_qq), the off-diagonals are O(tol)
    converged = !rotated || !big;
  }
  *sweeps_out = sweep;
  // column norms (uniform slot count so every lane reaches every shuffle)
  for (int sidx = 0; sidx < (n + NG - 1) / NG; ++sidx) {
    const int k = group + sidx * NG;
    float s[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      s[v] = 0.0f;
      if (k < n)
        for (int i = gl + G * v; i < n; i += G * V) s[v] = fmaf(M[(int64_t)k * ld + i], M[(int64_t)k * ld + i], s[v]);
    }
    const float t = virtual_sum<V>(s);
    if (k < n && gl == 0) sigma[k] = sqrtf(t);
  }
  __syncthreads();
  return converged;
}

// |apq| > tol sqrt(app) sqrt(aqq), and the same with big_tol, as the FP64
// expressions decide it.  FP32 settles it unless the two sides are within 1e-5
// of each other (the truncations and roots are off by 4e-7) or the norms are
// out of range: then the FP64 roots (773 clocks each) are taken.
__device__ __forceinline__ bool rotates(double app, double aqq, double apq, double tol, double big_tol, bool& big) {
  const int ep = exponent_field(app), eq = exponent_field(aqq), e = max(ep, eq);
  if (min(ep, eq) > 0 && e < 0x7FF && e - min(ep, eq) <= 100) {
    const float scale = sqrtf(bits_to_float(app, e - 1023)) * sqrtf(bits_to_float(aqq, e - 1023));
    const float x = fabsf(bits_to_float(apq, e - 1023)), a = (float)tol * scale, b = (float)big_tol * scale;
    const bool sure = fabsf(x - a) > 1e-5f * a && fabsf(x - b) > 1e-5f * b;
    if (sure) {
      big = x > b;
      return x > a;
    }
  }
  const double scale = sqrt(app) * sqrt(aqq);
  big = fabs(apq) > big_tol * scale;
  return fabs(apq) > tol * scale;
}

// The double version, with the roundings of groups of 8 V lanes in the same
// way: below order 96 the FP32 basis that comes in is orthonormal to FP32 only,
// its defect stays in the scaling matrices, and a different rounding anywhere
// before the next basis is enough to move that basis and with it the iterates
// by 1e-6.  A FP64 instruction holds its quarter of the SM for 64 clocks
// whatever the lanes do, so four pairs share a warp's instructions, the
// rotation test is settled in FP32, and rotations by less than 2^-27, whose
// cosine rounds to 1, leave out the products with it.  With 8 V lanes a pair, two
// roots in every test and one warp a matrix in the step lengths
// (pair_lanczos_min) three iterations of 512 problems of order 6 to 64 took
// 72 ms, now 41 to 42; free in its roundings this part allowed 39.6.
template <int V>
__device__ __noinline__ bool cta_jacobi_svd_f64(int n, int ld, double* M, double* B, double* sigma, int max_sweeps,
                                                int* sweeps_out) {
  constexpr int G = 8, NG = NTHREADS / G;
  constexpr int U = 4;  // rows a lane loads before the first store (the compiler cannot move loads past them)
  const int gl = threadIdx.x & (G - 1), group = threadIdx.x / G;
  const int N = (n % 2 == 0) ? n : n + 1;
  const double tol = sqrt((double)n) * Num<double>::eps(), big_tol = sqrt(tol);
  const int slots = (N / 2 + NG - 1) / NG;  // the same for every group: shuffles stay uniform
  bool converged = (n <= 1);
  int sweep = 0;
  for (; sweep < max_sweeps && !converged; ++sweep) {
    int rotated = 0, big = 0;
    for (int r = 0; r < N - 1; ++r) {
      for (int sidx = 0; sidx < slots; ++sidx) {
        const int k = group + sidx * NG;
        int p = -1, q = -1;
        if (k < N / 2) {
          if (k == 0) {
            p = N - 1;
            q = r;
          } else {
            p = r + k < N - 1 ? r + k : r + k - (N - 1);
            q = r - k >= 0 ? r - k : r - k + (N - 1);
          }
          if (p >= n || q >= n) p = q = -1;
        }
        double* mp = M + (int64_t)(p < 0 ? 0 : p) * ld;
        double* mq = M + (int64_t)(p < 0 ? 0 : q) * ld;
        double spp[V], sqq[V], spq[V];
#pragma unroll
        for (int v = 0; v < V; ++v) spp[v] = sqq[v] = spq[v] = 0.0;
        if (p >= 0)
          for (int i0 = gl; i0 < n; i0 += G * V) {
#pragma unroll
            for (int v = 0; v < V; ++v) {
              const int i = i0 + G * v;
              if (i < n) {
                const double x = mp[i], y = mq[i];
                spp[v] = fma(x, x, spp[v]);
                sqq[v] = fma(y, y, sqq[v]);
                spq[v] = fma(x, y, spq[v]);
              }
            }
          }
        const double app = virtual_sum<V>(spp), aqq = virtual_sum<V>(sqq), apq = virtual_sum<V>(spq);
        bool large = false;
        if (p >= 0 && rotates(app, aqq, apq, tol, big_tol, large)) {
          if (large) big = 1;
          // the angle only needs float accuracy (the next sweep removes what
          // is left); c and s are formed in FP64 so the rotation is orthogonal
          // to its rounding
          const float zf = (float)((aqq - app) / (2.0 * apq));
          const float tf = (zf >= 0.0f ? 1.0f : -1.0f) / (fabsf(zf) + sqrtf(1.0f + zf * zf));
          const double t = widen(tf);
          const bool tiny = fabsf(tf) < 7.4505806e-9f;  // 2^-27: 1 + t^2 rounds to 1
          const double c = tiny ? 1.0 : rsqrt(fma(t, t, 1.0)), sn = tiny ? t : __dmul_rn(c, t);
          double* bp = B + (int64_t)p * ld;
          double* bq = B + (int64_t)q * ld;
          for (int i0 = gl; i0 < n; i0 += G * U) {
            double x[U], y[U], u[U], w[U];
#pragma unroll
            for (int k4 = 0; k4 < U; ++k4) {
              const int i = min(i0 + G * k4, n - 1);
              x[k4] = mp[i];
              y[k4] = mq[i];
              u[k4] = bp[i];
              w[k4] = bq[i];
            }
#pragma unroll
            for (int k4 = 0; k4 < U; ++k4) {
              const int i = i0 + G * k4;
              if (i >= n) break;
              // written out: the choice of the fused product is part of the result
              if (tiny) {
                mp[i] = __dadd_rn(x[k4], -__dmul_rn(sn, y[k4]));
                mq[i] = fma(sn, x[k4], y[k4]);
                bp[i] = __dadd_rn(u[k4], -__dmul_rn(sn, w[k4]));
                bq[i] = fma(sn, u[k4], w[k4]);
              } else {
                mp[i] = fma(c, x[k4], -__dmul_rn(sn, y[k4]));
                mq[i] = fma(sn, x[k4], __dmul_rn(c, y[k4]));
                bp[i] = fma(c, u[k4], -__dmul_rn(sn, w[k4]));
                bq[i] = fma(sn, u[k4], __dmul_rn(c, w[k4]));
              }
            }
          }
          rotated = 1;
        }
        __syncwarp();
      }
      __syncthreads();
    }
    rotated = __syncthreads_or(rotated);
    big = __syncthreads_or(big);
    // quadratic convergence, as in the float version
    converged = !rotated || !big;
  }
  *sweeps_out = sweep;
  for (int sidx = 0; sidx < (n + NG - 1) / NG; ++sidx) {
    const int k = group + sidx * NG;
    double s[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      s[v] = 0.0;
      if (k < n)
        for (int i = gl + G * v; i < n; i += G * V) s[v] = fma(M[(int64_t)k * ld + i], M[(int64_t)k * ld + i], s[v]);
    }
    const double t = virtual_sum<V>(s);
    if (k < n && gl == 0) sigma[k] = sqrt(t);
  }
  __syncthreads();
  return converged;
}

// The same where the incoming basis is orthonormal to FP64 (above order 95).
// The squared norms of M's columns are fresh at the start of a sweep and
// carried through its rotations (they only enter the test and the angle, which
// are float accurate; a sweep whose rotations are small changes them by their
// squares, one with large rotations is followed by another), and a rotation is
// three shears: 7 FP64 operations a row and pair, 5 in a sweep of tiny
// rotations, instead of 11.  The operands are in global memory at these
// orders: four rows are loaded before the first store, or every row waits for
// the cache (max-cut slice of 64 problems, n = 50 to 128: 176 ms, now 126).
// Below, a basis with FP32's defect passes it on to the scaling (1e-6), and
// the sums and rotations keep their roundings: a different one is enough to
// move an FP32 entry of a later iteration's start, and with it the iterates by
// that 1e-6.
__device__ inline bool cta_jacobi_polish(int n, int ld, double* M, double* B, double* sigma, int max_sweeps,
                                         int* sweeps_out) {
  constexpr int G = 8, NG = NTHREADS / G;
  constexpr int U = 4;  // rows a lane loads before the first store (the compiler cannot move loads past them)
  const int lane = threadIdx.x & 31, gl = lane & (G - 1), group = threadIdx.x / G;
  const int N = (n % 2 == 0) ? n : n + 1;
  const float tol = sqrtf((float)n) * 2.220446e-16f, big_tol = sqrtf(tol);
  double* nrm = sigma;
  const int nslots = (n + NG - 1) / NG;
  auto norms = [&]() {
    for (int sidx = 0; sidx < nslots; ++sidx) {
      const int k = group + sidx * NG;
      double s = 0.0;
      if (k < n) {
        const double* mk = M + (int64_t)k * ld;
        for (int i = gl; i < n; i += G) s = fma(mk[i], mk[i], s);
      }
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (k < n && gl == 0) nrm[k] = s;
    }
    __syncthreads();
  };
  norms();
  bool converged = (n <= 1);
  int sweep = 0;
  for (; sweep < max_sweeps && !converged; ++sweep) {
    int rotated = 0, big = 0;
    const int slots = (N / 2 + NG - 1) / NG;  // the same for every group: shuffles stay uniform
    for (int r = 0; r < N - 1; ++r) {
      for (int sidx = 0; sidx < slots; ++sidx) {
        const int k = group + sidx * NG;
        int p = -1, q = -1;
        if (k < N / 2) {
          if (k == 0) { p = N - 1; q = r; }
          else { p = r + k < N - 1 ? r + k : r + k - (N - 1); q = r - k >= 0 ? r - k : r - k + (N - 1); }
          if (p >= n || q >= n) p = q = -1;
        }
        double* mp = M + (int64_t)(p < 0 ? 0 : p) * ld;
        double* mq = M + (int64_t)(p < 0 ? 0 : q) * ld;
        double app = 0.0, aqq = 0.0, apq = 0.0;
        if (p >= 0) {
          app = nrm[p];
          aqq = nrm[q];
#pragma unroll 8
          for (int i = gl; i < n; i += G) apq = fma(mp[i], mq[i], apq);
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) apq += __shfl_xor_sync(0xffffffffu, apq, o);
        // scaled by the larger of the two norms' exponents
        const int e = max((__double2hiint(app) >> 20) & 0x7FF, (__double2hiint(aqq) >> 20) & 0x7FF) - 1023;
        const float fp = bits_to_float(app, e), fq = bits_to_float(aqq, e), fpq = bits_to_float(apq, e);
        const float scale = sqrtf(fp) * sqrtf(fq);
        if (p >= 0 && e < 1024 && fabsf(fpq) > tol * scale) {  // e = 1024: infinite or NaN
          if (fabsf(fpq) > big_tol * scale) big = 1;
          // the angle only needs float accuracy (the next sweep removes what
          // is left)
          const float zf = bits_to_float(aqq - app, e) / (2.0f * fpq);
          const float tf = (zf >= 0.0f ? 1.0f : -1.0f) / (fabsf(zf) + sqrtf(1.0f + zf * zf));
          const double t = widen(tf);
          double* bp = B + (int64_t)p * ld;
          double* bq = B + (int64_t)q * ld;
          // three shears: h = tan(angle / 2), sn = 2 h / (1 + h^2), orthogonal to
          // the rounding of sn.  tiny: the cosine is 1 - 5e-19, below the
          // rounding of a whole sweep
          const bool tiny = fabsf(tf) < 1e-9f;
          double h = 0.0, sn = t;
          if (gl == 0) {
            nrm[p] = fabs(fma(-t, apq, app));
            nrm[q] = fabs(fma(t, apq, aqq));
          }
          if (!tiny) {
            const float hf = tf / (1.0f + sqrtf(1.0f + tf * tf));
            h = widen(hf);
            const double h2 = h * h, hh = h + h;
            if (fabsf(hf) < 1e-4f) {
              sn = fma(hh, fma(h2, h2, -h2), hh);
            } else {
              const double a = 1.0 + h2, y = widen(1.0f / fmaf(hf, hf, 1.0f)), d = fma(-a, y, 1.0);
              sn = hh * fma(y, fma(d, d, d), y);
            }
          }
          for (int i0 = gl; i0 < n; i0 += G * U) {
            double x[U], y[U], u[U], v[U];
#pragma unroll
            for (int k4 = 0; k4 < U; ++k4) {
              const int i = min(i0 + G * k4, n - 1);
              x[k4] = mp[i];
              y[k4] = mq[i];
              u[k4] = bp[i];
              v[k4] = bq[i];
            }
#pragma unroll
            for (int k4 = 0; k4 < U; ++k4) {
              const int i = i0 + G * k4;
              if (i >= n) break;
              if (tiny) {
                mp[i] = fma(-sn, y[k4], x[k4]);
                mq[i] = fma(sn, x[k4], y[k4]);
                bp[i] = fma(-sn, v[k4], u[k4]);
                bq[i] = fma(sn, u[k4], v[k4]);
              } else {
                const double x1 = fma(-h, y[k4], x[k4]), u1 = fma(-h, v[k4], u[k4]);
                const double y1 = fma(sn, x1, y[k4]), v1 = fma(sn, u1, v[k4]);
                mp[i] = fma(-h, y1, x1);
                mq[i] = y1;
                bp[i] = fma(-h, v1, u1);
                bq[i] = v1;
              }
            }
          }
          rotated = 1;
        }
        __syncwarp();
      }
      __syncthreads();
    }
    rotated = __syncthreads_or(rotated);
    big = __syncthreads_or(big);
    // quadratic convergence
    converged = !rotated || !big;
    norms();
  }
  *sweeps_out = sweep;
  for (int k = threadIdx.x; k < n; k += NTHREADS) sigma[k] = sqrt(nrm[k]);
  __syncthreads();
  return converged;
}

// Column stride of the operands in shared memory: 8 mod 32 floats (8 mod 16
// doubles) puts the pairs of a warp, whose columns are consecutive, on
// different banks.
template <class T> __host__ __device__ __forceinline__ int jacobi_ld(int n) {
  return sizeof(T) == 4 ? (n + 23) / 32 * 32 + 8 : (n + 7) / 16 * 16 + 8;
}
// ld: column stride of M and B.
template <class T>
__device__ bool cta_jacobi_svd(int n, int ld, T* M, T* B, T* sigma, int max_sweeps, int* sweeps_out) {
  if constexpr (sizeof(T) == 8) {
    if (n <= 16) return cta_jacobi_svd_f64<1>(n, ld, M, B, sigma, max_sweeps, sweeps_out);
    if (n <= 48) return cta_jacobi_svd_f64<2>(n, ld, M, B, sigma, max_sweeps, sweeps_out);
    return cta_jacobi_svd_f64<4>(n, ld, M, B, sigma, max_sweeps, sweeps_out);
  } else {
    if (n <= 16) return cta_jacobi_svd_f32<1>(n, ld, M, B, sigma, max_sweeps, sweeps_out);
    if (n <= 48) return cta_jacobi_svd_f32<2>(n, ld, M, B, sigma, max_sweeps, sweeps_out);
    return cta_jacobi_svd_f32<4>(n, ld, M, B, sigma, max_sweeps, sweeps_out);
  }
}

// ---------------------------------------------------------------- tridiagonal
// Number of eigenvalues of the symmetric tridiagonal (a[0..k), b[1..k))
// smaller than x (Sturm count).
template <class T>
__device__ __forceinline__ int sturm_count(int k, const T* a, const T* b, T x, T pivmin) {
  int cnt = 0;
  T d = a[0] - x;
  if (fabs(d) < pivmin) d = -pivmin;
  if (d < 0) ++cnt;
  for (int i = 1; i < k; ++i) {
    d = (a[i] - x) - b[i] * b[i] / d;
    if (fabs(d) < pivmin) d = -pivmin;
    if (d < 0) ++cnt;
  }
  return cnt;
}

// Smallest eigenvalue of the tridiagonal (a, b) by warp-parallel multisection.
// Called by one full warp; every lane returns the result.
template <class T>
__device__ T warp_tridiag_eigmin_t(int k, const T* a, const T* b);

template <class T>
__device__ __forceinline__ T warp_tridiag_eigmin(int k, const T* a, const T* b) {
  return warp_tridiag_eigmin_t<T>(k, a, b);
}

// float64: bracket the eigenvalue with float Sturm counts (cheap divisions),
// then a few float64 multisection rounds inside the bracket.
template <>
__device__ __forceinline__ double warp_tridiag_eigmin<double>(int k, const double* a, const double* b) {
  const int lane = threadIdx.x & 31;
  double scale = 0;
  for (int i = 0; i < k; ++i) scale = fmax(scale, fabs(a[i]) + (i > 0 ? fabs(b[i]) : 0.0) + (i + 1 < k ? fabs(b[i + 1]) : 0.0));
  if (!(scale > 0.0) || !isfinite(scale)) return warp_tridiag_eigmin_t<double>(k, a, b);
  // float multisection on the scaled tridiagonal (entries in [-1, 1])
  const float inv = (float)(1.0 / scale);
  float lo = -1.0f, hi = 1.0f;
  const float pivf = 1e-30f;
  for (int it = 0; it < 5; ++it) {
    const float x = lo + (hi - lo) * (float)(lane + 1) / 33.0f;
    int c = 0;
    float d = (float)a[0] * inv - x;
    if (fabsf(d) < pivf) d = -pivf;
    c += d < 0.0f;
    for (int i = 1; i < k; ++i) {
      const float bi = (float)b[i] * inv;
      d = ((float)a[i] * inv - x) - bi * bi / d;
      if (fabsf(d) < pivf) d = -pivf;
      c += d < 0.0f;
    }
    const unsigned ball = __ballot_sync(0xffffffffu, c >= 1);
    if (ball == 0) { lo = lo + (hi - lo) * 32.0f / 33.0f; continue; }
    const int first = __ffs(ball) - 1;
    const float nhi = lo + (hi - lo) * (float)(first + 1) / 33.0f;
    const float nlo = first == 0 ? lo : lo + (hi - lo) * (float)first / 33.0f;
    lo = nlo; hi = nhi;
  }
  // widen by the float rounding of the scaled problem and polish in float64
  const double w = 4e-6 * fmax(1.0, fabs((double)lo) + fabs((double)hi));
  double dlo = ((double)lo - w) * scale, dhi = ((double)hi + w) * scale;
  const double pivmin = 4.93e-32 * fmax(scale, 1e-30);
  // confirm the bracket (fall back to the full search if rounding moved it)
  const int cl = sturm_count<double>(k, a, b, dlo, pivmin);
  const int ch = sturm_count<double>(k, a, b, dhi, pivmin);
  if (cl != 0 || ch < 1) return warp_tridiag_eigmin_t<double>(k, a, b);
  for (int it = 0; it < 16; ++it) {
    if (dhi - dlo <= 2.0 * 2.220446049250313e-16 * fmax(fabs(dlo), fabs(dhi)) + pivmin) break;
    const double x = dlo + (dhi - dlo) * (double)(lane + 1) / 33.0;
    const int c = sturm_count<double>(k, a, b, x, pivmin);
    const unsigned ball = __ballot_sync(0xffffffffu, c >= 1);
    if (ball == 0) { dlo = dlo + (dhi - dlo) * 32.0 / 33.0; continue; }
    const int first = __ffs(ball) - 1;
    const double nhi = dlo + (dhi - dlo) * (double)(first + 1) / 33.0;
    const double nlo = first == 0 ? dlo : dlo + (dhi - dlo) * (double)first / 33.0;
    dlo = nlo; dhi = nhi;
  }
  return (dlo + dhi) / 2;
}

template <class T>
__device__ T warp_tridiag_eigmin_t(int k, const T* a, const T* b) {
  const int lane = threadIdx.x & 31;
  T lo = 0, hi = 0, scale = 0;
  // Gershgorin interval
  for (int i = 0; i < k; ++i) {
    const T r = (i > 0 ? fabs(b[i]) : (T)0) + (i + 1 < k ? fabs(b[i + 1]) : (T)0);
    const T l = a[i] - r, h = a[i] + r;
    if (i == 0 || l < lo) lo = l;
    if (i == 0 || h > hi) hi = h;
    scale = fmax(scale, fmax(fabs(l), fabs(h)));
  }
  const T pivmin = (T)(Num<T>::eps() * Num<T>::eps()) * fmax(scale, (T)1e-30);
  for (int it = 0; it < 64; ++it) {
    if (hi - lo <= (T)2 * Num<T>::eps() * fmax(fabs(lo), fabs(hi)) + pivmin) break;
    const T x = lo + (hi - lo) * (T)(lane + 1) / (T)33;
    const int c = sturm_count(k, a, b, x, pivmin);
    const unsigned ball = __ballot_sync(0xffffffffu, c >= 1);
    if (ball == 0) { lo = lo + (hi - lo) * (T)32 / (T)33; continue; }
    const int first = __ffs(ball) - 1;  // smallest lane with count >= 1
    const T nhi = lo + (hi - lo) * (T)(first + 1) / (T)33;
    const T nlo = first == 0 ? lo : lo + (hi - lo) * (T)first / (T)33;
    lo = nlo; hi = nhi;
  }
  return (lo + hi) / (T)2;
}

// The j-th smallest eigenvalue (0-based) of the tridiagonal by bisection,
// computed by one thread.
template <class T>
__device__ T thread_tridiag_eig(int k, const T* a, const T* b, int j) {
  T lo = 0, hi = 0, scale = 0;
  for (int i = 0; i < k; ++i) {
    const T r = (i > 0 ? fabs(b[i]) : (T)0) + (i + 1 < k ? fabs(b[i + 1]) : (T)0);
    const T l = a[i] - r, h = a[i] + r;
    if (i == 0 || l < lo) lo = l;
    if (i == 0 || h > hi) hi = h;
    scale = fmax(scale, fmax(fabs(l), fabs(h)));
  }
  const T pivmin = (T)(Num<T>::eps() * Num<T>::eps()) * fmax(scale, (T)1e-30);
  for (int it = 0; it < 200; ++it) {
    if (hi - lo <= (T)2 * Num<T>::eps() * fmax(fabs(lo), fabs(hi)) + pivmin) break;
    const T x = (lo + hi) / (T)2;
    if (sturm_count(k, a, b, x, pivmin) >= j + 1) hi = x;
    else lo = x;
  }
  return (lo + hi) / (T)2;
}

// ---------------------------------------------------------------- warp routines
// Smallest eigenvalue of the symmetric Z (n x n) by Lanczos with full
// reorthogonalization, run by ONE warp (the role of
// LowRankOpt.lanczos_eigmin!, src/step.jl:151-183).  Q (n x n) holds the
// basis; a, bb, coef are vectors of length n+1, w of length n.  Stops when
// the smallest Ritz value is stable to 64 eps or the Krylov space is
// exhausted (k = n or b_k ~ 0).
// ldq: column stride of the basis in shared memory, odd, so that the lanes that
// each sum over one column read different banks (at n = 64 an even stride put
// all 32 on one).
template <class T>
__device__ T warp_lanczos_eigmin(int n, const T* Z, T* Qs, int ldq, int kq, T* Qg, T* a, T* bb, T* w, T* coef,
                                 int* steps) {
  const int lane = threadIdx.x & 31;
  // column l of the basis: shared memory for l < kq, global memory after
  auto Qc = [&](int l) -> T* { return l < kq ? Qs + l * ldq : Qg + (int64_t)l * n; };
  T* Q = Qc(0);
  T nrm2 = 0;
  for (int i = lane; i < n; i += 32) {
    uint32_t h = (uint32_t)(i + 1) * 2654435761u;
    h ^= h >> 15; h *= 2246822519u; h ^= h >> 13;
    const T v = (T)((double)(h & 0xffffff) / 16777216.0 - 0.5) + (T)0.01;
    Q[i] = v;
    nrm2 = fma(v, v, nrm2);
  }
  nrm2 = warp_sum(nrm2);
  {
    const T inv = (T)1 / Num<T>::sqrt_(nrm2);
    for (int i = lane; i < n; i += 32) Q[i] *= inv;
  }
  __syncwarp();
  T theta = 0, theta_prev = (T)INFINITY, znorm = 0;
  int k = 0;
  for (int j = 0; j < n; ++j) {
    const T* qj = Qc(j);
    // w = Z q_j (Z symmetric; lanes read consecutive rows of each column)
    T wl[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) wl[t] = 0;
    for (int r = 0; r < n; ++r) {
      const T qr = qj[r];
      const T* zr = Z + (int64_t)r * n;
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const int i = lane + 32 * t;
        if (i < n) wl[t] = fma(zr[i], qr, wl[t]);
      }
    }
    T aj = 0;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int i = lane + 32 * t;
      if (i < n) aj = fma(qj[i], wl[t], aj);
    }
    aj = warp_sum(aj);
    const T bj = j > 0 ? bb[j] : (T)0;
    const T* qp = j > 0 ? Qc(j - 1) : qj;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int i = lane + 32 * t;
      if (i < n) {
        T v = wl[t] - aj * qj[i];
        if (j > 0) v -= bj * qp[i];
        wl[t] = v;
        w[i] = v;
      }
    }
    if (lane == 0) a[j] = aj;
    __syncwarp();
    // full reorthogonalization, twice: coef_l = Q_l . w (one lane per l)
    for (int pass = 0; pass < 2; ++pass) {
      for (int l = lane; l <= j; l += 32) {
        const T* ql = Qc(l);
        T s = 0;
        for (int i = 0; i < n; ++i) s = fma(ql[i], w[i], s);
        coef[l] = s;
      }
      __syncwarp();
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const int i = lane + 32 * t;
        if (i < n) {
          T v = wl[t];
          for (int l = 0; l <= j; ++l) v = fma(-coef[l], Qc(l)[i], v);
          wl[t] = v;
        }
      }
      __syncwarp();
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const int i = lane + 32 * t;
        if (i < n) w[i] = wl[t];
      }
      __syncwarp();
    }
    T bn = 0;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int i = lane + 32 * t;
      if (i < n) bn = fma(wl[t], wl[t], bn);
    }
    bn = Num<T>::sqrt_(warp_sum(bn));
    k = j + 1;
    znorm = fmax(znorm, fabs(aj) + bn + fabs(bj));
    if (lane == 0) bb[j + 1] = bn;
    __syncwarp();
    const bool exhausted = (k == n) || !(bn > Num<T>::eps() * znorm * (T)4);
    if (exhausted || (k >= 4 && (k % 4) == 0)) {
      theta = warp_tridiag_eigmin<T>(k, a, bb);
      const T tolr = Num<T>::eps() * (T)64 * fmax((T)1, fabs(theta));
      if (exhausted || fabs(theta - theta_prev) <= tolr) break;
      theta_prev = theta;
    }
    T* qn = Qc(j + 1);
    const T inv = (T)1 / bn;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int i = lane + 32 * t;
      if (i < n) qn[i] = wl[t] * inv;
    }
    __syncwarp();
  }
  *steps = k;
  return theta;
}

// x lies above the smallest eigenvalue of the tridiagonal (a, b2), by the
// count of sturm_count (the first negative pivot decides): the same values,
// with the squares of b formed once.
__device__ __forceinline__ bool sturm_below(int k, const double* a, const double* b2, double x, double pivmin) {
  double d = a[0] - x;
  if (fabs(d) < pivmin) d = -pivmin;
  bool neg = d < 0.0;
  for (int i = 1; i < k; ++i) {
    d = (a[i] - x) - b2[i] / d;
    if (fabs(d) < pivmin) d = -pivmin;
    neg = neg || d < 0.0;
  }
  return neg;
}

// Work vectors of tridiag_eigmin_as for k rows: squares of b, the scaled
// tridiagonal of the division-free counts, and the FP32 one.
struct TridiagWork {
  double *b2, *sa, *sb;
  float *af, *bf;
};

// The value of warp_tridiag_eigmin<double>, bit for bit, at about half of its
// FP64 instructions: one warp, `th32` gets the FP32 bracket's middle.
// The 32 points of a multisection round are compared with an eigenvalue known
// to 1e-14 of the norm from division-free counts (tridiag.cuh); only points
// within 2e-14 of that get the count with divisions (900 clocks a row).  Both
// kinds of count are exact for a matrix within a few eps of this one, so
// beyond 90 eps they agree.  want = false: the FP32 part alone.
__device__ __noinline__ inline double tridiag_eigmin_as(int k, const double* a, const double* b, const TridiagWork& W, bool want,
                                           double* scale_out, float* th32) {
  const int lane = threadIdx.x & 31;
  double scale = 0.0;
  for (int i = lane; i < k; i += 32)
    scale = fmax(scale, fabs(a[i]) + (i > 0 ? fabs(b[i]) : 0.0) + (i + 1 < k ? fabs(b[i + 1]) : 0.0));
#pragma unroll
  for (int o = 16; o; o >>= 1) scale = fmax(scale, __shfl_xor_sync(0xffffffffu, scale, o));
  *scale_out = scale;
  *th32 = 0.0f;
  if (!(scale > 1e-30 && scale < 1e30))  // the general form takes any scale
    return want ? warp_tridiag_eigmin<double>(k, a, b) : 0.0;
  const float inv = (float)(1.0 / scale);
  const int e = ((__double2hiint(scale) >> 20) & 0x7FF) - 1022;  // scale < 2^e
  const double f = __longlong_as_double((long long)(1023 - e) << 52);
  for (int i = lane; i < k; i += 32) {
    const float bi = i > 0 ? (float)b[i] * inv : 0.0f;
    W.af[i] = (float)a[i];
    W.bf[i] = __fmul_rn(bi, bi);
    if (want) {
      const double y = i > 0 ? b[i] : 0.0;
      W.b2[i] = __dmul_rn(y, y);
      W.sa[i] = a[i] * f;
      W.sb[i] = (y * f) * (y * f);
    }
  }
  __syncwarp();
  float lo = -1.0f, hi = 1.0f;
  const float pivf = 1e-30f;
  for (int it = 0; it < 5; ++it) {
    const float x = lo + (hi - lo) * (float)(lane + 1) / 33.0f;
    // the first row's product was rounded there, the others' were fused
    float d = __fsub_rn(__fmul_rn(W.af[0], inv), x);
    if (fabsf(d) < pivf) d = -pivf;
    bool neg = d < 0.0f;
    for (int i = 1; i < k; ++i) {
      d = __fadd_rn(fmaf(W.af[i], inv, -x), -(W.bf[i] / d));
      if (fabsf(d) < pivf) d = -pivf;
      neg = neg || d < 0.0f;
    }
    const unsigned ball = __ballot_sync(0xffffffffu, neg);
    if (ball == 0) { lo = lo + (hi - lo) * 32.0f / 33.0f; continue; }
    const int first = __ffs(ball) - 1;
    const float nhi = lo + (hi - lo) * (float)(first + 1) / 33.0f;
    const float nlo = first == 0 ? lo : lo + (hi - lo) * (float)first / 33.0f;
    lo = nlo; hi = nhi;
  }
  *th32 = 0.5f * (lo + hi);
  if (!want) return 0.0;
  const double w = 4e-6 * fmax(1.0, fabs((double)lo) + fabs((double)hi));
  double dlo = ((double)lo - w) * scale, dhi = ((double)hi + w) * scale;
  const double pivmin = 4.93e-32 * fmax(scale, 1e-30);
  // the eigenvalue to 1e-14 of the norm, [tl, tu] in units of 2^e
  double tl = dlo * f, tu = dhi * f;
  bool tested_l = false, tested_u = false;
  for (int it = 0; it < 8 && tu - tl > 1e-14; ++it) {
    const double h = (tu - tl) * (1.0 / 33.0);
    const unsigned above = __ballot_sync(0xffffffffu, sturm_above(k, W.sa, W.sb, fma(h, (double)(lane + 1), tl)));
    const int first = above == 0xffffffffu ? 32 : __ffs(~above) - 1;
    const double l = tl;
    tl = fma(h, (double)first, l);
    tested_l = tested_l || first > 0;
    if (first < 32) {
      tu = fma(h, (double)(first + 1), l);
      tested_u = true;
    }
  }
  // the FP32 bracket is 4e-6 to both sides: an end that never moved was not
  // tested, and the general form sees to it
  if (!tested_l || !tested_u) return warp_tridiag_eigmin<double>(k, a, b);
  const double g = __longlong_as_double((long long)(1023 + e) << 52);
  const double near_lo = (tl - 2e-14) * g, near_hi = (tu + 2e-14) * g;
  for (int it = 0; it < 16; ++it) {
    if (dhi - dlo <= 2.0 * 2.220446049250313e-16 * fmax(fabs(dlo), fabs(dhi)) + pivmin) break;
    const double x = dlo + (dhi - dlo) * (double)(lane + 1) / 33.0;
    bool neg = x > near_hi;
    const bool close = x >= near_lo && x <= near_hi;
    if (__any_sync(0xffffffffu, close)) {
      const bool c = sturm_below(k, a, W.b2, x, pivmin);
      if (close) neg = c;
    }
    const unsigned ball = __ballot_sync(0xffffffffu, neg);
    if (ball == 0) { dlo = dlo + (dhi - dlo) * 32.0 / 33.0; continue; }
    const int first = __ffs(ball) - 1;
    const double nhi = dlo + (dhi - dlo) * (double)(first + 1) / 33.0;
    const double nlo = first == 0 ? dlo : dlo + (dhi - dlo) * (double)first / 33.0;
    dlo = nlo; dhi = nhi;
  }
  return (dlo + dhi) / 2;
}

// Shared state of pair_lanczos_min, one entry a matrix.
struct LanczosShared {
  double alpha[2], inv[2], theta[2];
  int steps[2], stop[2];
};

// Smallest eigenvalues of two symmetric matrices (n x n, n <= 256) in float64,
// the iteration of warp_lanczos_eigmin with its roundings, two warps a matrix:
// a row of the vectors per lane, a coefficient per lane, the sums over the rows
// (alpha, the norm) and the tridiagonal on one warp of the two, as there.  Z,
// the first columns of the basis and the vectors live in shared memory as far
// as they fit.
// The roundings matter: the step length enters every entry of the next iterate
// (see cta_jacobi_svd_f64).  The FP64 Ritz value is formed only where the
// iteration can stop: while the FP32 one (good to 1e-6 of the norm) still moves
// by more than 2e-5 of the norm in four steps, the FP64 one moves by more than
// 64 eps max(1, |theta|).
// Bound by the FP64 units: a multiply-add of one warp holds a quarter of the SM
// for 64 clocks.  With one warp a matrix, all columns on one shared-memory bank
// at even orders and nine counts with divisions for each Ritz value it took
// about half of the iteration of a block of 64.
template <int R>  // rows a lane, n <= 64 R
__device__ __noinline__ void pair_lanczos_min_r(int n, const double* ZX, const double* ZS, double* QX, double* QS,
                                                unsigned char* smem, int64_t smem_bytes, LanczosShared& sh) {
  static_assert(NTHREADS == 128, "two warps a matrix");
  const double eps = 2.220446049250313e-16;
  const int side = threadIdx.x >> 6, gt = threadIdx.x & 63, gw = gt >> 5, lane = gt & 31;
  // the blocks of an SM (numbers 152 apart) take their one-warp parts on
  // different quarters of it
  const bool lead = gw == ((int)(blockIdx.x / 152) & 1);
  const int cl = lead ? lane + 32 : lane;  // coefficients 0-31 on the other warp
  const int64_t nn = (int64_t)n * n;
  const int ldq = n | 1;
  const int64_t vec = 8 * (int64_t)(n + 1), cap = smem_bytes / 16;  // doubles of one matrix
  const bool zs = cap - nn - vec >= (int64_t)ldq * min(n, 16);
  const int kq = (int)min((int64_t)n, max((int64_t)0, (cap - vec - (zs ? nn : 0)) / ldq));
  double* base = (double*)smem + (side ? cap : 0);
  double* a = base;
  double* bb = a + (n + 1);
  double* w = bb + (n + 1);
  double* coef = w + (n + 1);
  TridiagWork tw;
  tw.b2 = coef + (n + 1);
  tw.sa = tw.b2 + (n + 1);
  tw.sb = tw.sa + (n + 1);
  tw.af = (float*)(tw.sb + (n + 1));
  tw.bf = tw.af + (n + 1);
  double* Qs = base + vec;
  double* Zs = Qs + (int64_t)kq * ldq;
  const double* Zg = side ? ZS : ZX;
  double* Qg = side ? QS : QX;
  auto Qc = [&](int l) -> double* { return l < kq ? Qs + l * ldq : Qg + (int64_t)l * n; };
  auto bar = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + side) : "memory"); };
  // sum over the rows i = lane, lane + 32, ... of p_i q_i, then over the lanes
  auto dot = [&](const double* p, const double* q) {
    double s = 0.0;
#pragma unroll 4
    for (int i = lane; i < n; i += 32) s = fma(p[i], q[i], s);
    return warp_sum(s);
  };
  if (zs)
    for (int k = gt; k < (int)nn; k += 64) Zs[k] = Zg[k];
  const double* Z = zs ? Zs : Zg;
  if (lead) {
    double* Q = Qc(0);
    double nrm2 = 0.0;
    for (int i = lane; i < n; i += 32) {
      uint32_t h = (uint32_t)(i + 1) * 2654435761u;
      h ^= h >> 15; h *= 2246822519u; h ^= h >> 13;
      const double v = ((double)(h & 0xffffff) / 16777216.0 - 0.5) + 0.01;
      Q[i] = v;
      nrm2 = fma(v, v, nrm2);
    }
    const double inv = 1.0 / sqrt(warp_sum(nrm2));
    for (int i = lane; i < n; i += 32) Q[i] *= inv;
  }
  bar();
  double theta = 0.0, theta_prev = INFINITY, znorm = 0.0;  // the lead warp's
  float here = 0.0f, here_prev = INFINITY;
  bool have_prev = true;
  for (int j = 0; j < n; ++j) {
    const double* qj = Qc(j);
    const double* qp = j > 0 ? Qc(j - 1) : qj;
    double wl[R];
#pragma unroll
    for (int t = 0; t < R; ++t) wl[t] = 0.0;
    // w = Z q_j; the next columns are loaded while these are summed
    constexpr int P = R <= 2 ? 4 : 2;
    double z[P][R];
    auto load = [&](int r) {
#pragma unroll
      for (int u = 0; u < P; ++u)
#pragma unroll
        for (int t = 0; t < R; ++t) z[u][t] = Z[(int64_t)min(r + u, n - 1) * n + min(gt + 64 * t, n - 1)];
    };
    load(0);
    for (int r = 0; r < n; r += P) {
      double y[P][R];
#pragma unroll
      for (int u = 0; u < P; ++u)
#pragma unroll
        for (int t = 0; t < R; ++t) y[u][t] = z[u][t];
      if (r + P < n) load(r + P);
#pragma unroll
      for (int u = 0; u < P; ++u)
        if (r + u < n) {
          const double qr = qj[r + u];
#pragma unroll
          for (int t = 0; t < R; ++t)
            if (gt + 64 * t < n) wl[t] = fma(y[u][t], qr, wl[t]);
        }
    }
#pragma unroll
    for (int t = 0; t < R; ++t)
      if (gt + 64 * t < n) w[gt + 64 * t] = wl[t];
    bar();
    if (lead) {
      const double aj = dot(qj, w);
      if (lane == 0) {
        a[j] = aj;
        sh.alpha[side] = aj;
      }
    }
    bar();
    {
      const double aj = sh.alpha[side], bj = j > 0 ? bb[j] : 0.0;
#pragma unroll
      for (int t = 0; t < R; ++t) {
        const int i = gt + 64 * t;
        if (i < n) {
          double v = fma(-aj, qj[i], wl[t]);
          if (j > 0) v = fma(-bj, qp[i], v);
          wl[t] = v;
          w[i] = v;
        }
      }
    }
    bar();
    // full reorthogonalization, twice: coef_l = Q_l . w (one lane per l)
    for (int pass = 0; pass < 2; ++pass) {
      for (int l = cl; l <= j; l += 64) {
        const double* ql = Qc(l);
        double s = 0.0;
#pragma unroll 4
        for (int i = 0; i < n; ++i) s = fma(ql[i], w[i], s);
        coef[l] = s;
      }
      bar();
#pragma unroll
      for (int t = 0; t < R; ++t) {
        const int i = gt + 64 * t;
        if (i < n) {
          double v = wl[t];
#pragma unroll 4
          for (int l = 0; l <= j; ++l) v = fma(-coef[l], Qc(l)[i], v);
          wl[t] = v;
          w[i] = v;
        }
      }
      bar();
    }
    const int k = j + 1;
    if (lead) {
      const double aj = sh.alpha[side], bj = j > 0 ? bb[j] : 0.0;
      const double bn = sqrt(dot(w, w));
      znorm = fmax(znorm, fabs(aj) + bn + fabs(bj));
      if (lane == 0) bb[k] = bn;
      __syncwarp();
      const bool exhausted = (k == n) || !(bn > eps * znorm * 4.0);
      bool stop = exhausted;
      if (exhausted || (k >= 4 && (k % 4) == 0)) {
        double scale;
        float th;
        tridiag_eigmin_as(k, a, bb, tw, false, &scale, &th);
        here = th * (float)scale;
        const bool moves = scale > 1e-8 && scale < 1e30 && fabsf(here - here_prev) > 2e-5f * (float)scale;
        if (exhausted || !moves) {
          if (!exhausted && !have_prev) theta_prev = tridiag_eigmin_as(k - 4, a, bb, tw, true, &scale, &th);
          theta = tridiag_eigmin_as(k, a, bb, tw, true, &scale, &th);
          const double tolr = eps * 64.0 * fmax(1.0, fabs(theta));
          stop = exhausted || fabs(theta - theta_prev) <= tolr;
          theta_prev = theta;
          have_prev = true;
        } else {
          have_prev = false;
        }
        here_prev = here;
      }
      if (lane == 0) {
        sh.stop[side] = stop;
        sh.inv[side] = 1.0 / bn;
        if (stop) {
          sh.theta[side] = theta;
          sh.steps[side] = k;
        }
      }
    }
    bar();
    if (sh.stop[side]) break;
    {
      double* qn = Qc(k);
      const double inv = sh.inv[side];
#pragma unroll
      for (int t = 0; t < R; ++t)
        if (gt + 64 * t < n) qn[gt + 64 * t] = wl[t] * inv;
    }
    bar();
  }
  __syncthreads();
}
__device__ inline void pair_lanczos_min(int n, const double* ZX, const double* ZS, double* QX, double* QS,
                                        unsigned char* smem, int64_t smem_bytes, LanczosShared& sh) {
  if (n <= 64) pair_lanczos_min_r<1>(n, ZX, ZS, QX, QS, smem, smem_bytes, sh);
  else if (n <= 128) pair_lanczos_min_r<2>(n, ZX, ZS, QX, QS, smem, smem_bytes, sh);
  else pair_lanczos_min_r<4>(n, ZX, ZS, QX, QS, smem, smem_bytes, sh);
}

// Solve L L' x = b in place (L lower, ld m) by ONE warp; x (and L, when
// the caller staged it) in shared memory.
template <class T, class V>
__device__ void warp_potrs(int m, const T* __restrict__ L, V* x, V* rdiag) {
  const int lane = threadIdx.x & 31;
  // reciprocal diagonal once (lanes in parallel) instead of a division per row
  for (int k = lane; k < m; k += 32) rdiag[k] = (V)1 / (V)widen(L[k + (int64_t)k * m]);
  __syncwarp();
  for (int k = 0; k < m; ++k) {
    const V xk = x[k] * rdiag[k];
    __syncwarp();
    if (lane == 0) x[k] = xk;
    const T* lk = L + (int64_t)k * m;
    for (int i = k + 1 + lane; i < m; i += 32) x[i] -= (V)widen(lk[i]) * xk;
    __syncwarp();
  }
  for (int k = m - 1; k >= 0; --k) {
    const T* lk = L + (int64_t)k * m;
    V s = 0;
    for (int i = k + 1 + lane; i < m; i += 32) s += (V)widen(lk[i]) * x[i];
    s = warp_sum(s);
    if (lane == 0) x[k] = (x[k] - s) * rdiag[k];
    __syncwarp();
  }
}

// Full Lanczos tridiagonalization of the symmetric Z (n x n) by ONE warp:
// n steps with full reorthogonalization; when the Krylov space closes early
// (b ~ 0) it restarts from a new vector orthogonal to the basis (b = 0 in
// T), so T (a[0..n), bb[1..n)) has exactly the eigenvalues of Z.
template <class T>
__device__ void warp_lanczos_full(int n, const T* Z, T* Q, T* a, T* bb, T* w, T* coef) {
  const int lane = threadIdx.x & 31;
  auto start_vector = [&](int j, uint32_t seed) {
    T* q = Q + (int64_t)j * n;
    for (int i = lane; i < n; i += 32) {
      uint32_t h = (uint32_t)(i + 1) * 2654435761u + seed * 40503u;
      h ^= h >> 15; h *= 2246822519u; h ^= h >> 13;
      q[i] = (T)((double)(h & 0xffffff) / 16777216.0 - 0.5) + (T)0.01;
    }
    __syncwarp();
    // orthogonalize twice against the previous columns, then normalize
    for (int pass = 0; pass < 2; ++pass) {
      for (int l = lane; l < j; l += 32) {
        const T* ql = Q + (int64_t)l * n;
        T s = 0;
        for (int i = 0; i < n; ++i) s = fma(ql[i], q[i], s);
        coef[l] = s;
      }
      __syncwarp();
      for (int i = lane; i < n; i += 32) {
        T v = q[i];
        for (int l = 0; l < j; ++l) v = fma(-coef[l], Q[i + (int64_t)l * n], v);
        q[i] = v;
      }
      __syncwarp();
    }
    T nrm = 0;
    for (int i = lane; i < n; i += 32) nrm = fma(q[i], q[i], nrm);
    nrm = Num<T>::sqrt_(warp_sum(nrm));
    const T inv = nrm > (T)0 ? (T)1 / nrm : (T)0;
    for (int i = lane; i < n; i += 32) q[i] *= inv;
    __syncwarp();
  };
  start_vector(0, 1u);
  T znorm = 0;
  for (int j = 0; j < n; ++j) {
    const T* qj = Q + (int64_t)j * n;
    for (int i = lane; i < n; i += 32) {
      T s = 0;
      for (int r = 0; r < n; ++r) s = fma(Z[i + (int64_t)r * n], qj[r], s);
      w[i] = s;
    }
    __syncwarp();
    T aj = 0;
    for (int i = lane; i < n; i += 32) aj = fma(qj[i], w[i], aj);
    aj = warp_sum(aj);
    const T bj = j > 0 ? bb[j] : (T)0;
    const T* qp = j > 0 ? Q + (int64_t)(j - 1) * n : qj;
    for (int i = lane; i < n; i += 32) {
      T v = w[i] - aj * qj[i];
      if (j > 0) v -= bj * qp[i];
      w[i] = v;
    }
    if (lane == 0) a[j] = aj;
    __syncwarp();
    for (int pass = 0; pass < 2; ++pass) {
      for (int l = lane; l <= j; l += 32) {
        const T* ql = Q + (int64_t)l * n;
        T s = 0;
        for (int i = 0; i < n; ++i) s = fma(ql[i], w[i], s);
        coef[l] = s;
      }
      __syncwarp();
      for (int i = lane; i < n; i += 32) {
        T v = w[i];
        for (int l = 0; l <= j; ++l) v = fma(-coef[l], Q[i + (int64_t)l * n], v);
        w[i] = v;
      }
      __syncwarp();
    }
    if (j + 1 == n) break;
    T bn = 0;
    for (int i = lane; i < n; i += 32) bn = fma(w[i], w[i], bn);
    bn = Num<T>::sqrt_(warp_sum(bn));
    znorm = fmax(znorm, fabs(aj) + bn + fabs(bj));
    T* qn = Q + (int64_t)(j + 1) * n;
    if (bn > Num<T>::eps() * fmax(znorm, (T)1e-300) * (T)4) {
      const T inv = (T)1 / bn;
      for (int i = lane; i < n; i += 32) qn[i] = w[i] * inv;
      if (lane == 0) bb[j + 1] = bn;
      __syncwarp();
    } else {
      if (lane == 0) bb[j + 1] = (T)0;
      __syncwarp();
      start_vector(j + 1, (uint32_t)(j + 2));
    }
  }
}

// ---------------------------------------------------------------- Bunch-Kaufman
// Symmetric indefinite factorization A = P L D L' P' with 1x1 and 2x2
// pivots (Bunch-Kaufman partial pivoting, the LAPACK sytf2 "lower"
// algorithm), in place on the lower triangle of the m x m matrix `a`
// (leading dimension lda).  piv[k] = kp for a 1x1 pivot (rows k and kp
// swapped); piv[k] = piv[k+1] = -(kp + 1) for a 2x2 pivot whose second row
// was swapped with kp.  Returns false when a pivot column is exactly zero
// (singular).  `work` holds 2m scratch values.
template <class T>
__device__ bool cta_sytrf_lower(int m, T* a, int lda, double* piv, T* work, RedBuf* rb, int* flag) {
  const T alpha = (T)((1.0 + sqrt(17.0)) / 8.0);
  auto A = [&](int i, int j) -> T& { return a[i + (int64_t)j * lda]; };
  int k = 0;
  while (k < m) {
    // colmax and its row (smallest index on ties)
    double cm = -1.0;
    int ci = m;
    for (int i = k + 1 + threadIdx.x; i < m; i += NTHREADS) {
      const double v = fabs((double)A(i, k));
      if (v > cm) { cm = v; ci = i; }
    }
    // block argmax: encode (value, -index) through two reductions
    const double colmax_all = block_max(cm, rb);
    int cand = (cm == colmax_all && cm >= 0.0) ? ci : m;
    // smallest index attaining the max
    if (threadIdx.x == 0) *flag = m;
    __syncthreads();
    if (cand < m) atomicMin(flag, cand);
    __syncthreads();
    const int imax = *flag;
    __syncthreads();
    const double colmax = (k + 1 < m) ? fmax(colmax_all, 0.0) : 0.0;
    const double absakk = fabs((double)A(k, k));
    if (!(fmax(absakk, colmax) > 0.0)) return false;  // zero column (or NaN): singular
    int kp = k, kstep = 1;
    if (!(absakk >= (double)alpha * colmax)) {
      // rowmax: largest off-diagonal magnitude in row/column imax of the trailing matrix
      double rm = 0.0;
      for (int j = k + threadIdx.x; j < m; j += NTHREADS) {
        if (j == imax) continue;
        const double v = j < imax ? fabs((double)A(imax, j)) : fabs((double)A(j, imax));
        rm = fmax(rm, v);
      }
      const double rowmax = block_max(rm, rb);
      if (absakk >= (double)alpha * colmax * (colmax / rowmax)) kp = k;
      else if (fabs((double)A(imax, imax)) >= (double)alpha * rowmax) kp = imax;
      else { kp = imax; kstep = 2; }
    }
    const int kk = k + kstep - 1;
    if (kp != kk) {
      // symmetric interchange of rows/columns kk and kp in the trailing matrix
      for (int i = kp + 1 + threadIdx.x; i < m; i += NTHREADS) {
        const T t = A(i, kk); A(i, kk) = A(i, kp); A(i, kp) = t;
      }
      for (int j = kk + 1 + threadIdx.x; j < kp; j += NTHREADS) {
        const T t = A(j, kk); A(j, kk) = A(kp, j); A(kp, j) = t;
      }
      if (threadIdx.x == 0) {
        const T t = A(kk, kk); A(kk, kk) = A(kp, kp); A(kp, kp) = t;
        if (kstep == 2) { const T u = A(k + 1, k); A(k + 1, k) = A(kp, k); A(kp, k) = u; }
      }
      __syncthreads();
    }
    if (kstep == 1) {
      const T r1 = (T)1 / A(k, k);
      const int r = m - k - 1;
      const int rr = r * r;
      for (int idx = threadIdx.x; idx < rr; idx += NTHREADS) {
        const int ii = idx % r, jj = idx / r;
        if (ii >= jj) {
          const int i = k + 1 + ii, j = k + 1 + jj;
          A(i, j) -= r1 * A(i, k) * A(j, k);
        }
      }
      __syncthreads();
      for (int i = k + 1 + threadIdx.x; i < m; i += NTHREADS) A(i, k) *= r1;
      if (threadIdx.x == 0) piv[k] = (double)kp;
      __syncthreads();
    } else {
      if (k + 2 < m) {
        T d21 = A(k + 1, k);
        const T d11 = A(k + 1, k + 1) / d21, d22 = A(k, k) / d21;
        const T t = (T)1 / (d11 * d22 - (T)1);
        d21 = t / d21;
        T* wk = work;
        T* wk1 = work + m;
        for (int j = k + 2 + threadIdx.x; j < m; j += NTHREADS) {
          wk[j] = d21 * (d11 * A(j, k) - A(j, k + 1));
          wk1[j] = d21 * (d22 * A(j, k + 1) - A(j, k));
        }
        __syncthreads();
        const int r = m - k - 2;
        const int rr = r * r;
        for (int idx = threadIdx.x; idx < rr; idx += NTHREADS) {
          const int ii = idx % r, jj = idx / r;
          if (ii >= jj) {
            const int i = k + 2 + ii, j = k + 2 + jj;
            A(i, j) -= A(i, k) * wk[j] + A(i, k + 1) * wk1[j];
          }
        }
        __syncthreads();
        for (int j = k + 2 + threadIdx.x; j < m; j += NTHREADS) { A(j, k) = wk[j]; A(j, k + 1) = wk1[j]; }
      }
      if (threadIdx.x == 0) { piv[k] = (double)(-(kp + 1)); piv[k + 1] = (double)(-(kp + 1)); }
      __syncthreads();
    }
    k += kstep;
  }
  return true;
}

// Solve with the factorization of cta_sytrf_lower (the LAPACK sytrs
// "lower" algorithm), one warp, x in place.
template <class T, class V>
__device__ void warp_sytrs_lower(int m, const T* a, int lda, const double* piv, V* x) {
  const int lane = threadIdx.x & 31;
  auto A = [&](int i, int j) -> V { return (V)a[i + (int64_t)j * lda]; };
  int k = 0;
  while (k < m) {
    if (piv[k] >= 0.0) {
      const int kp = (int)piv[k];
      if (lane == 0 && kp != k) { const V t = x[k]; x[k] = x[kp]; x[kp] = t; }
      __syncwarp();
      const V xk = x[k];
      for (int i = k + 1 + lane; i < m; i += 32) x[i] -= A(i, k) * xk;
      __syncwarp();
      if (lane == 0) x[k] = xk / A(k, k);
      __syncwarp();
      k += 1;
    } else {
      const int kp = (int)(-piv[k]) - 1;
      if (lane == 0 && kp != k + 1) { const V t = x[k + 1]; x[k + 1] = x[kp]; x[kp] = t; }
      __syncwarp();
      const V xk = x[k], xk1 = x[k + 1];
      for (int i = k + 2 + lane; i < m; i += 32) x[i] -= A(i, k) * xk + A(i, k + 1) * xk1;
      __syncwarp();
      if (lane == 0) {
        const V akm1k = A(k + 1, k);
        const V akm1 = A(k, k) / akm1k, ak = A(k + 1, k + 1) / akm1k;
        const V denom = akm1 * ak - (V)1;
        const V bkm1 = xk / akm1k, bk = xk1 / akm1k;
        x[k] = (ak * bkm1 - bk) / denom;
        x[k + 1] = (akm1 * bk - bkm1) / denom;
      }
      __syncwarp();
      k += 2;
    }
  }
  k = m - 1;
  while (k >= 0) {
    if (piv[k] >= 0.0) {
      V s = 0;
      for (int i = k + 1 + lane; i < m; i += 32) s += A(i, k) * x[i];
      s = warp_sum(s);
      if (lane == 0) {
        x[k] -= s;
        const int kp = (int)piv[k];
        if (kp != k) { const V t = x[k]; x[k] = x[kp]; x[kp] = t; }
      }
      __syncwarp();
      k -= 1;
    } else {
      V s = 0, s1 = 0;
      for (int i = k + 1 + lane; i < m; i += 32) { s += A(i, k) * x[i]; s1 += A(i, k - 1) * x[i]; }
      s = warp_sum(s);
      s1 = warp_sum(s1);
      if (lane == 0) {
        x[k] -= s;
        x[k - 1] -= s1;
        const int kp = (int)(-piv[k]) - 1;
        if (kp != k) { const V t = x[k]; x[k] = x[kp]; x[kp] = t; }
      }
      __syncwarp();
      k -= 2;
    }
  }
}
