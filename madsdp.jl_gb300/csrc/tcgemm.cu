// Split-precision products on the tcgen05 tensor cores; see tcgemm.h.
#include "tcgemm.h"

#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "../../include/madsdp_gpu.h"

namespace tcg {
namespace {

constexpr int BM = 128, BK = 32;             // tile rows, K per stage (64 B of bf16)
constexpr int TILE = BM * BK * 2;            // bytes of one 128 x 32 bf16 slice tile of A
constexpr int kEpiThreads = 256;             // 8 epilogue warps
constexpr int kThreads = kEpiThreads + 64;   // and the TMA and the MMA warp
constexpr unsigned long long kWaitNs = 2000000000ull;  // bound of every wait (2 s)

// Slice pairs (t, u) with t + u <= NS - 1 in order of t + u; pairs of order
// s accumulate in group min(s, NG - 1).
template <int NS, int NG>
struct Pairs {
  static constexpr int N = NS * (NS + 1) / 2;
  int t[N], u[N], g[N], first[N];
  constexpr Pairs() : t(), u(), g(), first() {
    int p = 0;
    int seen[NG] = {};
    for (int s = 0; s < NS; ++s)
      for (int a = 0; a <= s; ++a) {
        t[p] = a;
        u[p] = s - a;
        g[p] = s < NG ? s : NG - 1;
        first[p] = seen[g[p]] ? 0 : 1;
        seen[g[p]] = 1;
        ++p;
      }
  }
};

struct Args {
  int64_t M, N, rpad_a, rpad_b, ldc, ldfix;
  int32_t tiles_n, lower, kblocks, chunk_kb, block_kb, U;
  // alpha: 0: 1, 1: -1, 2: other; beta: 0: 0, 1: 1, 2: other.  As integers: a
  // comparison of doubles holds the FP64 unit as long as a multiply-add
  int32_t alpha_kind, beta_kind;
  double alpha, beta;
  const int32_t* exa;
  const int32_t* exb;
  double* C;
  unsigned long long* fix;  // K split over blocks: fixed-point sums (else null, C is written)
  int* err;
};

// ---------------------------------------------------------------- PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ unsigned long long gtime() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait on a phase parity: false when the deadline passed first.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, unsigned long long deadline) {
  for (uint32_t it = 0;; ++it) {
    if (mbar_try(bar, parity)) return true;
    if ((it & 255u) == 255u && gtime() > deadline) return false;
  }
}
__device__ __forceinline__ void tma_load_2d(const CUtensorMap* map, uint32_t dst, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"((unsigned long long)map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major operand tile of 64 or 128 rows x 64 bytes with the 64-byte swizzle:
// 8-row groups 512 bytes apart, descriptor version 1, layout SWIZZLE_64B.
__device__ __forceinline__ unsigned long long smem_desc(uint32_t saddr) {
  unsigned long long d = (unsigned long long)((saddr & 0x3FFFFu) >> 4);
  d |= 1ull << 16;                 // leading byte offset (unused for swizzled K-major)
  d |= (unsigned long long)(512 >> 4) << 32;
  d |= 1ull << 46;
  d |= 4ull << 61;
  return d;
}
// kind::f16 instruction descriptor: FP32 accumulator, bf16 A and B, both
// K-major, N = BN, M = BM.
template <int BN>
constexpr uint32_t idesc() {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

template <int BN>
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, unsigned long long adesc, unsigned long long bdesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc<BN>()), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Eight columns of the calling warp's 32 tensor-memory lanes; the caller
// waits (tcgen05.wait::ld) before it uses them.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}

// v * 2^E for a fixed-point integer v, rounded once (to nearest even).  Built
// with integer instructions: GB300's 64-bit conversions and float64 adds share
// the narrow FP64 pipe (1.6 lanes per clock and SM).
__device__ __forceinline__ double fix_to_double(long long v, int E) {
  if (v == 0) return 0.0;
  const unsigned long long u = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  const int lz = __clzll((long long)u);
  const int ex = 1086 - lz + E;
  if (ex > 0 && ex < 2046) {
    const unsigned long long norm = u << lz;
    unsigned long long mant = norm >> 11;
    const unsigned rem = (unsigned)norm & 0x7FFu;
    mant += (rem > 0x400u || (rem == 0x400u && (mant & 1ull))) ? 1ull : 0ull;
    // the implicit bit (and a carry out of the rounding) adds to the exponent
    const unsigned long long bits = ((unsigned long long)(ex - 1) << 52) + mant;
    return __longlong_as_double((long long)(bits | ((unsigned long long)v & 0x8000000000000000ull)));
  }
  return scalbn(__ll2double_rn(v), E);
}

// v * 2^U rounded to nearest even for |v * 2^U| < 2^62, with integer
// instructions (as fix_to_double).
__device__ __forceinline__ long long float_to_fixed(float v, int U) {
  const int b = __float_as_int(v);
  const int field = (b >> 23) & 0xFF;
  if (field == 0) return 0;  // the accumulators hold no subnormal values above 2^-U / 2
  const unsigned mant = ((unsigned)b & 0x7FFFFFu) | 0x800000u;
  const int sh = field - 150 + U;
  long long r;
  if (sh >= 0) {
    r = (long long)((unsigned long long)mant << min(sh, 39));
  } else if (sh < -25) {
    r = 0;
  } else {
    const unsigned q = mant >> -sh, rem = mant & ((1u << -sh) - 1u), half = 1u << (-sh - 1);
    r = (long long)(q + ((rem > half || (rem == half && (q & 1u))) ? 1u : 0u));
  }
  return b < 0 ? -r : r;
}

// ---------------------------------------------------------------- the product
// One BM x BN output tile per thread block and a range of its K chunks
// (blockIdx.y).  Warp 8 issues the TMA loads, one thread of warp 9 the MMAs;
// warps 0-7 drain the accumulators of every finished chunk into 64-bit
// fixed-point sums kept in registers (row = tensor-memory lane, half of the
// columns per warp) while the TMA loads of the next chunk are in flight, and
// write C (or, when K is split over blocks, add to the fixed-point workspace)
// once at the end.
//
// What bounds it: for long K the slice tiles' traffic from L2 and the drain
// between chunks; for the K = 32 updates of the Cholesky factorization the
// latency of one load, one MMA group and the write-back.  A block per chunk,
// with 64-bit conversions, an integer atomic per entry and chunk and one load
// of C at a time, took 2.9 ms for the whole 1999 x 1999 x 5051 lower product
// (msdp_tc_gemm) against 0.94 ms with this and the slicing below; a single
// 128 x 64 x 32 tile takes 12.9 us.
template <int NS, int NG, int BN, int NST>
__global__ void __launch_bounds__(kThreads, 1)
    k_tc_gemm(const __grid_constant__ CUtensorMap ma, const __grid_constant__ CUtensorMap mb, const Args a) {
  constexpr Pairs<NS, NG> P{};
  constexpr int TILE_B = BN * BK * 2;
  constexpr int STAGE = NS * (TILE + TILE_B);
  constexpr uint32_t TCOLS = NG * BN <= 128 ? 128u : (NG * BN <= 256 ? 256u : 512u);
  constexpr int HALF = BN / 2;  // columns per epilogue warp
  static_assert(NG * BN <= 512, "tensor memory holds 512 columns");
  static_assert(HALF % 8 == 0 && TILE_B % 512 == 0, "column segments of 8, swizzle atoms of 512 bytes");

  extern __shared__ unsigned char smem_raw[];
  __shared__ int exb_s[BN];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sb = (raw + 1023u) & ~1023u;       // 1 KiB aligned stage buffers
  unsigned char* gb = smem_raw + (sb - raw);
  const uint32_t bar0 = sb + NST * STAGE;           // full[NST], empty[NST], done, drained
  uint32_t* tslot = (uint32_t*)(gb + NST * STAGE + 8 * (2 * NST + 2));
  volatile int* abort_flag = (volatile int*)(tslot + 1);
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (NST + s); };
  const uint32_t done = bar0 + 8u * (2 * NST), drained = done + 8u;
  auto tileA = [&](int s, int t) { return sb + (uint32_t)(s * STAGE + t * TILE); };
  auto tileB = [&](int s, int u) { return sb + (uint32_t)(s * STAGE + NS * TILE + u * TILE_B); };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tm = (int)(blockIdx.x / a.tiles_n), tn = (int)(blockIdx.x % a.tiles_n);
  // lower triangle only: tiles entirely above the diagonal have nothing to do
  if (a.lower && (int64_t)tn * BN > (int64_t)tm * BM + BM - 1) return;
  const int kb0 = (int)blockIdx.y * a.block_kb;
  const int nkb = min(a.block_kb, a.kblocks - kb0);
  const int nch = (nkb + a.chunk_kb - 1) / a.chunk_kb;

  if (threadIdx.x == kEpiThreads) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    mbar_init(done, 1);
    mbar_init(drained, kEpiThreads / 32);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == kEpiThreads / 32 + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                 "r"(TCOLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (threadIdx.x < BN) {
    const int64_t col = (int64_t)tn * BN + threadIdx.x;
    exb_s[threadIdx.x] = col < a.N ? a.exb[col] : 0;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;
  const unsigned long long deadline = gtime() + kWaitNs;

  if (warp == kEpiThreads / 32) {
    if (lane == 0) {
      // TMA producer: every slice of A and B for one 32-wide K block per stage
      int issued = 0;
      for (int i = 0; i < nkb; ++i) {
        const int s = i % NST;
        if (i >= NST && !mbar_wait(empty(s), ((i / NST) & 1) ^ 1, deadline)) {
          *abort_flag = 1;
          atomicExch(a.err, 1);
          break;
        }
        if (*abort_flag) break;
        mbar_expect_tx(full(s), STAGE);
        const int x = (kb0 + i) * BK;
#pragma unroll
        for (int t = 0; t < NS; ++t) {
          tma_load_2d(&ma, tileA(s, t), x, (int)(t * a.rpad_a + (int64_t)tm * BM), full(s));
          tma_load_2d(&mb, tileB(s, t), x, (int)(t * a.rpad_b + (int64_t)tn * BN), full(s));
        }
        issued = i + 1;
      }
      if (*abort_flag) {
        // let the copies already issued land before the block exits
        const unsigned long long d2 = gtime() + kWaitNs / 4;
        for (int i = max(0, issued - NST); i < issued; ++i) mbar_wait(full(i % NST), (i / NST) & 1, d2);
      }
    }
    __syncwarp();
  } else if (warp == kEpiThreads / 32 + 1) {
    if (lane == 0) {
      // MMA issuer: all slice pairs of the stage into their group accumulators
      bool ok = true;
      int i = 0;
      for (int c = 0; c < nch && ok; ++c) {
        // the accumulators of the chunk before have been read
        if (c > 0 && (!mbar_wait(drained, (c - 1) & 1, deadline) || *abort_flag)) {
          *abort_flag = 1;
          atomicExch(a.err, 4);
          ok = false;
          break;
        }
        tc_fence_after();
        const int i1 = min(nkb, (c + 1) * a.chunk_kb);
        for (bool first = true; i < i1; ++i, first = false) {
          const int s = i % NST;
          if (!mbar_wait(full(s), (i / NST) & 1, deadline) || *abort_flag) {
            *abort_flag = 1;
            atomicExch(a.err, 2);
            ok = false;
            break;
          }
          tc_fence_after();
#pragma unroll
          for (int p = 0; p < Pairs<NS, NG>::N; ++p) {
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk) {
              const unsigned long long ad = smem_desc(tileA(s, P.t[p]) + kk * 32);
              const unsigned long long bd = smem_desc(tileB(s, P.u[p]) + kk * 32);
              mma_bf16<BN>(tbase + (uint32_t)(P.g[p] * BN), ad, bd, (!first || !P.first[p] || kk > 0) ? 1u : 0u);
            }
          }
          mma_commit(empty(s));
        }
        if (ok) mma_commit(done);
      }
    }
    __syncwarp();
  } else {
    // epilogue: thread = one row of the tile (tensor-memory lane), columns
    // [c0, c0 + HALF)
    const int c0 = (warp >> 2) * HALF;
    const int64_t row = (int64_t)tm * BM + (warp & 3) * 32 + lane;
    const bool row_ok = row < a.M;
    // the last orders' sum, below 2^-7, is taken in units of 2^-38, which fit 32
    // bits, and what is below that (U > 38, K up to 256) by its remainder
    const int up = max(a.U - 38, 0);
    const float scale_hi = __int_as_float((127 + a.U - up) << 23), scale_lo = __int_as_float((127 + up) << 23);
    const uint32_t tw = tbase + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
    long long acc[HALF];
#pragma unroll
    for (int j = 0; j < HALF; ++j) acc[j] = 0;
    // narrow tiles: the old C is loaded while the MMAs run
    constexpr bool kEarly = HALF <= 32;
    double early[kEarly ? HALF : 1];
    if (kEarly && !a.fix && a.beta_kind) {
#pragma unroll
      for (int j = 0; j < (kEarly ? HALF : 0); ++j) {
        const int64_t col = (int64_t)tn * BN + c0 + j;
        early[j] = (row_ok && col < a.N && !(a.lower && row < col)) ? a.C[row + col * a.ldc] : 0.0;
      }
    }
    bool ok = true;
    for (int c = 0; c < nch; ++c) {
      ok = mbar_wait(done, c & 1, deadline) && !*abort_flag;
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        *abort_flag = 1;
        if (lane == 0) atomicExch(a.err, 3);
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int sg = 0; sg < HALF / 8; ++sg) {
        uint32_t v[NG][8];
#pragma unroll
        for (int g = 0; g < NG; ++g) tmem_ld8(tw + (uint32_t)(g * BN + sg * 8), v[g]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if constexpr (NG == 5) {
            // orders 0-3: integers below 2^24 times 2^-8g, gathered in units
            // of 2^-24 by wide multiply-adds; the rest as one 64-bit rounding
            // of v 2^U would give it: v has 24 bits, so the remainder of the
            // first conversion is exact
            long long tsum = (long long)__float2int_rn(__uint_as_float(v[0][j])) * (1 << 24);
            tsum += (long long)__float2int_rn(__uint_as_float(v[1][j]) * 0x1p8f) * (1 << 16);
            tsum += (long long)__float2int_rn(__uint_as_float(v[2][j]) * 0x1p16f) * (1 << 8);
            tsum += (long long)__float2int_rn(__uint_as_float(v[3][j]) * 0x1p24f);
            const float x = __uint_as_float(v[4][j]) * scale_hi;
            const int h = __float2int_rn(x);
            long long rest = h;
            if (up) rest = rest * (1ll << up) + __float2int_rn((x - __int2float_rn(h)) * scale_lo);
            acc[sg * 8 + j] += (tsum << (a.U - 24)) + rest;
          } else {
            // an exact integer and a remainder below 2^18
            acc[sg * 8 + j] += (long long)__float2int_rn(__uint_as_float(v[0][j])) << a.U;
            acc[sg * 8 + j] += float_to_fixed(__uint_as_float(v[NG - 1][j]), a.U);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0 && c + 1 < nch) mbar_arrive(drained);
    }
    if (ok && row_ok) {
      const int ea = a.exa[row] - a.U - 14;
#pragma unroll
      for (int sg = 0; sg < HALF / 8; ++sg) {
        const int64_t col0 = (int64_t)tn * BN + c0 + sg * 8;
        if (a.fix) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int64_t col = col0 + j;
            if (col < a.N && !(a.lower && row < col))
              atomicAdd(a.fix + row + col * a.ldfix, (unsigned long long)acc[sg * 8 + j]);
          }
          continue;
        }
        // eight independent loads of C before the first store
        double old[8];
        if (a.beta_kind) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int64_t col = col0 + j;
            if (kEarly) old[j] = early[kEarly ? sg * 8 + j : 0];
            else old[j] = (col < a.N && !(a.lower && row < col)) ? a.C[row + col * a.ldc] : 0.0;
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int64_t col = col0 + j;
          double d = fix_to_double(acc[sg * 8 + j], ea + exb_s[c0 + sg * 8 + j]);
          if (a.alpha_kind == 1) d = -d;
          else if (a.alpha_kind == 2) d = a.alpha * d;
          if (a.beta_kind == 1) d = old[j] + d;
          else if (a.beta_kind == 2) d = d + a.beta * old[j];
          if (col < a.N && !(a.lower && row < col)) a.C[row + col * a.ldc] = d;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kEpiThreads / 32 + 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(TCOLS) : "memory");
  }
}

// C = alpha * fix * 2^(ea + eb - U - 14) + beta * C
__global__ void k_finish(int64_t M, int64_t N, const long long* __restrict__ fix, int64_t ldfix,
                         const int32_t* __restrict__ exa, const int32_t* __restrict__ exb, int U, int alpha_kind,
                         double alpha, int beta_kind, double beta, double* C, int64_t ldc, int lower) {
  const int64_t total = M * N;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = idx / M, r = idx - c * M;
    if (lower && r < c) continue;
    double v = fix_to_double(fix[r + c * ldfix], exa[r] + exb[c] - U - 14);
    if (alpha_kind == 1) v = -v;
    else if (alpha_kind == 2) v = alpha * v;
    double* o = C + r + c * ldc;
    *o = beta_kind == 0 ? v : beta_kind == 1 ? v + *o : v + beta * *o;
  }
}

// ---------------------------------------------------------------- slicing
// Start of row R of a source; element k is at p[k * ks] or, with kmap, at
// p[a * rs + b * ks] for k -> (a, b).
__device__ __forceinline__ const double* src_row(const Source& s, int64_t R) {
  const uint32_t j = (uint32_t)R / (uint32_t)s.nr;
  const int64_t i = R - (int64_t)j * s.nr;
  return s.p + (int64_t)j * s.bs + (s.kmap ? 0 : i * s.rs);
}
__device__ __forceinline__ double src_at(const Source& s, const double* row, int64_t k) {
  if (s.kmap) {
    const int2 ab = s.kmap[k];
    const double v = row[ab.x * s.rs + ab.y * s.ks];
    return ab.x == ab.y ? v : v * 1.4142135623730951;
  }
  return row[k * s.ks];
}
// Row exponents, one warp per row (rows read along k).
__global__ void k_rowexp_warp(Source s, int64_t Rpad, int32_t* __restrict__ ex) {
  const int64_t R = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (R >= Rpad) return;
  int m = 0;
  if (R < s.rows) {
    const double* row = src_row(s, R);
#pragma unroll 4
    for (int64_t k = lane; k < s.K; k += 32) m = max(m, exp_field(src_at(s, row, k)));
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) ex[R] = row_exp(m);
}
// Row exponents of rows contiguous in memory: 32 rows per block, one per
// lane (256-byte loads), the 32 warps take every 32nd k.  One thread per row
// left 2000 rows to 8 SMs: 560 us for 1999 x 5051, against 30 us of copy time.
__global__ void __launch_bounds__(1024) k_rowexp_lanes(Source s, int64_t Rpad, int32_t* __restrict__ ex) {
  __shared__ int part[32][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t R = (int64_t)blockIdx.x * 32 + lane;
  int m = 0;
  if (R < s.rows) {
    const double* row = src_row(s, R);
#pragma unroll 8
    for (int64_t k = w; k < s.K; k += 32) m = max(m, exp_field(row[k * s.ks]));
  }
  part[w][lane] = m;
  __syncthreads();
  if (w == 0 && R < Rpad) {
#pragma unroll
    for (int q = 1; q < 32; ++q) m = max(m, part[q][lane]);
    ex[R] = row_exp(m);
  }
}

// Tiles of 32 rows x 64 k: read (through shared memory when rows are the
// contiguous direction), cut into NS slices, write K-major bf16 pairs (zeros
// in the padding).  Kpad is a multiple of 32: the second half of the last
// tile may lie outside.
template <int NS>
__global__ void __launch_bounds__(256) k_slice(Source s, int64_t Rpad, int64_t Kpad, const int32_t* __restrict__ ex,
                                              __nv_bfloat16* __restrict__ out) {
  __shared__ double tile[32][66];
  const int64_t r0 = (int64_t)blockIdx.x * 32, k0 = (int64_t)blockIdx.y * 64;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const bool along_k = s.kmap != nullptr || s.ks == 1 || s.rs != 1;
  if (along_k) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t R = r0 + ty + 8 * i;
      const double* row = R < s.rows ? src_row(s, R) : nullptr;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int64_t k = k0 + tx + 32 * h;
        tile[ty + 8 * i][tx + 32 * h] = (row && k < s.K) ? src_at(s, row, k) : 0.0;
      }
    }
  } else {
    const int64_t R = r0 + tx;
    const double* row = R < s.rows ? src_row(s, R) : nullptr;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int64_t k = k0 + ty + 8 * i;
      tile[tx][ty + 8 * i] = (row && k < s.K) ? row[k * s.ks] : 0.0;
    }
  }
  __syncthreads();
  if (k0 + 2 * tx >= Kpad) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t R = r0 + ty + 8 * i;
    const int e = R < s.rows ? ex[R] : 0;
    const double2 v = *(const double2*)&tile[ty + 8 * i][2 * tx];
    write_slice_pair<NS>(v.x, v.y, e, (uint32_t*)(out + R * Kpad + k0 + 2 * tx), Rpad * Kpad / 2);
  }
}

int64_t rup(int64_t x, int64_t a) { return (std::max<int64_t>(x, 1) + a - 1) / a * a; }

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  });
  return fn;
}

template <int NS, int BN, int NST>
constexpr int smem_bytes() {
  return NST * NS * (TILE + BN * BK * 2) + 1024 + 8 * (2 * NST + 2) + 16;
}

template <int NS, int NG, int BN, int NST>
cudaError_t launch(const Sliced& A, const Sliced& B, const Args& a, int64_t ntiles, int splits, cudaStream_t st) {
  constexpr int smem = smem_bytes<NS, BN, NST>();
  static_assert(smem <= 232448, "shared memory per block");
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(k_tc_gemm<NS, NG, BN, NST>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  });
  if (attr != cudaSuccess) return attr;
  const CUtensorMap& mb = BN == 64 ? B.map64 : BN == 96 ? B.map96 : B.map;
  k_tc_gemm<NS, NG, BN, NST><<<dim3((unsigned)ntiles, (unsigned)splits), kThreads, smem, st>>>(A.map, mb, a);
  return cudaGetLastError();
}

}  // namespace

int slices_of(Mode m) { return m == kMixed ? 3 : 7; }

int64_t sliced_bytes(int64_t rows, int64_t K, int ns) {
  const int64_t Rpad = rup(rows, BM), Kpad = rup(K, BK);
  return rup(ns * Rpad * Kpad * 2, 256) + rup(Rpad * 4, 256);
}

cudaError_t sliced_init(Sliced* s, void* mem, int64_t rows, int64_t K, int ns, cudaStream_t st, bool zero) {
  s->rows = rows;
  s->K = K;
  s->ns = ns;
  s->Rpad = rup(rows, BM);
  s->Kpad = rup(K, BK);
  s->s = (__nv_bfloat16*)mem;
  s->ex = (int32_t*)((char*)mem + rup(ns * s->Rpad * s->Kpad * 2, 256));
  if (zero) {
    const cudaError_t e = cudaMemsetAsync(mem, 0, (size_t)sliced_bytes(rows, K, ns), st);
    if (e != cudaSuccess) return e;
  }
  auto enc = encode_fn();
  if (!enc) return cudaErrorNotSupported;
  const cuuint64_t dims[2] = {(cuuint64_t)s->Kpad, (cuuint64_t)(ns * s->Rpad)};
  const cuuint64_t strides[1] = {(cuuint64_t)(s->Kpad * 2)};
  const cuuint32_t box[2] = {BK, BM}, box64[2] = {BK, 64}, box96[2] = {BK, 96};
  const cuuint32_t es[2] = {1, 1};
  if (ns * s->Rpad >= (int64_t)1 << 31) return cudaErrorInvalidValue;
  CUresult r = enc(&s->map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, s->s, dims, strides, box, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r == CUDA_SUCCESS)
    r = enc(&s->map64, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, s->s, dims, strides, box64, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r == CUDA_SUCCESS)
    r = enc(&s->map96, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, s->s, dims, strides, box96, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t slice(const Source& src, Sliced* d, cudaStream_t st) {
  if (src.rows != d->rows || src.K != d->K || src.nr <= 0) return cudaErrorInvalidValue;
  const bool along_k = src.kmap != nullptr || src.ks == 1 || src.rs != 1;
  if (along_k)
    k_rowexp_warp<<<(unsigned)((d->Rpad + 7) / 8), 256, 0, st>>>(src, d->Rpad, d->ex);
  else
    k_rowexp_lanes<<<(unsigned)(d->Rpad / 32), 1024, 0, st>>>(src, d->Rpad, d->ex);
  const dim3 grid((unsigned)(d->Rpad / 32), (unsigned)((d->Kpad + 63) / 64));
  switch (d->ns) {
    case 3: k_slice<3><<<grid, 256, 0, st>>>(src, d->Rpad, d->Kpad, d->ex, d->s); break;
    case 7: k_slice<7><<<grid, 256, 0, st>>>(src, d->Rpad, d->Kpad, d->ex, d->s); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

int64_t fix_bytes(int64_t M, int64_t N) { return std::max<int64_t>(M, 1) * std::max<int64_t>(N, 1) * 8; }

namespace {
// K per chunk: the order-0 group (1 pair) of the mixed mode is exact up to
// 1024; the order-3 group (4 pairs) of the FP64 mode up to 256.
int chunk_kb_of(Mode m) { return m == kMixed ? 32 : 8; }

// Column width of the tiles and the number of blocks K is split over.
struct Plan {
  int bn = 128, splits = 1;
};
int64_t tile_count(int64_t M, int64_t N, int bn, bool lower) {
  const int64_t tm = (M + BM - 1) / BM, tn = (N + bn - 1) / bn;
  if (!lower) return tm * tn;
  int64_t t = 0;
  for (int64_t i = 0; i < tm; ++i) t += std::min<int64_t>(tn, (i * BM + BM - 1) / bn + 1);
  return t;
}
// The plan with the smallest estimate of rounds of the 152 SMs times the time
// of a block: its chunks, a fixed part (pipeline fill, write-back), and the
// memset and finish pass when K is split.  Wider FP64 tiles reread A less
// but leave fewer blocks.
Plan plan(const Sliced& A, const Sliced& B, Mode mode, const Out& o) {
  const int ck = chunk_kb_of(mode);
  const int kblocks = (int)(A.Kpad / BK), nch = (kblocks + ck - 1) / ck;
  const double part = std::min(1.0, (double)kblocks / ck);  // a single short chunk
  Plan best;
  double best_t = INFINITY;
  const int widths[2] = {mode == kMixed ? 128 : 64, mode == kMixed ? 128 : 96};
  for (int w = 0; w < (mode == kMixed ? 1 : 2); ++w) {
    const int bn = widths[w];
    const double tc = part * (mode == kMixed ? 11.0 : bn == 64 ? 12.0 : 15.0);
    const double fixed = mode == kMixed ? 6.0 : bn == 64 ? 6.0 : 7.0;
    const int64_t tiles = tile_count(A.rows, B.rows, bn, o.lower);
    for (int sp = 1; sp <= (o.fix ? std::min(nch, 64) : 1); ++sp) {
      const int per = (nch + sp - 1) / sp;
      const int used = (nch + per - 1) / per;
      if (used != sp) continue;  // the same blocks with fewer splits
      const double rounds = (double)((tiles * sp + 151) / 152);
      const double t = rounds * (per * tc + fixed) + (sp > 1 ? 6.0 + 4e-6 * (double)(A.rows * B.rows) : 0.0);
      if (t < 0.97 * best_t) {
        best_t = t;
        best.bn = bn;
        best.splits = sp;
      }
    }
  }
  return best;
}
}  // namespace

bool needs_fix(const Sliced& A, const Sliced& B, Mode mode, const Out& o) { return plan(A, B, mode, o).splits > 1; }

cudaError_t gemm(const Sliced& A, const Sliced& B, Mode mode, const Out& o, cudaStream_t st, int64_t* launches) {
  const int ns = slices_of(mode);
  if (A.ns != ns || B.ns != ns || A.Kpad != B.Kpad || A.K != B.K) return cudaErrorInvalidValue;
  if (o.lower && A.rows != B.rows) return cudaErrorInvalidValue;
  const int64_t M = A.rows, N = B.rows;
  if (M == 0 || N == 0) return cudaSuccess;
  Args a{};
  a.M = M;
  a.N = N;
  a.rpad_a = A.Rpad;
  a.rpad_b = B.Rpad;
  a.kblocks = (int)(A.Kpad / BK);
  a.chunk_kb = chunk_kb_of(mode);
  const int nchunks = (a.kblocks + a.chunk_kb - 1) / a.chunk_kb;
  if (nchunks > 65535) return cudaErrorInvalidValue;
  const Plan pl = plan(A, B, mode, o);
  a.block_kb = (nchunks + pl.splits - 1) / pl.splits * a.chunk_kb;
  int lg = 0;
  while (((int64_t)1 << lg) < std::max<int64_t>(A.K, 2)) ++lg;
  a.U = std::max(24, std::min(46, 47 - lg));  // K is below 2^22 (grid of the slicing), so 47 - lg is at least 25
  a.exa = A.ex;
  a.exb = B.ex;
  a.C = o.C;
  a.ldc = o.ldc;
  a.alpha = o.alpha;
  a.beta = o.beta;
  a.alpha_kind = o.alpha == 1.0 ? 0 : o.alpha == -1.0 ? 1 : 2;
  a.beta_kind = o.beta == 0.0 ? 0 : o.beta == 1.0 ? 1 : 2;
  a.fix = pl.splits > 1 ? (unsigned long long*)o.fix : nullptr;
  a.ldfix = o.ldfix;
  a.err = o.err;
  a.lower = o.lower ? 1 : 0;
  const int64_t tm = (M + BM - 1) / BM, tn = (N + pl.bn - 1) / pl.bn;
  a.tiles_n = (int32_t)tn;
  const int64_t ntiles = tm * tn;
  if (ntiles >= ((int64_t)1 << 31)) return cudaErrorInvalidValue;
  cudaError_t e = cudaSuccess;
  if (a.fix) {
    e = cudaMemset2DAsync(o.fix, (size_t)(o.ldfix * 8), 0, (size_t)(M * 8), (size_t)N, st);
    if (e != cudaSuccess) return e;
  }
  // mixed: orders 0 | 1-2 (2 groups, 128-column tiles, 4 stages);
  // FP64: orders 0 | 1 | 2 | 3 | 4-6 (5 groups, 64- or 96-column tiles, 2 stages)
  e = mode == kMixed ? launch<3, 2, 128, 4>(A, B, a, ntiles, pl.splits, st)
      : pl.bn == 64  ? launch<7, 5, 64, 2>(A, B, a, ntiles, pl.splits, st)
                     : launch<7, 5, 96, 2>(A, B, a, ntiles, pl.splits, st);
  if (e != cudaSuccess) return e;
  if (launches) *launches += 1;
  if (a.fix) {
    const int64_t total = M * N;
    const unsigned grid = (unsigned)std::min<int64_t>((total + 255) / 256, 152 * 32);
    k_finish<<<grid, 256, 0, st>>>(M, N, o.fix, o.ldfix, A.ex, B.ex, a.U, a.alpha_kind, o.alpha, a.beta_kind, o.beta, o.C, o.ldc, a.lower);
    if (launches) *launches += 1;
    e = cudaGetLastError();
  }
  return e;
}

}  // namespace tcg

// ---------------------------------------------------------------- C ABI
// C = alpha op(A) op(B) + beta C on the tensor cores (include/madsdp_gpu.h).
extern "C" int msdp_tc_gemm(int32_t precision, int32_t transa, int32_t transb, int64_t M, int64_t N, int64_t K,
                            double alpha, const double* A, int64_t lda, const double* B, int64_t ldb, double beta,
                            double* C, int64_t ldc, int32_t lower, void* stream) {
  using namespace tcg;
  if (M < 0 || N < 0 || K < 0 || (M && !C) || ldc < std::max<int64_t>(M, 1)) return MSDP_ERR_INVALID_ARGUMENT;
  if (precision != MSDP_FP64 && precision != MSDP_MIXED) return MSDP_ERR_INVALID_ARGUMENT;
  if (lower && M != N) return MSDP_ERR_INVALID_ARGUMENT;
  if (M == 0 || N == 0) return MSDP_OK;
  if (K == 0 || (!A || !B)) return MSDP_ERR_INVALID_ARGUMENT;
  if (lda < (transa ? K : M) || ldb < (transb ? N : K)) return MSDP_ERR_INVALID_ARGUMENT;
  const Mode mode = precision == MSDP_MIXED ? kMixed : kFp64;
  const int ns = slices_of(mode);
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t ba = sliced_bytes(M, K, ns), bb = sliced_bytes(N, K, ns), bf = fix_bytes(M, N);
  char* mem = nullptr;
  if (cudaMalloc(&mem, (size_t)(ba + bb + bf + 256)) != cudaSuccess) return MSDP_ERR_OUT_OF_MEMORY;
  Sliced SA, SB;
  int* err = (int*)(mem + ba + bb + bf);
  int rc = MSDP_OK;
  cudaError_t e = sliced_init(&SA, mem, M, K, ns, st);
  if (e == cudaSuccess) e = sliced_init(&SB, mem + ba, N, K, ns, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(int), st);
  Source sa, sb;
  // A operand rows = rows of op(A): op(A)(r, k)
  sa.p = A; sa.rows = M; sa.K = K; sa.nr = M; sa.bs = 0;
  sa.rs = transa ? lda : 1; sa.ks = transa ? 1 : lda;
  // B operand rows = columns of op(B): op(B)(k, c)
  sb.p = B; sb.rows = N; sb.K = K; sb.nr = N; sb.bs = 0;
  sb.rs = transb ? 1 : ldb; sb.ks = transb ? ldb : 1;
  if (e == cudaSuccess) e = slice(sa, &SA, st);
  // op(A) op(A)': the rows of both operands are the same elements
  const bool same = A == B && M == N && sa.rs == sb.rs && sa.ks == sb.ks;
  if (e == cudaSuccess && !same) e = slice(sb, &SB, st);
  Out o;
  o.C = C; o.ldc = ldc; o.alpha = alpha; o.beta = beta; o.lower = lower != 0;
  o.fix = (long long*)(mem + ba + bb); o.ldfix = M; o.err = err;
  if (e == cudaSuccess) e = gemm(SA, same ? SA : SB, mode, o, st, nullptr);
  int herr = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) rc = MSDP_ERR_CUDA;
  else if (herr) rc = MSDP_ERR_CUDA;
  cudaFree(mem);
  return rc;
}
