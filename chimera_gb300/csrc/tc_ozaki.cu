// FP64 products on the BF16 tensor cores (the FP64 form's DHT and
// mode-coupling products), by error-free slicing (K. Ozaki, T. Ogita,
// S. Oishi, S. M. Rump, Numer. Algorithms 59 (2012) 95-118).
//
// Each row of A and each column of B is scaled by a power of two to 62-bit
// fixed point and cut into 8 balanced base-256 digits, -128 .. 127 (the first
// one within +-64), which BF16 holds exactly.  A product of two digits is an
// integer below 2^14, and a sum of them that stays within 2^24 is exact in
// the tensor core's FP32 accumulator.  The digit pairs (i, j) of equal weight
// 256^-(i+j) share an accumulator: S_d = sum over k and i + j = d, for d =
// 0 .. 7 (36 pairs; the pairs past d = 7 lie below 2^-62 of the row's and
// column's largest elements).  Over 256 K values S_0 .. S_4 are at most 2^24
// whatever the digits are, so they are exact; S_5 .. S_7 are exact too unless
// nearly all digits are at their extremes, and then off by a few units of
// weight 2^-52 or less of the largest elements' product.
// The weighted sum of S_0 .. S_7 is formed in a 64-bit integer per output whose
// unit is 2^-(54 + D) of 2^(ea + eb), the bound of the row's times the column's
// elements (D = 8 - log2 of the K values, so that it cannot overflow), and
// rounded once to FP64 with integer instructions: GB300's FP64 pipe retires 2
// operations a clock and SM, a conversion there would take longer than the
// product.
//
// What it gives: the products of a field step at 2048 x 256 x 2 modes (33.4
// GFLOP) took 31.5 ms on the FP64 pipe (its peak); with these 1.3 and the slices
// 0.36.
//
// The error is one rounding of the result plus about half a unit, 2^-55 of
// the largest elements' product; the FP64 pipe's sum rounds K times
// (tests/test_zy_fp64_products_gpu.py compares both with longer sums).
//
// oz_split: the digits in the tensor-core operand layout (8-row
// x 16-byte core matrices), a block of 8 slices per (row tile, 16-wide K
// step).
// oz_kernel: persistent, one CTA per SM.  A tile of 128 rows x TNC columns and
// 256 K values takes four groups of MMAs, from the lowest weights up: S_6 S_7
// (15 pairs), S_4 S_5 (11), S_2 S_3 (7), S_0 S_1 (3).  A group has two
// accumulators of TNC <= 128 columns; groups take turns over two such TMEM
// buffers, so the tensor core runs one group while the row threads drain the
// one before it.  (All of d = 0 .. 3, then 4 .. 7 in four accumulators needs
// fewer operand loads, but at 128 columns it fills TMEM: nothing overlapped,
// and a tile took 1.2 times as long.)  A stage holds 8 slices of both operands:
// one K step of the first two groups, two of the third, four of the last, so
// every stage feeds 11 to 15 MMAs.
//   warps 0..15: the row threads (TMEM lane quarter w % 4, column quarter
//   w / 4), which drain the accumulators, combine and write;
//   warp 16 issues the MMAs, warp 17 the bulk copies, each as a whole warp
//   with one elected lane (as in umma_kernel, tc_umma.cu: a branch on a
//   thread's own index cost 134 clocks an MMA).  An instruction takes some 100
//   clocks to issue, the tensor core 64 for 128 columns, so the two weights of
//   a group share one of 256: 20 instructions a K step instead of 36.
// Every mbarrier wait has an iteration limit, after which the CTA records an
// error, writes NaN to its unfinished tiles, waits for its own copies and MMAs
// (again with a limit), frees its TMEM and returns.
//
// A row or column holding an infinity or a NaN has no fixed-point form; its
// outputs are summed directly (slow_dot), with the FP64 kernel's result.
#include <cuda_bf16.h>

#include <type_traits>

#include "tc_gemm.cuh"
#include "tc_ozaki.cuh"
#include "tc_ptx.cuh"

using namespace chm;

namespace {

constexpr int NS = 8;             // slices
constexpr int TH = 128;           // rows per tile
constexpr int KB = 16;            // K step
constexpr int kChunk = 16;        // K steps per accumulation (256 K values)
constexpr int kRowWarps = 16;     // a TMEM lane quarter and a column quarter each
constexpr int kRowThreads = 32 * kRowWarps;
constexpr int kMmaWarp = kRowWarps, kLoadWarp = kRowWarps + 1;
constexpr int kThreads = kRowThreads + 128;  // five warpgroups
// registers: launched with 96 a thread (640 x 96 = 61440); the issuing
// warpgroup keeps 32 and the four of the row threads, which hold 32 outputs
// each, take 112 (128 x 32 + 512 x 112 = 61440)
constexpr int kIssueRegs = 32, kRowRegs = 112;
constexpr int kColGroups = kRowWarps / 4;
constexpr int kMaxStages = 6;
constexpr uint32_t kASlice = TH * KB * 2;  // bytes of one A slice block
constexpr uint32_t kSmemMax = 200 * 1024;
constexpr int kNonFinite = 1 << 20;  // row / column exponent: holds Inf or NaN
constexpr long long kSpin = 1LL << 20;

__device__ int g_oz_error;

// ----------------------------------------------------------------------
// operand slicing
// ----------------------------------------------------------------------
struct SplitSet {
  const double *X[kOzMaxProblems];
  uint8_t *T[kOzMaxProblems];
  int *E[kOzMaxProblems];
  int reflect[kOzMaxProblems];
};

// a 2^(62 - (E - 1022)) rounded to an integer (|a| < 2^(E - 1022)), plus the
// digits' bias: byte 7 - s of the result is digit s + 128
__device__ __forceinline__ unsigned long long fixed62(double a, int E) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(a);
  const int e = (int)((b >> 52) & 0x7ff);
  unsigned long long m = b & 0xfffffffffffffULL;
  if (e) m |= 1ULL << 52;
  const int sh = 9 - (E - (e ? e : 1));
  unsigned long long q;
  if (sh >= 0) q = m << sh;
  else if (sh > -56) q = (m + (1ULL << (-sh - 1))) >> -sh;
  else q = 0;
  if (b >> 63) q = 0ULL - q;
  return q + 0x8080808080808080ULL;
}

// the 8 slices of 8 consecutive K values, 16 bytes per slice at p + s stride
__device__ __forceinline__ void store_slices(const unsigned long long (&u)[8], uint8_t *p, uint32_t stride) {
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float f[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t word = s < 4 ? (uint32_t)(u[2 * q + h] >> 32) : (uint32_t)u[2 * q + h];
        // 2^23 + byte as a float, less 2^23 + 128: the digit
        f[h] = __uint_as_float(__byte_perm(word, 0x4B000000u, 0x7440u | (3 - (s & 3)))) - 8388736.0f;
      }
      w[q] = __byte_perm(__float_as_uint(f[0]), __float_as_uint(f[1]), 0x7632);  // BF16 pair
    }
    *reinterpret_cast<uint4 *>(p + s * stride) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// 32 rows (block bx) of one A plane, all K: the rows' largest exponents, then
// the slices (the second read comes from L1 / L2).  HBM bound: 8 B read and
// 16 B written per element.
__device__ __forceinline__ void split_rows(const SplitSet &J, int job, int bx, int M, int K, int nkb) {
  __shared__ int emax[8][32];
  const int r = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int gm = bx * 32 + r;
  const bool ok = gm < M;
  long long src = gm;
  bool neg = false;
  if (J.reflect[job] && ok) {
    const int x = gm >> 1;
    src = 2 * (long long)(x == 0 ? 0 : (M >> 1) - x) + (gm & 1);
    neg = (gm & 1) == 0;
  }
  const double *a = J.X[job] + src;
  int e = 0;
  if (ok)
    for (int k = g; k < K; k += 8) e = max(e, __double2hiint(__ldg(a + (long long)k * M)) & 0x7fffffff);
  emax[g][r] = e;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 8; ++q) e = max(e, emax[q][r]);
  e >>= 20;
  const bool fin = e < 0x7ff;
  const int E = max(e, 1);
  if (g == 0) J.E[job][gm] = fin ? E : kNonFinite;
  const int mt = gm / TH, rt = gm % TH;
  uint8_t *T = J.T[job] + (long long)mt * nkb * NS * kASlice + (rt >> 3) * 256 + (rt & 7) * 16;
  for (int kg = g; kg < 2 * nkb; kg += 8) {
    unsigned long long u[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int k = kg * 8 + q;
      double v = (ok && fin && k < K) ? __ldg(a + (long long)k * M) : 0.0;
      u[q] = fixed62(neg ? -v : v, E);
    }
    store_slices(u, T + (long long)(kg >> 1) * NS * kASlice + (kg & 1) * 128, kASlice);
  }
}

// 8 columns (block bx) of one B matrix, a warp per column
__device__ __forceinline__ void split_cols(const SplitSet &J, int job, int bx, int N, int K, int nkb, int tnc) {
  const int lane = threadIdx.x & 31;
  const int n = bx * 8 + (threadIdx.x >> 5);
  const bool ok = n < N;
  const double *b = J.X[job] + (long long)n * K;
  int e = 0;
  if (ok)
    for (int k = lane; k < K; k += 32) e = max(e, __double2hiint(__ldg(b + k)) & 0x7fffffff);
  e = __reduce_max_sync(0xffffffffu, e) >> 20;
  const bool fin = e < 0x7ff;
  const int E = max(e, 1);
  if (lane == 0) J.E[job][n] = fin ? E : kNonFinite;
  const uint32_t slice = (uint32_t)tnc * KB * 2;
  const int nt = n / tnc, nn = n % tnc;
  uint8_t *T = J.T[job] + (long long)nt * nkb * NS * slice + (nn >> 3) * 256 + (nn & 7) * 16;
  for (int kg = lane; kg < 2 * nkb; kg += 32) {
    unsigned long long u[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int k = kg * 8 + q;
      u[q] = fixed62((ok && fin && k < K) ? __ldg(b + k) : 0.0, E);
    }
    store_slices(u, T + (long long)(kg >> 1) * NS * slice + (kg & 1) * 128, slice);
  }
}

// one launch for the batch's operands: na blocks for the A planes (ax per
// plane), then the B matrices' (bx each)
__global__ void __launch_bounds__(256) oz_split(const __grid_constant__ SplitSet A, const __grid_constant__ SplitSet B,
                                                int na, int ax, int bx, int M, int N, int K, int nkb, int tnc) {
  const int b = (int)blockIdx.x;
  if (b < na) split_rows(A, b / ax, b % ax, M, K, nkb);
  else split_cols(B, (b - na) / bx, (b - na) % bx, N, K, nkb, tnc);
}

// ----------------------------------------------------------------------
// product
// ----------------------------------------------------------------------
struct OzProb {
  const uint8_t *TA, *TB;
  const int *EA, *EB;
  const double *A, *B;
  double *C;
  const double *fac;
  int reflect;
};
struct OzBatch {
  OzProb p[kOzMaxProblems];
};
struct OzArgs {
  int M, N, K, nkb;
  int tnc, ntn, nmt, ntiles;
  int stages;
  int dlt;  // D of the integer sum's unit
  const double2 *shift;
};

// 4 consecutive accumulator columns of this warp's 32 TMEM lanes
__device__ __forceinline__ void tmem_ld4(uint32_t (&v)[4], uint32_t taddr) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(taddr));
}

// (a denormal result or an overflow)
__device__ __noinline__ double round_rare(unsigned long long r, int e, bool neg) {
  const double v = scalbn((double)r, e - 1075);
  return neg ? -v : v;
}

// t 2^ex rounded to FP64
__device__ __forceinline__ double round_sum(long long t, int ex) {
  if (t == 0) return 0.0;
  const bool neg = t < 0;
  const unsigned long long x = neg ? 0ULL - (unsigned long long)t : (unsigned long long)t;
  const int n = __clzll((long long)x);
  const unsigned long long y = x << n;
  const int e = 1023 + 63 - n + ex;
  const unsigned long long r = (y >> 11) + ((y >> 10) & 1);  // 2^52 .. 2^53
  if (e < 1 || e > 2045) return round_rare(r, e, neg);
  const unsigned long long b = ((unsigned long long)(e - 1) << 52) + r;
  return __longlong_as_double((long long)(b | ((unsigned long long)neg << 63)));
}

// K steps of a stage and slices of a K step of each group
__device__ __forceinline__ int group_ksteps(int g) { return g < 2 ? 1 : 2 * (g - 1); }
__device__ __forceinline__ uint32_t group_slices(int g) { return 8 - 2 * g; }

// the sum of K values k0 .. k1 - 1 of one output in FP64 (operands with an infinity
// or a NaN)
__device__ __noinline__ double slow_dot(const OzProb *Q, const OzArgs *A, int gm, int n, int k0) {
  const int M = A->M, K = A->K;
  if (gm >= M || n >= A->N) return 0.0;
  long long src = gm;
  double sg = 1.0;
  if (Q->reflect) {
    const int x = gm >> 1;
    src = 2 * (long long)(x == 0 ? 0 : (M >> 1) - x) + (gm & 1);
    if ((gm & 1) == 0) sg = -1.0;
  }
  double s = 0.0;
  for (int k = k0; k < min(K, k0 + kChunk * KB); ++k)
    s = fma(sg * Q->A[src + (long long)k * M], Q->B[k + (long long)n * K], s);
  return s;
}

// CH: columns a row thread may hold, at least TNC / kColGroups
template <bool SHIFT, int CH>
__global__ void __launch_bounds__(kThreads, 1)
    oz_kernel(const __grid_constant__ OzBatch P, const __grid_constant__ OzArgs A) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], dfull[2], dempty[2], done;
  __shared__ uint32_t tmem_base;
  __shared__ int fail;
  const int warp = threadIdx.x >> 5;
  const int tnc = A.tnc, nkb = A.nkb, stages = A.stages;
  const int nchunk = (nkb + kChunk - 1) / kChunk;
  const uint32_t b_slice = (uint32_t)tnc * KB * 2;
  const uint32_t stage_bytes = NS * (kASlice + b_slice);
  volatile int *vfail = &fail;
  // this CTA's tiles; the column tile varies fastest, so CTAs running at once
  // share A rows in L2
  const int my_tiles = A.ntiles > (int)blockIdx.x ? (A.ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&dfull[b], 1);
      mbar_init(&dempty[b], kRowThreads);
    }
    mbar_init(&done, 1);
    fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);  // (uniform over the warp)
  const uint32_t smem0 = __shfl_sync(0xffffffffu, smem_u32(smem), 0);

  if (warp >= kRowWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kIssueRegs));
    if (warp == kLoadWarp) {
      const bool lead = elect_one();
      int s = 0, round = 0;
      bool ok = true;
      for (int i = 0; i < my_tiles && ok; ++i) {
        const int t = (int)blockIdx.x + i * (int)gridDim.x;
        const int rest = t % (A.nmt * A.ntn), prob = t / (A.nmt * A.ntn);
        const int mt = rest / A.ntn, nt = rest % A.ntn;
        const uint8_t *TA = P.p[prob].TA + (long long)mt * nkb * NS * kASlice;
        const uint8_t *TB = P.p[prob].TB + (long long)nt * nkb * NS * b_slice;
        for (int cg = 0; cg < 4 * nchunk && ok; ++cg) {
          const int kb0 = (cg >> 2) * kChunk, kb1 = min(nkb, kb0 + kChunk);
          const int ks = group_ksteps(cg & 3);
          const uint32_t ns = group_slices(cg & 3);
          for (int kb = kb0; kb < kb1; kb += ks) {
            const bool go = !*vfail && (round == 0 || mbar_wait(&empty[s], (uint32_t)(round - 1) & 1u, kSpin));
            if (!__all_sync(0xffffffffu, go)) {
              *vfail = 1;
              if (lead) atomicCAS(&g_oz_error, 0, 13);
              ok = false;
              break;
            }
            if (lead) {
              const uint32_t st = smem0 + (uint32_t)s * stage_bytes, bar = smem_u32(&full[s]);
              const int n = min(ks, kb1 - kb);
              mbar_expect_tx(&full[s], (uint32_t)n * ns * (kASlice + b_slice));
              for (int q = 0; q < n; ++q) {
                bulk_g2s(st + (uint32_t)q * ns * kASlice, TA + (long long)(kb + q) * NS * kASlice, ns * kASlice,
                         bar);
                bulk_g2s(st + NS * kASlice + (uint32_t)q * ns * b_slice,
                         TB + (long long)(kb + q) * NS * b_slice, ns * b_slice, bar);
              }
            }
            __syncwarp();
            if (++s == stages) s = 0, ++round;
          }
        }
      }
      // the copies issued last on every stage land before the CTA goes on
      for (int q = 0; q < stages; ++q) {
        const int last = q < s ? round : round - 1;
        if (last >= 0 && !mbar_wait(&full[q], (uint32_t)last & 1u, kSpin) && lead) atomicCAS(&g_oz_error, 0, 15);
      }
    } else if (warp == kMmaWarp) {
      const bool lead = elect_one();
      const uint32_t idesc = idesc_bf16(TH, tnc), idesc2 = idesc_bf16(TH, 2 * tnc);
      const uint32_t dhi = (uint32_t)(smem_desc<KB>(0) >> 32), bs = b_slice >> 4;
      long long lim = kSpin;
      int s = 0, round = 0, u = 0;
      bool ready = false;  // stage s polled complete
      // (a time-out changes no control flow: see umma_kernel)
      auto wait = [&](uint64_t *bar, int phase) {
        if (!mbar_wait(bar, (uint32_t)phase & 1u, lim)) {
          lim = 0;
          *vfail = 1;
        }
      };
      for (int i = 0; i < my_tiles; ++i)
        for (int cg = 0; cg < 4 * nchunk; ++cg, ++u) {
          const int kb0 = (cg >> 2) * kChunk, kb1 = min(nkb, kb0 + kChunk);
          const int grp = cg & 3, ks = group_ksteps(grp), b = u & 1, use = u >> 1;
          if (use > 0) wait(&dempty[b], use - 1);
          const uint32_t d0 = tmem + (uint32_t)(2 * b * tnc), d1 = d0 + (uint32_t)tnc;
          for (int kb = kb0; kb < kb1; kb += ks) {
            if (!ready) wait(&full[s], round);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t st = smem0 + (uint32_t)s * stage_bytes;
            const uint32_t alo = (uint32_t)smem_desc<KB>(st), blo = (uint32_t)smem_desc<KB>(st + NS * kASlice);
            uint64_t *const freed = &empty[s];
            if (++s == stages) s = 0, ++round;
            ready = mbar_test(&full[s], (uint32_t)round & 1u);
            // (the first K step overwrites the accumulators)
            const uint32_t more = kb != kb0;
            // the pairs (i, W - i) and (i, W + 1 - i) of the group's two weights
            // W = 6 - 2 grp (into d0) and W + 1 (into d1) of one K step: one
            // MMA of 2 TNC columns, the slices W - i and W + 1 - i of B being
            // neighbours in shared memory as d0 and d1 are in TMEM
            auto step = [&](auto wt, int q, uint32_t acc) {
              constexpr int W = decltype(wt)::value;
              const uint32_t a = alo + (uint32_t)q * (W + 2) * (kASlice >> 4), bb = blo + (uint32_t)q * (W + 2) * bs;
#pragma unroll
              for (int i = 0; i <= W; ++i)
                umma_bf16<kDiscard>(d0, a + i * (kASlice >> 4), bb + (W - i) * bs, dhi, idesc2, i == 0 ? acc : 1u);
              umma_bf16<kDiscard>(d1, a + (W + 1) * (kASlice >> 4), bb, dhi, idesc, 1u);
            };
            if (lead) {
              const int n = min(ks, kb1 - kb);
              if (grp == 0) step(std::integral_constant<int, 6>{}, 0, more);
              else if (grp == 1) step(std::integral_constant<int, 4>{}, 0, more);
              else if (grp == 2)
                for (int q = 0; q < n; ++q) step(std::integral_constant<int, 2>{}, q, more | (q > 0));
              else
                for (int q = 0; q < n; ++q) step(std::integral_constant<int, 0>{}, q, more | (q > 0));
              umma_commit(freed);
              if (kb + ks >= kb1) umma_commit(&dfull[b]);
            }
            __syncwarp();
          }
        }
      if (lead) umma_commit(&done);
      if (lim == 0 && lead) atomicCAS(&g_oz_error, 0, 11);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRowRegs));
    const int ncol = tnc / kColGroups;  // this thread's columns (a multiple of 4)
    const int col0 = (warp >> 2) * ncol;
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)col0;
    const int row = (warp & 3) * 32 + (threadIdx.x & 31);
    long long t64[CH];  // the integer sums, then the values' bits
    int u = 0;
    bool ok = true;
    const int dlt = A.dlt;
    // waits for the next group; its first accumulator's address, 0 on a time-out
    auto ready = [&]() -> uint32_t {
      const int b = u & 1;
      const bool got = !*vfail && mbar_wait(&dfull[b], (uint32_t)(u >> 1) & 1u, kSpin) && !*vfail;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      ok = __all_sync(0xffffffffu, got) != 0;
      return lane_base + (uint32_t)(2 * b * tnc);
    };
    auto release = [&]() {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive(&dempty[u & 1]);
      ++u;
    };
    // f(column, S_W, S_W+1) over this thread's columns of the group
    auto drain = [&](uint32_t ta, auto f) {
#pragma unroll
      for (int g = 0; g < CH / 4; ++g)
        if (g * 4 < ncol) {
          uint32_t v0[4], v1[4];
          tmem_ld4(v0, ta + (uint32_t)(g * 4));
          tmem_ld4(v1, ta + (uint32_t)(tnc + g * 4));
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 4; ++j)
            f(g * 4 + j, __float2int_rn(__uint_as_float(v0[j])), __float2int_rn(__uint_as_float(v1[j])));
        }
    };
    int i = 0;
    for (; i < my_tiles && ok; ++i) {
      const int t = (int)blockIdx.x + i * (int)gridDim.x;
      const int rest = t % (A.nmt * A.ntn), prob = t / (A.nmt * A.ntn);
      const int mt = rest / A.ntn, nt = rest % A.ntn;
      const OzProb &Q = P.p[prob];
      const int gm = mt * TH + row;
      const bool rok = gm < A.M;
      const int ea = Q.EA[gm];
      const int n0 = nt * tnc + col0;
      // the exponents of this warp's columns, one to a lane
      const int lane = threadIdx.x & 31, ebl = lane < ncol ? __ldg(Q.EB + n0 + lane) : 0;
      double2 sh = make_double2(1.0, 0.0);
      if (SHIFT && rok) sh = A.shift[gm >> 1];
      for (int c = 0; c < nchunk; ++c) {
        uint32_t ta = ready();
        if (!ok) break;
        {  // S_6, S_7: (S_6 + S_7 / 256) 2^(D - 6), rounded
          const int rs = 6 - dlt, half = 1 << (rs - 1);
          drain(ta, [&](int j, int s6, int s7) { t64[j] = (s6 + ((s7 + 128) >> 8) + half) >> rs; });
        }
        release();
        ta = ready();
        if (!ok) break;
        {
          const int m4 = 1 << (10 + dlt), m5 = 1 << (2 + dlt);
          drain(ta, [&](int j, int s4, int s5) { t64[j] += (long long)s4 * m4 + (long long)s5 * m5; });
        }
        release();
        ta = ready();
        if (!ok) break;
        {
          const int m2 = 1 << (26 + dlt), m3 = 1 << (18 + dlt);
          drain(ta, [&](int j, int s2, int s3) { t64[j] += (long long)s2 * m2 + (long long)s3 * m3; });
        }
        release();
        ta = ready();
        if (!ok) break;
        // |S_0| <= 2^20, |S_1| <= 2^22: 256 S_0 + S_1 fits 32 bits
        drain(ta, [&](int j, int s0, int s1) {
          t64[j] += (long long)((unsigned long long)(long long)(s0 * 256 + s1) << (34 + dlt));
        });
        release();
#pragma unroll
        for (int j = 0; j < CH; ++j)
          if (j < ncol) {
            const int eb = __shfl_sync(0xffffffffu, ebl, j);
            double r = round_sum(t64[j], ea + eb - 2098 - dlt);
            if (max(ea, eb) >= kNonFinite) r = slow_dot(&Q, &A, gm, n0 + j, c * kChunk * KB);
            t64[j] = __double_as_longlong(r);
          }
        // the tile's values from registers, while the tensor core goes on
#pragma unroll
        for (int j = 0; j < CH; ++j)
          if (j < ncol) {
            const int n = n0 + j;
            const bool in = rok && n < A.N;
            double *pc = Q.C + gm + (long long)n * A.M;
            double x = __longlong_as_double(t64[j]);
            if (c > 0 && in) x += *pc;
            if (SHIFT && c == nchunk - 1) {
              // rows 2x (re) and 2x + 1 (im) sit in adjacent lanes
              const double other = __shfl_xor_sync(0xffffffffu, x, 1);
              x = (row & 1) ? other * sh.y + x * sh.x : x * sh.x - other * sh.y;
              if (Q.fac && in) x *= Q.fac[(gm >> 1) + (long long)(A.M >> 1) * n];
            }
            if (in) *pc = x;
          }
      }
    }
    if (!ok) {
      // the tiles not written read as NaN, so a caller that polls no status
      // (the FP64 entry points have none) does not go on with stale values
      *vfail = 1;
      atomicCAS(&g_oz_error, 0, 14);
      for (--i; i < my_tiles; ++i) {
        const int t = (int)blockIdx.x + i * (int)gridDim.x;
        const int rest = t % (A.nmt * A.ntn), gm = rest / A.ntn * TH + row;
        double *C = P.p[t / (A.nmt * A.ntn)].C;
        for (int j = 0; j < ncol; ++j) {
          const int n = rest % A.ntn * tnc + col0 + j;
          if (gm < A.M && n < A.N) C[gm + (long long)n * A.M] = __longlong_as_double(0x7ff8000000000000LL);
        }
      }
    }
  }
  __syncthreads();
  // every MMA complete before the TMEM is freed
  if (!mbar_wait(&done, 0, kSpin) && threadIdx.x == 0) atomicCAS(&g_oz_error, 0, 12);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

inline i64 rup(i64 a, i64 b) { return (a + b - 1) / b * b; }

inline i64 plane_bytes(i64 rows, i64 K) { return rup(2 * NS * rows * rup(K, KB), 256) + rup(4 * rows, 256); }

// column-tile width: the widest one (less shared-memory traffic per MMA),
// narrowed while the batch has fewer tiles than the GPU has SMs
int tile_width(int N, i64 row_tiles) {
  const int Np = tc_np(N);
  int w = tc_tile_cols(N);
  for (int c = w - 16; c >= 32; c -= 16)
    if (Np % c == 0 && row_tiles * (Np / w) < sm_count()) w = c;
  return w;
}

}  // namespace

namespace chm {

i64 oz_ws_bytes(i64 M, i64 N, i64 K, i64 nA, i64 nB) {
  return nA * plane_bytes(rup(M, TH), K) + nB * plane_bytes(tc_np((int)N), K) + 256;
}

// (every size the index arithmetic holds; from 16 x 4 to 4096 x 512 grids the
// transform with this product was never slower than on the FP64 pipe: 40.2
// against 40.2 us at 512 x 4, 55.9 against 104 at 512 x 64, 2 modes)
bool oz_takes(i64 M, i64 N, i64 K, int count) {
  return M % 2 == 0 && M < (1 << 30) && N <= 65536 && K < (1 << 20) && count > 0;
}

int oz_gemm_launch(const OzProblem *p, int count, int M, int N, int K, const double2 *shift, void *ws,
                   i64 ws_bytes, cudaStream_t st) {
  SplitSet JA, JB;
  OzBatch ob;
  int ia[kOzMaxProblems], ib[kOzMaxProblems], nA = 0, nB = 0;
  for (int i = 0; i < count; ++i) {
    int a = 0, b = 0;
    while (a < nA && !(JA.X[a] == p[i].A && JA.reflect[a] == p[i].reflect)) ++a;
    if (a == nA) {
      JA.X[a] = p[i].A;
      JA.reflect[a] = p[i].reflect;
      ++nA;
    }
    while (b < nB && JB.X[b] != p[i].B) ++b;
    if (b == nB) JB.X[nB++] = p[i].B;
    ia[i] = a;
    ib[i] = b;
  }
  if (!ws || oz_ws_bytes(M, N, K, nA, nB) > ws_bytes) {
    set_error("fp64 product: workspace too small for the operand slices");
    return CHM_ERR_WS;
  }
  const int nkb = (int)(rup(K, KB) / KB), nmt = (int)(rup(M, TH) / TH), Np = tc_np(N);
  OzArgs A{};
  A.M = M;
  A.N = N;
  A.K = K;
  A.nkb = nkb;
  A.nmt = nmt;
  A.tnc = tile_width(N, (i64)nmt * count);
  A.ntn = Np / A.tnc;
  A.ntiles = count * nmt * A.ntn;
  A.dlt = 8;
  for (int k = 1; k < (K < kChunk * KB ? K : kChunk * KB); k *= 2) --A.dlt;
  if (A.dlt > 4) A.dlt = 4;
  A.shift = shift;
  const uint32_t stage = NS * (kASlice + (uint32_t)A.tnc * KB * 2);
  A.stages = (int)(kSmemMax / stage);
  if (A.stages > kMaxStages) A.stages = kMaxStages;
  char *c = reinterpret_cast<char *>(rup(reinterpret_cast<i64>(ws), 256));
  auto take = [&](i64 rows, uint8_t **T, int **E) {
    *T = reinterpret_cast<uint8_t *>(c);
    *E = reinterpret_cast<int *>(c + rup(2 * NS * rows * nkb * KB, 256));
    c += plane_bytes(rows, K);
  };
  for (int a = 0; a < nA; ++a) take((i64)nmt * TH, &JA.T[a], &JA.E[a]);
  for (int b = 0; b < nB; ++b) take(Np, &JB.T[b], &JB.E[b]);
  for (int i = 0; i < count; ++i)
    ob.p[i] = OzProb{JA.T[ia[i]], JB.T[ib[i]], JA.E[ia[i]], JB.E[ib[i]], p[i].A, p[i].B, p[i].C, p[i].fac,
                     p[i].reflect};
  const int ax = nmt * TH / 32, bx = Np / 8;
  oz_split<<<(unsigned)(nA * ax + nB * bx), 256, 0, st>>>(JA, JB, nA * ax, ax, bx, M, N, K, nkb, A.tnc);
  count_launch();
  const int smem = (int)(stage * A.stages) + 1024;
  const int grid = A.ntiles < sm_count() ? A.ntiles : sm_count();
  // a row thread's columns, unrolled: the code for the 32 of a wide tile, fetched
  // once for a single narrow one, took most of its time (K = 64, 8 columns: 28 us,
  // 13.5 so; the columns' exponents one after the other from L2 the rest)
  const int ncol = A.tnc / kColGroups;
  void (*kern)(const OzBatch, const OzArgs);
  if (shift) kern = ncol <= 8 ? oz_kernel<true, 8> : ncol <= 16 ? oz_kernel<true, 16> : oz_kernel<true, 32>;
  else kern = ncol <= 8 ? oz_kernel<false, 8> : ncol <= 16 ? oz_kernel<false, 16> : oz_kernel<false, 32>;
  // (one limit for every size: calls from other threads may have others)
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax + 1024);
  kern<<<grid, kThreads, smem, st>>>(ob, A);
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("fp64 product: %s", cudaGetErrorString(e));
    return CHM_ERR_CUDA;
  }
  return CHM_OK;
}

int oz_status() {
  int v = 0, z = 0;
  cudaMemcpyFromSymbol(&v, g_oz_error, sizeof(int));
  if (v) cudaMemcpyToSymbol(g_oz_error, &z, sizeof(int));
  return v;
}

}  // namespace chm
