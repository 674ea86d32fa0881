// FP64 products on the BF16 tensor cores (the FP64 form's DHT and
// mode-coupling products), by error-free slicing (K. Ozaki, T. Ogita,
// S. Oishi, S. M. Rump, Numer. Algorithms 59 (2012) 95-118).
//
// Each row of A and each column of B is scaled by a power of two to 70-bit
// fixed point and cut into 9 balanced base-256 digits, -128 .. 127 (the first
// one within +-64), which BF16 holds exactly.  A product of two digits is an
// integer below 2^14, and a sum of them that stays within 2^24 is exact in
// the tensor core's FP32 accumulator.  The digit pairs (i, j) of equal weight
// 256^-(i+j) share an accumulator: S_d = sum over k and i + j = d, for d =
// 0 .. 8 (45 pairs).  Over 256 K values S_0 .. S_4 are at most 2^24
// whatever the digits are, so they are exact.  S_5 and S_6 are exact where they end
// below 2^23 (a partial sum above 2^24 takes 67 % of the terms at their largest, and
// the others cannot bring it back that far); S_7 and S_8 may be off by a few units
// of 2^-68 of the largest elements' product.
// The weighted sum of S_0 .. S_8 is formed in integers (S_2 .. S_8 in 64 bits,
// S_0 and S_1 in 32 above them) in units of 2^-66 of 2^(ea + eb), the bound of
// the row's times the column's elements, and rounded once to FP64.  (GB300's FP64
// pipe retires 2 operations a clock and SM: a conversion of each S_d there would
// take longer than the product.)
//
// Error.  One rounding of the result (for each 256 K values) and what is left
// out: a unit, the operands' rounding and the pairs d >= 9, together 2^-66 of
// 2^(ea + eb) rms over random digits and at most (0.3 K + 2) 2^-65, K up to 256.
// That is relative to the row's and the column's largest elements, where a sum in
// FP64 is off by some 2^-55 of sum |a b| (its terms' roundings) and at most K 2^-53.
// Two things keep the first below the second:
// - Before they are cut, A(:, k) is multiplied by 2^s_k and B(k, :) divided by it,
//   2^s_k being the size of B's largest element for this k (oz_scale).  A spectrum
//   that falls over k times an operator that grows over it (the mode coupling of
//   a smooth field: Dp and Dm grow with kr) otherwise spends the fixed-point
//   form's upper digits on elements that do not meet: with 8 digits and no scaling
//   the error of a Gaussian profile's coupling was 1.1e-14 of the result's norm
//   where the FP64 pipe's is 7.5e-16; now it is 4.6e-17 (256 x 256, profile of 0.2
//   of the radius; for noise 4.8e-17, of the pipe 3.7e-16).
// - A tenth slice holds |a| and |b| in BF16 (rounded down), whose product is a
//   lower estimate of sum |a b| for every output.  Where it is below kGuard, 2^-12
//   of 2^(ea + eb), the output is summed again in FP64 (fp64_sums).  (Errors over
//   sum |a b| of outputs between 2^-12 and 2^-11, in units of 2^-53: 0.33 rms, 1.4
//   at most, of the FP64 sum 1.27 and 13; a factor of 2 lower 0.59 and 2.5, 1.33 and
//   8.4; K = 256, spectra falling by e^25.)  So are outputs whose S_5 or S_6 is 2^23
//   or more, and rows and columns holding an infinity or a NaN, which have no
//   fixed-point form.
//
// oz_scale: the s_k of each B matrix.  oz_split: the digits in the tensor-core
// operand layout (8-row x 16-byte core matrices), a block of 10 slices per (row
// tile, 16-wide K step): |x|, then the digits.
// oz_kernel: persistent, one CTA per SM.  A tile of 128 rows x TNC columns and
// 256 K values takes five groups of MMAs: S_7 S_8 (17 pairs), S_5 S_6 (13), S_3
// S_4 (9), S_2 and the estimate of sum |a b| (4), S_0 S_1 (3).  A group has two
// accumulators of TNC <= 128 columns; groups take turns over two such TMEM
// buffers, so the tensor core runs one group while the row threads drain the
// one before it.  A stage holds 9 slices of both operands: one K step of the
// first three groups, two of the fourth, four of the last.  What bounds it: a tile
// takes 67 thousand clocks, in which MMAs are issued throughout, where its 46 pairs
// need 47 thousand on the tensor core (64 % of its cycles active); its copies, 27
// slices of 8 KB a K step, come at 54 bytes a clock and SM beside them.  Four
// accumulators a group need 17, but nothing of a drain overlaps: a curl of 9 products
// 2048 x 256 x 256 took 314 us where this takes 287.
// The products of a field step at 2048 x 256 x 2 modes (33.4 GFLOP) took 31.5 ms on
// the FP64 pipe (its peak); with these 1.63, the slices 0.53 and the scales 0.13.
//   warps 0..15: the row threads (TMEM lane quarter w % 4, column quarter
//   w / 4), which drain the accumulators, combine and write;
//   warp 16 issues the MMAs, warp 17 the bulk copies, each as a whole warp
//   with one elected lane (as in umma_kernel, tc_umma.cu: a branch on a
//   thread's own index cost 134 clocks an MMA).  The two weights of a group
//   share one instruction of 256 columns: 27 a K step instead of 46, each reading
//   its slice of A once for both.
// Every mbarrier wait has an iteration limit (the pipeline's from the host, as
// umma_kernel's), after which the CTA records an error, writes NaN to its unfinished
// tiles, waits for its own copies and MMAs (again with a limit), frees its TMEM and
// returns.  A time-out changes no control flow of the MMA warp, which goes on and may
// overwrite sums that are still being drained: the row threads look at the failure
// flag, which is set before that, after they have read a tile's last sums as well.
#include <cuda_bf16.h>
#include <limits.h>

#include <type_traits>

#include "tc_gemm.cuh"
#include "tc_ozaki.cuh"
#include "tc_ptx.cuh"

using namespace chm;

namespace {

constexpr int ND = 9;             // digits
constexpr int NS = ND + 1;        // slices of a block: |x|, the digits
constexpr int kStageSlices = 9;   // slices of each operand in a stage
constexpr int TH = 128;           // rows per tile
constexpr int KB = 16;            // K step
constexpr int kChunk = 16;        // K steps per accumulation (256 K values)
constexpr int kRowWarps = 16;     // a TMEM lane quarter and a column quarter each
constexpr int kRowThreads = 32 * kRowWarps;
constexpr int kMmaWarp = kRowWarps, kLoadWarp = kRowWarps + 1;
constexpr int kThreads = kRowThreads + 128;  // five warpgroups
// registers: launched with 96 a thread (640 x 96 = 61440); the issuing
// warpgroup keeps 64 and the four of the row threads, which hold 32 outputs
// each, take 104 (128 x 64 + 512 x 104 = 61440; with 32 and 112 the issuing
// warps spilled)
constexpr int kIssueRegs = 64, kRowRegs = 104;
constexpr int kColGroups = kRowWarps / 4;
constexpr int kMaxStages = 6;
constexpr uint32_t kASlice = TH * KB * 2;  // bytes of one A slice block
constexpr uint32_t kSmemMax = 217 * 1024;
constexpr int kMaxK = 65536;         // scales in shared memory
// row / column exponents: holds Inf or NaN; all zero
constexpr int kNonFinite = 1 << 20, kZero = -kNonFinite;
constexpr float kGuard = 1.0f / 4096, kExact = 8388608.0f;
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

// biased exponent (at least 1) of a finite nonzero value, 0 of zero, kNonFinite
__device__ __forceinline__ int exponent_of(double a) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(a) << 1;
  const int e = (int)(b >> 53);
  return b == 0 ? 0 : e == 0x7ff ? kNonFinite : max(e, 1);
}

// S[k]: the largest exponent of the finite elements of row k of a B matrix (0: none)
__global__ void __launch_bounds__(512) oz_scale(const __grid_constant__ SplitSet B, int16_t *S, int N, int K) {
  __shared__ int part[16][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, k = blockIdx.x * 32 + lane;
  const double *b = B.X[blockIdx.y] + k;
  int e = 0;
  if (k < K) {
#pragma unroll 8
    for (int n = g; n < N; n += 16) {
      const int x = exponent_of(__ldg(b + (long long)n * K));
      if (x < kNonFinite) e = max(e, x);
    }
  }
  part[g][lane] = e;
  __syncthreads();
  if (g == 0 && k < K) {
    for (int q = 1; q < 16; ++q) e = max(e, part[q][lane]);
    S[(long long)blockIdx.y * K + k] = (int16_t)e;
  }
}

// The digits and sizes of 8 consecutive K values.  hi: digits 0 .. 7 + 128 (byte
// 7 - s is digit s); lo: digit 8 + 128, a byte each; g: |x| 2^-E in BF16 (rounded down).
struct Digits {
  unsigned long long hi[8];
  uint32_t lo[2], g[4];
};

// value i: a 2^(70 - E) rounded to an integer, |a| < 2^E; base less the exponent of a
// is the number of bits between them (nonnegative)
__device__ __forceinline__ void set_digits(Digits &D, int i, double a, int base, bool keep) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(a);
  const int e = (int)((b >> 52) & 0x7ff), d = base - max(e, 1);
  // the significand's upper bit at 2^63
  unsigned long long m = (b << 11) & 0x7ffffffffffff800ULL;
  if (e) m |= 1ULL << 63;
  if (!keep) m = 0;
  uint32_t g = (uint32_t)(126 - d) << 7 | ((uint32_t)(b >> 45) & 0x7f);
  if (m >> 63 == 0 || d >= 126) g = 0;
  // 8 bits below hi: the lowest bits of the significand below 2^11 are zero
  unsigned long long hi = m >> min(2 + d, 63);
  uint32_t lo = 0;
  if (d > 6) {
    const unsigned long long q = d < 71 ? ((m >> (d - 7)) + 1) >> 1 : 0ULL;
    hi = q >> 8;
    lo = (uint32_t)q & 255;
  }
  if (b >> 63) {
    hi = ~hi + (lo == 0);
    lo = (256 - lo) & 255;
  }
  lo += 128;
  D.hi[i] = hi + (lo >> 8) + 0x8080808080808080ULL;
  lo &= 255;
  if (i & 3) D.lo[i >> 2] |= lo << (8 * (i & 3));
  else D.lo[i >> 2] = lo;
  if (i & 1) D.g[i >> 1] |= g << 16;
  else D.g[i >> 1] = g;
}

// their slices, 16 bytes per slice at p + slice stride
__device__ __forceinline__ void store_slices(const Digits &D, uint8_t *p, uint32_t stride) {
  *reinterpret_cast<uint4 *>(p) = make_uint4(D.g[0], D.g[1], D.g[2], D.g[3]);
#pragma unroll
  for (int s = 0; s < ND; ++s) {
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float f[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = 2 * q + h;
        const uint32_t word = s < 4 ? (uint32_t)(D.hi[i] >> 32) : s < 8 ? (uint32_t)D.hi[i] : D.lo[i >> 2];
        // 2^23 + byte as a float, less 2^23 + 128: the digit
        f[h] = __uint_as_float(__byte_perm(word, 0x4B000000u, 0x7440u | (s < 8 ? 3 - (s & 3) : i & 3))) - 8388736.0f;
      }
      w[q] = __byte_perm(__float_as_uint(f[0]), __float_as_uint(f[1]), 0x7632);  // BF16 pair
    }
    *reinterpret_cast<uint4 *>(p + (s + 1) * stride) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// 32 rows (block bx) of one A plane, all K: the rows' largest exponents, then
// the slices (the second read comes from L1 / L2).  HBM bound: 8 B read and
// 20 B written per element.  sk: the K values' exponents
__device__ __forceinline__ void split_rows(const SplitSet &J, const int16_t *sk, int job, int bx, int M, int K,
                                           int nkb) {
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
  int e = 0;  // the scaled elements' largest exponent (0: all zero, or times zero)
  if (ok)
    for (int k = g; k < K; k += 8) {
      const int x = exponent_of(__ldg(a + (long long)k * M)), s = sk[k];
      e = max(e, x == kNonFinite ? x : x && s ? x + s : 0);
    }
  emax[g][r] = e;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 8; ++q) e = max(e, emax[q][r]);
  const bool has = e > 0 && e < kNonFinite;
  if (g == 0) J.E[job][gm] = e == 0 ? kZero : e;
  const int mt = gm / TH, rt = gm % TH;
  uint8_t *T = J.T[job] + (long long)mt * nkb * NS * kASlice + (rt >> 3) * 256 + (rt & 7) * 16;
  for (int kg = g; kg < 2 * nkb; kg += 8) {
    Digits u;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int k = kg * 8 + q;
      const bool in = has && k < K;
      const int s = in ? sk[k] : 0;
      const double v = in ? __ldg(a + (long long)k * M) : 0.0;
      set_digits(u, q, neg ? -v : v, e - s, s != 0);
    }
    store_slices(u, T + (long long)(kg >> 1) * NS * kASlice + (kg & 1) * 128, kASlice);
  }
}

// 8 columns (block bx) of one B matrix, a warp per column
__device__ __forceinline__ void split_cols(const SplitSet &J, const int16_t *sk, int job, int bx, int N, int K,
                                           int nkb, int tnc) {
  constexpr int kUp = 4096;  // (keeps the scaled exponents positive)
  const int lane = threadIdx.x & 31;
  const int n = bx * 8 + (threadIdx.x >> 5);
  const bool ok = n < N;
  const double *b = J.X[job] + (long long)n * K;
  int e = 0;
  if (ok)
    for (int k = lane; k < K; k += 32) {
      const int x = exponent_of(__ldg(b + k));
      e = max(e, x == kNonFinite ? x : x ? x - sk[k] + kUp : 0);
    }
  e = __reduce_max_sync(0xffffffffu, e);
  const bool has = e > 0 && e < kNonFinite;
  if (lane == 0) J.E[job][n] = e == 0 ? kZero : e < kNonFinite ? e - kUp : e;
  const uint32_t slice = (uint32_t)tnc * KB * 2;
  const int nt = n / tnc, nn = n % tnc;
  uint8_t *T = J.T[job] + (long long)nt * nkb * NS * slice + (nn >> 3) * 256 + (nn & 7) * 16;
  for (int kg = lane; kg < 2 * nkb; kg += 32) {
    Digits u;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int k = kg * 8 + q;
      const bool in = has && k < K;
      set_digits(u, q, in ? __ldg(b + k) : 0.0, e - kUp + (in ? sk[k] : 0), in);
    }
    store_slices(u, T + (long long)(kg >> 1) * NS * slice + (kg & 1) * 128, slice);
  }
}

// one launch for the batch's operands: na blocks for the A planes (ax per
// plane), then the B matrices' (bx each).  A K value's scale is the largest of the
// nb matrices' (they share the slices of A).
__global__ void __launch_bounds__(256) oz_split(const __grid_constant__ SplitSet A, const __grid_constant__ SplitSet B,
                                                const int16_t *__restrict__ S, int nb, int na, int ax, int bx, int M,
                                                int N, int K, int nkb, int tnc) {
  extern __shared__ int16_t sk[];  // [K]
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    int s = 0;
    for (int q = 0; q < nb; ++q) s = max(s, (int)S[(long long)q * K + k]);
    sk[k] = (int16_t)s;
  }
  __syncthreads();
  const int b = (int)blockIdx.x;
  if (b < na) split_rows(A, sk, b / ax, b % ax, M, K, nkb);
  else split_cols(B, sk, (b - na) / bx, (b - na) % bx, N, K, nkb, tnc);
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
  const double2 *shift;
  long long spin;  // iteration limit of the pipeline waits
};

// 4 consecutive accumulator columns of this warp's 32 TMEM lanes
__device__ __forceinline__ void tmem_ld4(uint32_t (&v)[4], uint32_t taddr) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(taddr));
}

// h 2^46 + t rounded to FP64, |h| < 2^30, |t| < 2^62: both parts as the low bits of
// doubles with fixed exponents, less these (exact), and one rounded sum.  Two FP64
// operations; normalising in integers took 40 dependent instructions.
__device__ __forceinline__ double round_sum(int h, long long t) {
  const int hh = h + (int)(t >> 46);
  const double low = __hiloint2double((int)(t >> 32 & 0x3fff) | 0x43300000, (int)t);  // 2^52 + (t mod 2^46)
  const double top = __hiloint2double(0x43300000 + (46 << 20), hh ^ INT_MIN);  // 2^98 + (hh + 2^31) 2^46
  return (top - (0x1p98 + 0x1p77 + 0x1p52)) + low;
}

// (a denormal result or an overflow)
__device__ __noinline__ double scaled_rare(double v, int ex) { return scalbn(v, ex); }

// K steps of a stage, slices of a K step and the first of them, of each group
__device__ __forceinline__ int group_ksteps(int g) { return g < 3 ? 1 : 2 * (g - 2); }
__device__ __forceinline__ uint32_t group_slices(int g) { return g < 3 ? 9 - 2 * g : g == 3 ? 4 : 2; }
__device__ __forceinline__ uint32_t group_first(int g) { return g == 3 ? 0 : 1; }

// Row gm of a problem's A: its first element; sg: its sign (reflected planes).
__device__ __forceinline__ const double *row_of(const OzProb *Q, int M, int gm, double &sg) {
  sg = 1.0;
  if (!Q->reflect) return Q->A + gm;
  const int x = gm >> 1;
  if ((gm & 1) == 0) sg = -1.0;
  return Q->A + 2 * (long long)(x == 0 ? 0 : (M >> 1) - x) + (gm & 1);
}

// The sums in FP64 of column n for the rows gm of the lanes in `want` (the whole
// warp calls).  The lanes are shared out evenly, a power of two to a row, each of
// which takes every so many terms: one to eight rows take some 1 to 2.5 thousand
// clocks at K = 256, one row to a lane 17.  (Above 16 rows: a lane to a row, in
// the order and with the result of the FP64 pipe's kernel.)
__device__ __noinline__ double fp64_sums(const OzProb *Q, const OzArgs *A, int gm, int n, uint32_t want) {
  const int M = A->M, K = A->K, lane = threadIdx.x & 31, rows = __popc(want);
  const int each = rows == 1 ? 32 : 1 << (__clz(rows - 1) - 27);  // lanes to a row
  const int r = lane / each;
  const int from = __shfl_sync(0xffffffffu, gm, r < rows ? (int)__fns(want, 0, r + 1) : lane);
  double s = 0.0, sg;
  if (r < rows) {
    const double *a = row_of(Q, M, from, sg), *b = Q->B + (long long)n * K;
#pragma unroll 8
    for (int k = lane & (each - 1); k < K; k += each)
      s = fma(sg * __ldg(a + (long long)k * M), __ldg(b + k), s);
  }
  for (int o = each >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return __shfl_sync(0xffffffffu, s, __popc(want & ((1u << lane) - 1)) * each & 31);
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
  const uint32_t stage_bytes = kStageSlices * (kASlice + b_slice);
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
        for (int cg = 0; cg < 5 * nchunk && ok; ++cg) {
          const int grp = cg % 5, kb0 = cg / 5 * kChunk, kb1 = min(nkb, kb0 + kChunk);
          const int ks = group_ksteps(grp);
          const uint32_t ns = group_slices(grp), s0 = group_first(grp);
          for (int kb = kb0; kb < kb1; kb += ks) {
            const bool go = !*vfail && (round == 0 || mbar_wait(&empty[s], (uint32_t)(round - 1) & 1u, A.spin));
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
                bulk_g2s(st + (uint32_t)q * ns * kASlice, TA + ((long long)(kb + q) * NS + s0) * kASlice,
                         ns * kASlice, bar);
                bulk_g2s(st + kStageSlices * kASlice + (uint32_t)q * ns * b_slice,
                         TB + ((long long)(kb + q) * NS + s0) * b_slice, ns * b_slice, bar);
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
      long long lim = A.spin;
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
        for (int cg = 0; cg < 5 * nchunk; ++cg, ++u) {
          const int grp = cg % 5, kb0 = cg / 5 * kChunk, kb1 = min(nkb, kb0 + kChunk);
          const int ks = group_ksteps(grp), b = u & 1, use = u >> 1;
          if (use > 0) wait(&dempty[b], use - 1);
          const uint32_t d0 = tmem + (uint32_t)(2 * b * tnc), d1 = d0 + (uint32_t)tnc;
          for (int kb = kb0; kb < kb1; kb += ks) {
            if (!ready) wait(&full[s], round);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t st = smem0 + (uint32_t)s * stage_bytes;
            const uint32_t alo = (uint32_t)smem_desc<KB>(st), blo = (uint32_t)smem_desc<KB>(st + kStageSlices * kASlice);
            uint64_t *const freed = &empty[s];
            if (++s == stages) s = 0, ++round;
            ready = mbar_test(&full[s], (uint32_t)round & 1u);
            // (the first K step overwrites the accumulators)
            const uint32_t more = kb != kb0;
            // the pairs (i, W - i) and (i, W + 1 - i) of the group's two weights
            // W (into d0) and W + 1 (into d1) of one K step: one
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
              if (grp == 0) step(std::integral_constant<int, 7>{}, 0, more);
              else if (grp == 1) step(std::integral_constant<int, 5>{}, 0, more);
              else if (grp == 2) step(std::integral_constant<int, 3>{}, 0, more);
              else if (grp == 3)
                for (int q = 0; q < n; ++q) {  // |a| |b| into d1, the pairs of weight 2 into d0
                  const uint32_t a = alo + (uint32_t)q * 4 * (kASlice >> 4), bb = blo + (uint32_t)q * 4 * bs;
                  umma_bf16<kDiscard>(d1, a, bb, dhi, idesc, more | (q > 0));
#pragma unroll
                  for (int i = 1; i <= 3; ++i)
                    umma_bf16<kDiscard>(d0, a + i * (kASlice >> 4), bb + (4 - i) * bs, dhi, idesc,
                                        i == 1 ? more | (q > 0) : 1u);
                }
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
    long long t64[CH];  // the integer sums, then their FP64 bits
    int u = 0;
    bool ok = true;
    // waits for the next group; its first accumulator's address, 0 on a time-out
    auto ready = [&]() -> uint32_t {
      const int b = u & 1;
      const bool got = !*vfail && mbar_wait(&dfull[b], (uint32_t)(u >> 1) & 1u, A.spin) && !*vfail;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      ok = __all_sync(0xffffffffu, got) != 0;
      return lane_base + (uint32_t)(2 * b * tnc);
    };
    auto release = [&]() {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive(&dempty[u & 1]);
      ++u;
    };
    // f(column, d0, d1) over this thread's columns of the group (FP32 bits)
    auto drain = [&](uint32_t ta, auto f) {
#pragma unroll
      for (int g = 0; g < CH / 4; ++g)
        if (g * 4 < ncol) {
          uint32_t v0[4], v1[4];
          tmem_ld4(v0, ta + (uint32_t)(g * 4));
          tmem_ld4(v1, ta + (uint32_t)(tnc + g * 4));
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 4; ++j) f(g * 4 + j, __uint_as_float(v0[j]), __uint_as_float(v1[j]));
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
      // columns whose sum |a b| is not known to be above kGuard; whose S_5 or S_6 may be inexact
      uint32_t low = 0xffffffffu, over = 0;
      for (int c = 0; c < nchunk; ++c) {
        uint32_t ta = ready();
        if (!ok) break;
        drain(ta, [&](int j, float s7, float s8) {
          t64[j] = (__float2int_rn(s7) + ((__float2int_rn(s8) + 128) >> 8) + 2) >> 2;
        });
        release();
        ta = ready();
        if (!ok) break;
        drain(ta, [&](int j, float s5, float s6) {
          t64[j] += (long long)__float2int_rn(s5) * (1 << 14) + (long long)__float2int_rn(s6) * (1 << 6);
          if (fmaxf(fabsf(s5), fabsf(s6)) >= kExact) over |= 1u << j;
        });
        release();
        ta = ready();
        if (!ok) break;
        drain(ta, [&](int j, float s3, float s4) {
          t64[j] += (long long)__float2int_rn(s3) * (1 << 30) + (long long)__float2int_rn(s4) * (1 << 22);
        });
        release();
        ta = ready();
        if (!ok) break;
        drain(ta, [&](int j, float s2, float sum) {
          t64[j] += (long long)((unsigned long long)(long long)__float2int_rn(s2) << 38);
          if (sum >= kGuard) low &= ~(1u << j);
        });
        release();
        ta = ready();
        if (!ok) break;
        // The last sums and the tile's values, four columns at a time: their chains of
        // dependent instructions side by side, and what is rare behind one vote for
        // them (one column after the other, normalised in integers: 55 of a tile's 95
        // thousand clocks; now 23, next to the MMAs of the next tile).  A loop that
        // moves the array along: unrolled, its code takes twice as long the first time.
#pragma unroll 1
        for (int j0 = 0; j0 < ncol; j0 += 4) {
          uint32_t v0[4], v1[4];
          tmem_ld4(v0, ta + (uint32_t)j0);
          tmem_ld4(v1, ta + (uint32_t)(tnc + j0));
          tmem_wait_ld();
          double x[4];
          uint32_t odd = 0, want = 0;
          const bool final = c == nchunk - 1;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            // |S_0| <= 2^20, |S_1| <= 2^22: 256 S_0 + S_1 fits 32 bits
            const int h = __float2int_rn(__uint_as_float(v0[j])) * 256 + __float2int_rn(__uint_as_float(v1[j]));
            const int eb = __shfl_sync(0xffffffffu, ebl, j0 + j), ex = ea + eb - 2110;
            x[j] = round_sum(h, t64[j]);
            const int hi = __double2hiint(x[j]), e = ((hi >> 20) & 0x7ff) + ex;
            if (hi != 0 && (e < 1 || e > 2046)) odd |= 1u << j;
            else if (hi != 0) x[j] = __hiloint2double(hi + (int)((uint32_t)ex << 20), __double2loint(x[j]));
            if (max(ea, eb) >= kNonFinite || ((((low | over) >> (j0 + j)) & 1) && min(ea, eb) > kZero))
              want |= 1u << j;
          }
          const int n = n0 + j0;
          double *pc = Q.C + gm + (long long)n * A.M;
          if (!rok || !final) want = 0;
          if (__any_sync(0xffffffffu, (odd | want) != 0)) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int eb = __shfl_sync(0xffffffffu, ebl, j0 + j);
              if ((odd >> j) & 1) x[j] = scaled_rare(x[j], ea + eb - 2110);
            }
          }
          if (c > 0 && rok) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (n + j < A.N) x[j] += pc[(long long)j * A.M];
          }
          if (__any_sync(0xffffffffu, want != 0)) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const bool one = ((want >> j) & 1) && n + j < A.N;
              const uint32_t lanes = __ballot_sync(0xffffffffu, one);
              if (lanes) {
                const double s = fp64_sums(&Q, &A, gm, n + j, lanes);
                if (one) x[j] = s;
              }
            }
          }
          if (SHIFT && final) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              // rows 2x (re) and 2x + 1 (im) sit in adjacent lanes
              const double other = __shfl_xor_sync(0xffffffffu, x[j], 1);
              x[j] = (row & 1) ? other * sh.y + x[j] * sh.x : x[j] * sh.x - other * sh.y;
              if (Q.fac && rok && n + j < A.N) x[j] *= Q.fac[(gm >> 1) + (long long)(A.M >> 1) * (n + j)];
            }
          }
          if (rok) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (n + j < A.N) pc[(long long)j * A.M] = x[j];
          }
#pragma unroll
          for (int j = 0; j + 4 < CH; ++j) t64[j] = t64[j + 4];
        }
        release();
        // (what was read of an accumulator that a late MMA had overwritten is not a value)
        ok = __all_sync(0xffffffffu, !*vfail) != 0;
        if (!ok) break;
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
inline i64 scale_bytes(i64 K, i64 nB) { return rup(2 * K * nB, 256); }

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
  return nA * plane_bytes(rup(M, TH), K) + nB * plane_bytes(tc_np((int)N), K) + scale_bytes(K, nB) + 256;
}

// (every size the index arithmetic holds; from 16 x 4 to 4096 x 100 grids a curl of
// 2 modes with this product was never slower than on the FP64 pipe: 14.0 against
// 20.1 us at 16 x 4, 16.2 against 21.2 at 512 x 4, 26.6 against 77 at 512 x 64)
bool oz_takes(i64 M, i64 N, i64 K, int count) {
  return M % 2 == 0 && M < (1 << 30) && N <= 65536 && K <= kMaxK && count > 0;
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
  A.shift = shift;
  // (a tile whose outputs are all summed in FP64 keeps its accumulators for 8192 K
  // clocks, the FP64 pipe's time; a poll takes at least some 40)
  A.spin = tc_spin_limit() * (1 + K / 1024);
  const uint32_t stage = kStageSlices * (kASlice + (uint32_t)A.tnc * KB * 2);
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
  int16_t *S = reinterpret_cast<int16_t *>(c);
  for (int i = 0; i < count; ++i)
    ob.p[i] = OzProb{JA.T[ia[i]], JB.T[ib[i]], JA.E[ia[i]], JB.E[ib[i]], p[i].A, p[i].B, p[i].C, p[i].fac,
                     p[i].reflect};
  const int ax = nmt * TH / 32, bx = Np / 8;
  oz_scale<<<dim3((unsigned)((K + 31) / 32), (unsigned)nB), 512, 0, st>>>(JB, S, N, K);
  count_launch();
  if (2 * K > 32 * 1024) cudaFuncSetAttribute(oz_split, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * kMaxK);
  oz_split<<<(unsigned)(nA * ax + nB * bx), 256, 2 * K, st>>>(JA, JB, S, nB, nA * ax, ax, bx, M, N, K, nkb, A.tnc);
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
