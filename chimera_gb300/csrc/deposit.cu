// Deterministic charge / current deposition (grid_deps*.f90), FP64.
//
// Each particle's 2x2-node x (modes) x (components) complex contribution is
// converted to 64-bit fixed point and summed with integer atomics.  Integer
// addition is associative, so the accumulated grid is bitwise identical
// whatever order the particles are processed in: no float atomics reach
// memory and two runs give the same bits.
//
// The fixed-point scale is a power of two chosen from a deterministic bound
// B >= sum_p |w_p| (|w_p|^2 for the envelope density, which applies the
// weight twice): scale = 2^(61 - ceil(log2 B)), so no partial sum can
// overflow and the quantum is B * 2^-61 (~1e-18 relative to B).
//
// Work is privatised per thread block: each block takes a contiguous range
// of particles, and when the cells they touch fit a shared-memory box the
// block accumulates there and flushes the box once with global integer
// atomics; otherwise it adds straight to the global accumulator.  Particles
// kept in cell order (genparts order or after a sort) almost always fit.
//
// What bounds it: GB300's FP64 pipe, 2 operations a clock and SM.  So a
// particle's geometry is computed once (shared memory keeps it between the two
// passes), roots and divisions share one rsqrt, and a value is turned into a
// 63-bit integer mantissa once and multiplied by the four nodes' weights, 62-bit
// fixed point, in integer instructions (55 FP64 operations a particle where the
// products, scalings and conversions in FP64 took 268, for a current of 2 modes).
// The product keeps 62 bits and is rounded once to the quantum.  The box's 64-bit
// sums are two native 32-bit atomics with a carry (a 64-bit one on shared memory
// is a compare-and-swap loop), and a thread takes four neighbours in the
// particle order, so that a warp's lanes hit other cells and not all the same.
// 2.1 million particles, 2 modes: current 1345 -> 308 us, density 621 -> 188 us
// (the FP64 pipe 62 and 73 % busy; waits for the atomics' old values next); 1
// million unordered ones, 3 envelope modes, no box: current 446 -> 249 us.
#include <math.h>

#include "common.cuh"

using namespace chm;

namespace {

constexpr int kDepThreads = 256;
constexpr int kPartPerBlock = 1024;  // particles per block
constexpr int kPerThread = kPartPerBlock / kDepThreads;
constexpr int kGeoBytes = 32 * kPartPerBlock;  // the particles' geometry
// shared accumulator budget (two blocks to an SM); larger boxes go to global sums (2.1
// million particles: a current of 2 modes over 76 KB 426 us, 84 KB 500, of 3 modes 71 KB
// 536, 81 KB 728; with 96 KB and FP64 weights these took 1282, 1287, 1645 and 1647)
constexpr int kBoxBytes = 78 * 1024;
constexpr int kRedBlocks = 1024;

enum Kind { CURR = 0, DENS = 1, CURR_ENV = 2, DENS_ENV = 3 };

__host__ __device__ constexpr int ncomp_of(int kind) { return (kind == CURR || kind == CURR_ENV) ? 3 : 1; }

// Deterministic partial sums of |w| (or w^2), fixed tree order.
__global__ void wsum_partial_kernel(const double *__restrict__ w, i64 w_ps, i64 np, int squared,
                                    double *__restrict__ partial) {
  __shared__ double sh[kDepThreads];
  i64 per = (np + gridDim.x - 1) / gridDim.x;
  i64 b0 = blockIdx.x * per, b1 = min(np, b0 + per);
  double s = 0.0;
  // (eight loads in flight: one at a time, 2 thousand weights a block took 20.5 us, now 16)
  constexpr int kAhead = 8;
  for (i64 i = b0 + threadIdx.x; i < b1; i += kAhead * (i64)blockDim.x) {
    double v[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const i64 ik = i + k * (i64)blockDim.x;
      v[k] = ik < b1 ? fabs(w[ik * w_ps]) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k) s += squared ? v[k] * v[k] : v[k];
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int st = blockDim.x / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

__global__ void wsum_final_kernel(const double *__restrict__ partial, int n, double *scale_out) {
  __shared__ double sh[kRedBlocks];
  for (int i = threadIdx.x; i < kRedBlocks; i += blockDim.x) sh[i] = i < n ? partial[i] : 0.0;
  __syncthreads();
  for (int st = kRedBlocks / 2; st > 0; st >>= 1) {
    for (int i = threadIdx.x; i < st; i += blockDim.x) sh[i] += sh[i + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    double B = sh[0];
    if (!(B > 0.0) || !isfinite(B)) B = 1.0;
    int e;
    frexp(B, &e);  // B < 2^e
    scale_out[0] = ldexp(1.0, 61 - e);
  }
}

__global__ void set_one_kernel(double *p) { p[0] = 1.0; }

struct DepArgs {
  const double *x;
  i64 x_cs, x_ps;
  const double *p;
  i64 p_cs, p_ps;
  const double *w;
  i64 w_ps;
  double leftX, dx_inv, dr_inv, kx0;
  const double *rgrid;
  i64 np, nx, nr;
  int nm;
  const int32_t *ind;  // chunk offsets or null
  int nchnk;
  i64 cs, guards;
  unsigned long long *acc;  // (nx, nr, nm, ncomp) x {re, im} int64
  const double *scale;
};

// A value in quanta as m 2^(n + 2 - 64), |m| in [2^62, 2^63); n < 0: outside the
// range of this form (2^61 quanta or more, infinite, NaN)
struct Fixed {
  long long m;
  int n;
};

__device__ __forceinline__ Fixed to_fixed(double v) {
  const long long b = __double_as_longlong(v);
  const int e = (int)((unsigned long long)b >> 52) & 0x7ff;
  const long long m = ((b & 0xfffffffffffffLL) | 0x10000000000000LL) << 10;
  Fixed f{b < 0 ? -m : m, 60 - (e - 1023)};
  if (f.n > 62) f = {0, 62};  // below a quarter of a quantum: 0 with any weight below 2
  return f;
}

// Tests and conversions by integer instructions: on the FP64 pipe each costs as
// much as a product.
__device__ __forceinline__ bool is_zero(double v) { return ((unsigned long long)__double_as_longlong(v) << 1) == 0; }
// |v| below a power of two, given by the upper word of its bits
__device__ __forceinline__ bool below(double v, unsigned hi) { return ((unsigned)__double2hiint(v) & 0x7fffffffu) < hi; }

// v 2^62 rounded, |v| < 2
__device__ __forceinline__ long long weight_fixed(double v) {
  const long long b = __double_as_longlong(v);
  const int e = (int)((unsigned long long)b >> 52) & 0x7ff, n = (1023 - e) & 63;
  if (e < 1023 - 63) return 0;  // below 2^-63
  const unsigned long long m = ((unsigned long long)(b & 0xfffffffffffffLL) | 0x10000000000000ULL) << 10;
  const long long q = (long long)((m + ((1ULL << n) >> 1)) >> n);
  return b < 0 ? -q : q;
}

// value x weight, w = weight 2^62, rounded to quanta
__device__ __forceinline__ long long weighted(Fixed f, long long w) {
  const int n = f.n & 63;  // (n < 0: the caller does not use the value)
  return (__mul64hi(f.m, w) + ((1LL << n) >> 1)) >> n;
}

// the same in FP64, for what the integer form does not take
__device__ __noinline__ long long weighted_any(double v, double w) { return __double2ll_rn(v * w); }

// Where contributions go: the block's box in shared memory or the global sums.
// Offsets count 64-bit words; a node's real and imaginary sums are neighbours.
struct BoxSink {
  unsigned long long *sum;
  int ml, row;  // words between (mode, component) planes and between rows
  // q[j][k] to row j, node k of the stencil, k with ok[k]; the four low words
  // first, so that their atomics are in flight together
  __device__ __forceinline__ void add(int at, const long long (&q)[2][2], const bool (&ok)[2]) const {
    uint32_t *w = reinterpret_cast<uint32_t *>(sum + at), old[2][2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (ok[k]) old[j][k] = atomicAdd(w + 2 * j * row + 4 * k, (uint32_t)q[j][k]);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (ok[k])
          atomicAdd(w + 2 * j * row + 4 * k + 1,
                    (uint32_t)((unsigned long long)q[j][k] >> 32) +
                        (old[j][k] + (uint32_t)q[j][k] < old[j][k] ? 1u : 0u));
  }
  using Off = int;
};
struct GridSink {
  unsigned long long *sum;
  i64 ml, row;
  __device__ __forceinline__ void add(i64 at, const long long (&q)[2][2], const bool (&ok)[2]) const {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (ok[k] && q[j][k]) atomicAdd(sum + at + j * row + 2 * k, (unsigned long long)q[j][k]);
  }
  using Off = i64;
};

// A particle's geometry, from the first pass to the second
struct Geo {
  double sx1, sr1, rinv;
  unsigned ix1, ir;  // x cell + 1 (0: the cell left of the grid), r cell
};
constexpr unsigned kNoCell = 0xffffffffu;

__device__ __forceinline__ Geo geometry(const DepArgs &A, i64 i) {
  Geo g{};
  g.ir = kNoCell;
  const double xp = A.x[i * A.x_ps], yp = A.x[A.x_cs + i * A.x_ps], zp = A.x[2 * A.x_cs + i * A.x_ps];
  double rp;
  root_and_inverse(yp * yp + zp * zp, rp, g.rinv);
  const double fx = (xp - A.leftX) * A.dx_inv;
  if (!(rp < A.rgrid[A.nr - 1]) || !below(fx, 0x43100000u)) return g;  // (2^50)
  const double fl = floor(fx);
  const i64 ix = (i64)fl, ir = (i64)floor((rp - A.rgrid[0]) * A.dr_inv);
  if (ir < 0 || ir > A.nr - 2 || ix < -1 || ix >= A.nx) return g;
  g.sx1 = fx - fl;
  g.sr1 = (rp - A.rgrid[ir]) * A.dr_inv;
  g.ix1 = (unsigned)(ix + 1);
  g.ir = (unsigned)ir;
  return g;
}

// Adds one particle's values; at: the sink's offset of its lower left node,
// mode 0, component 0.
template <int KIND, typename Sink>
__device__ __forceinline__ void particle_contrib(const DepArgs &A, i64 i, int chunk, const Geo &g, double scale,
                                                 const Sink &S, typename Sink::Off at) {
  using Off = typename Sink::Off;
  const double wp = A.w[i * A.w_ps];
  if (is_zero(wp)) return;
  constexpr bool env = KIND == CURR_ENV || KIND == DENS_ENV;
  double v[3] = {0.0, 0.0, 0.0};
  if (KIND == CURR || KIND == CURR_ENV) {
    v[0] = A.p[i * A.p_ps];
    v[1] = A.p[A.p_cs + i * A.p_ps];
    v[2] = A.p[2 * A.p_cs + i * A.p_ps];
    const unsigned long long any = (unsigned long long)(__double_as_longlong(v[0]) | __double_as_longlong(v[1]) |
                                                        __double_as_longlong(v[2]));
    if ((any << 1) == 0) return;  // all three zero
    const double ginv = rsqrt(1.0 + v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    const double f = KIND == CURR ? ginv * (wp * scale) : ginv;
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] *= f;
  }
  // the value of mode 0 for the kinds of one component (in quanta)
  double2 one = make_double2(wp * scale, 0.0);
  if (env) {
    double s, c;
    sincos(A.x[i * A.x_ps] * A.kx0, &s, &c);
    const double2 wc = make_double2(wp * c, -wp * s);
    const double f = KIND == CURR_ENV ? v[2] * scale : scale;
    one = KIND == CURR_ENV ? wc : cmul(wc, wc);
    one = cscale(one, f);
  }

  // x-node acceptance (grid bounds + chunk guard semantics)
  bool okx[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const i64 gx = (i64)g.ix1 - 1 + k;
    bool ok = (gx >= 0 && gx < A.nx);
    if (ok && A.ind) {
      i64 nxleft = (i64)chunk * A.cs;
      i64 lx = gx - nxleft;
      if (lx <= 0) ok = (nxleft - A.guards >= 0) && (lx >= -A.guards);
      else if (lx >= A.cs) ok = (nxleft + A.cs + A.guards <= A.nx - 1) && (lx <= A.cs + A.guards);
    }
    okx[k] = ok;
  }
  const double sx[2] = {1.0 - g.sx1, g.sx1}, sr[2] = {1.0 - g.sr1, g.sr1};
  // (the r weights are within [0, 1] on a uniform r grid, to rounding)
  const bool exact = below(sr[0], 0x40000000u) && below(sr[1], 0x40000000u);
  long long w[2][2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
#pragma unroll
    for (int j = 0; j < 2; ++j) w[j][k] = weight_fixed(sx[k] * sr[j]);
  }
  auto emit = [&](Off o, double val) {
    const Fixed f = to_fixed(val);
    if (f.m == 0) return;
    long long q[2][2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < 2; ++k) q[j][k] = weighted(f, w[j][k]);
    if (!exact || f.n < 0) {
      for (int j = 0; j < 2; ++j)
        for (int k = 0; k < 2; ++k) q[j][k] = weighted_any(val, sx[k] * sr[j]);
    }
    S.add(o, q, okx);
  };
  auto emit2 = [&](Off o, double2 val) {
    emit(o, val.x);
    emit(o + 1, val.y);
  };
  const int K = env ? (A.nm - 1) / 2 : 0;
  const int nph = env ? K + 1 : A.nm;
  // mode 0 has phase 1
  if (KIND == CURR) {
#pragma unroll
    for (int l = 0; l < 3; ++l) emit(at + (Off)A.nm * l * S.ml, v[l]);
  } else {
    emit2(at + (Off)(K + (KIND == CURR_ENV ? 2 * A.nm : 0)) * S.ml, one);  // z alone: grid_deps_env.f90:76
  }
  if (nph == 1) return;
  const double yp = A.x[A.x_cs + i * A.x_ps], zp = A.x[2 * A.x_cs + i * A.x_ps];
  const double2 ph = make_double2(yp * g.rinv, -zp * g.rinv);  // 0 on the axis
  double2 phm = ph;
  for (int mi = 1; mi < nph; ++mi) {
    if (mi > 1) phm = cmul(phm, ph);
    if (KIND == CURR) {
#pragma unroll
      for (int l = 0; l < 3; ++l) emit2(at + (Off)(mi + A.nm * l) * S.ml, cscale(phm, v[l]));
    } else if (KIND == DENS) {
      emit2(at + (Off)mi * S.ml, cscale(phm, one.x));
    } else {
      const Off o = at + (KIND == CURR_ENV ? (Off)(2 * A.nm) * S.ml : (Off)0);
      emit2(o + (Off)(K + mi) * S.ml, cmul(phm, one));
      emit2(o + (Off)(K - mi) * S.ml, cmul(cconj(phm), one));
    }
  }
}

__device__ __forceinline__ int chunk_of(const int32_t *ind_sh, int nchnk, i64 i) {
  // ind_sh sorted; returns c with ind[c] <= i < ind[c+1], or -1
  if (i < ind_sh[0] || i >= ind_sh[nchnk]) return -1;
  int lo = 0, hi = nchnk;  // invariant ind[lo] <= i < ind[hi]
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (ind_sh[mid] <= i) lo = mid;
    else hi = mid;
  }
  return lo;
}

template <int KIND>
__global__ void __launch_bounds__(kDepThreads, 2) deposit_kernel(DepArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int32_t ind_sh[257];
  __shared__ unsigned box_sh[4];  // least and largest x cell + 1 and r cell
  double *geo = reinterpret_cast<double *>(smem_raw);  // [4][kPartPerBlock]
  unsigned long long *box = reinterpret_cast<unsigned long long *>(smem_raw + kGeoBytes);
  const double scale = A.scale[0];
  const i64 p0 = (i64)blockIdx.x * kPartPerBlock;
  const int np = (int)min((i64)kPartPerBlock, A.np - p0);
  if (A.ind) {
    for (int t = threadIdx.x; t <= A.nchnk; t += blockDim.x) ind_sh[t] = A.ind[t];
  }
  if (threadIdx.x == 0) {
    box_sh[0] = box_sh[2] = kNoCell;
    box_sh[1] = box_sh[3] = 0;
  }
  __syncthreads();
  // 1) the particles' geometry and the box of the cells they touch
  {
    unsigned x0 = kNoCell, x1 = 0, r0 = kNoCell, r1 = 0;
#pragma unroll
    for (int s = 0; s < kPerThread; ++s) {
      const int t = kPerThread * threadIdx.x + s;
      if (t >= np) break;
      const Geo g = geometry(A, p0 + t);
      const int slot = s * kDepThreads + threadIdx.x;
      geo[slot] = g.sx1;
      geo[kPartPerBlock + slot] = g.sr1;
      geo[2 * kPartPerBlock + slot] = g.rinv;
      reinterpret_cast<uint2 *>(geo)[3 * kPartPerBlock + slot] = make_uint2(g.ix1, g.ir);
      if (g.ir == kNoCell) continue;
      x0 = min(x0, g.ix1);
      x1 = max(x1, g.ix1);
      r0 = min(r0, g.ir);
      r1 = max(r1, g.ir);
    }
    // a warp's bounds, then one atomic per warp (integer min/max: order-free)
    x0 = __reduce_min_sync(0xffffffffu, x0);
    x1 = __reduce_max_sync(0xffffffffu, x1);
    r0 = __reduce_min_sync(0xffffffffu, r0);
    r1 = __reduce_max_sync(0xffffffffu, r1);
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&box_sh[0], x0);
      atomicMax(&box_sh[1], x1);
      atomicMin(&box_sh[2], r0);
      atomicMax(&box_sh[3], r1);
    }
  }
  __syncthreads();
  if (box_sh[0] == kNoCell) return;  // no particle of the block reaches the grid
  // nodes: x from bx0 (cells start one left of the grid) to the last cell + 1
  const i64 bx0 = (i64)box_sh[0] - 1, br0 = box_sh[2];
  const i64 bnx = (i64)box_sh[1] - bx0 + 1, bnr = (i64)box_sh[3] - br0 + 2;
  const i64 most = kBoxBytes / 8, planes = (i64)A.nm * ncomp_of(KIND) * 2;
  const bool use_box = bnx <= most && bnr <= most && planes <= most && bnx * bnr <= most / planes;
  const int nvals = use_box ? (int)(bnx * bnr * planes) : 0;
  for (int t = threadIdx.x; t < nvals; t += blockDim.x) box[t] = 0ull;
  __syncthreads();
  const BoxSink bs{box, use_box ? (int)(bnx * bnr) * 2 : 0, use_box ? (int)bnx * 2 : 0};
  const GridSink gs{A.acc, 2 * A.nx * A.nr, 2 * A.nx};
#pragma unroll 1
  for (int s = 0; s < kPerThread; ++s) {
    const int t = kPerThread * threadIdx.x + s;
    if (t >= np) break;
    const int slot = s * kDepThreads + threadIdx.x;
    const uint2 cell = reinterpret_cast<const uint2 *>(geo)[3 * kPartPerBlock + slot];
    if (cell.y == kNoCell) continue;
    const Geo g{geo[slot], geo[kPartPerBlock + slot], geo[2 * kPartPerBlock + slot], cell.x, cell.y};
    const i64 i = p0 + t;
    int chunk = 0;
    if (A.ind) {
      chunk = chunk_of(ind_sh, A.nchnk, i);
      if (chunk < 0) continue;
    }
    const i64 ix = (i64)cell.x - 1;
    if (use_box)
      particle_contrib<KIND>(A, i, chunk, g, scale, bs, (int)(((i64)cell.y - br0) * bnx + (ix - bx0)) * 2);
    else
      particle_contrib<KIND>(A, i, chunk, g, scale, gs, ((i64)cell.y * A.nx + ix) * 2);
  }
  if (use_box) {
    __syncthreads();
    // a warp to a row of the box
    const int rows = nvals / (2 * (int)bnx), lane = threadIdx.x & 31;
    for (int row = threadIdx.x >> 5; row < rows; row += kDepThreads / 32) {
      const i64 ml = row / (int)bnr, r = row % (int)bnr + br0;
      unsigned long long *dst = A.acc + ((ml * A.nr + r) * A.nx + bx0) * 2;
      for (int c = lane; c < 2 * (int)bnx; c += 32) {
        const unsigned long long q = box[row * 2 * (int)bnx + c];
        if (q) atomicAdd(dst + c, q);
      }
    }
  }
}

// out = existing + acc / scale, then the ghost-row fold
// (grid_deps.f90:80-84): row1 -= row0; row0 = 0.
__global__ void finalize_kernel(double2 *__restrict__ out, const long long *__restrict__ acc,
                                const double *__restrict__ scale_p, i64 nx, i64 nr, i64 nml) {
  const double inv = 1.0 / scale_p[0];
  const i64 n = nx * nr * nml;
  for (i64 t = blockIdx.x * (i64)blockDim.x + threadIdx.x; t < n;
       t += (i64)gridDim.x * blockDim.x) {
    const i64 x = t % nx;
    const i64 rest = t / nx;
    const i64 r = rest % nr;
    if (r == 0) continue;
    double2 v = out[t];
    v.x += (double)acc[2 * t] * inv;
    v.y += (double)acc[2 * t + 1] * inv;
    if (r == 1) {
      const i64 t0 = t - nx;
      double2 g = out[t0];
      g.x += (double)acc[2 * t0] * inv;
      g.y += (double)acc[2 * t0 + 1] * inv;
      v = csub(v, g);
      out[t0] = make_double2(0.0, 0.0);
    }
    out[t] = v;
    (void)x;
  }
}

int deposit_common(int kind, const double *coord, i64 x_cs, i64 x_ps, const double *momenta,
                   i64 p_cs, i64 p_ps, const double *wghts, i64 w_ps, chm_c128 *grid,
                   const int32_t *ind, i64 nchnk, i64 guards, double leftX,
                   const double *rgrid, double dx_inv, double dr_inv, double kx0, i64 np, i64 nx,
                   i64 nr, i64 nm, void *ws, i64 ws_bytes, void *stream) {
  const int ncomp = ncomp_of(kind);
  CHM_REQUIRE(np >= 0 && nx > 1 && nr > 1 && nm >= 1, "deposit: bad dims");
  CHM_REQUIRE(kind < 2 || (nm % 2 == 1), "deposit env: nm must be odd");
  CHM_REQUIRE(grid && rgrid, "deposit: null grid/rgrid");
  CHM_REQUIRE(!ind || (nchnk >= 1 && nchnk <= 256), "deposit: nchnk must be in [1, 256]");
  const i64 need = chm_dep_ws_bytes(nx, nr, nm, ncomp, np);
  if (!ws || ws_bytes < need) {
    set_error("deposit: workspace %lld bytes < %lld required", (long long)ws_bytes,
              (long long)need);
    return CHM_ERR_WS;
  }
  cudaStream_t st = as_stream(stream);
  const i64 nacc = nx * nr * nm * ncomp * 2;
  unsigned long long *acc = reinterpret_cast<unsigned long long *>(ws);
  double *partial = reinterpret_cast<double *>(acc + nacc);
  double *scale = partial + kRedBlocks;
  if (cudaMemsetAsync(acc, 0, sizeof(unsigned long long) * nacc, st) != cudaSuccess) {
    set_error("deposit: memset failed");
    return CHM_ERR_CUDA;
  }
  if (np > 0) {
    CHM_REQUIRE(coord && wghts && (ncomp == 1 || momenta), "deposit: null particle array");
    wsum_partial_kernel<<<kRedBlocks, kDepThreads, 0, st>>>(wghts, w_ps, np, kind == DENS_ENV,
                                                            partial); chm::count_launch();
    wsum_final_kernel<<<1, 256, 0, st>>>(partial, kRedBlocks, scale); chm::count_launch();
    DepArgs A{};
    A.x = coord;
    A.x_cs = x_cs;
    A.x_ps = x_ps;
    A.p = momenta;
    A.p_cs = p_cs;
    A.p_ps = p_ps;
    A.w = wghts;
    A.w_ps = w_ps;
    A.leftX = leftX;
    A.dx_inv = dx_inv;
    A.dr_inv = dr_inv;
    A.kx0 = kx0;
    A.rgrid = rgrid;
    A.np = np;
    A.nx = nx;
    A.nr = nr;
    A.nm = (int)nm;
    A.ind = ind;
    A.nchnk = (int)nchnk;
    A.cs = ind ? nx / nchnk : nx;
    A.guards = guards;
    A.acc = acc;
    A.scale = scale;
    const unsigned blocks = (unsigned)((np + kPartPerBlock - 1) / kPartPerBlock);
    switch (kind) {
#define LAUNCH(K)                                                                         \
  case K:                                                                                 \
    cudaFuncSetAttribute(deposit_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                         kGeoBytes + kBoxBytes);                                          \
    deposit_kernel<K><<<blocks, kDepThreads, kGeoBytes + kBoxBytes, st>>>(A); chm::count_launch();            \
    break;
      LAUNCH(CURR)
      LAUNCH(DENS)
      LAUNCH(CURR_ENV)
      LAUNCH(DENS_ENV)
#undef LAUNCH
    }
    CHM_CHECK_LAUNCH();
  } else {
    // nothing deposited: only the fold of the existing content
    set_one_kernel<<<1, 1, 0, st>>>(scale); chm::count_launch();
  }
  const i64 nml = nm * ncomp;
  finalize_kernel<<<grid_for(nx * nr * nml, 256), 256, 0, st>>>(
      reinterpret_cast<double2 *>(grid), reinterpret_cast<const long long *>(acc), scale, nx,
      nr, nml); chm::count_launch();
  CHM_CHECK_LAUNCH();
  return CHM_OK;
}

}  // namespace

extern "C" {

int64_t chm_dep_ws_bytes(int64_t nx, int64_t nr, int64_t nm, int64_t ncomp, int64_t np) {
  (void)np;
  return 8 * (nx * nr * nm * ncomp * 2) + 8 * kRedBlocks + 256;
}

int chm_dep_curr(const double *coord, int64_t x_cs, int64_t x_ps, const double *momenta,
                 int64_t p_cs, int64_t p_ps, const double *wghts, int64_t w_ps, chm_c128 *curr,
                 double leftX, const double *rgrid, double dx_inv, double dr_inv, int64_t np,
                 int64_t nx, int64_t nr, int64_t nm, void *ws, int64_t ws_bytes, void *stream) {
  return deposit_common(CURR, coord, x_cs, x_ps, momenta, p_cs, p_ps, wghts, w_ps, curr, nullptr,
                        0, 0, leftX, rgrid, dx_inv, dr_inv, 0.0, np, nx, nr, nm, ws, ws_bytes,
                        stream);
}

int chm_dep_dens(const double *coord, int64_t x_cs, int64_t x_ps, const double *wghts,
                 int64_t w_ps, chm_c128 *dens, double leftX, const double *rgrid, double dx_inv,
                 double dr_inv, int64_t np, int64_t nx, int64_t nr, int64_t nm, void *ws,
                 int64_t ws_bytes, void *stream) {
  return deposit_common(DENS, coord, x_cs, x_ps, nullptr, 0, 0, wghts, w_ps, dens, nullptr, 0, 0,
                        leftX, rgrid, dx_inv, dr_inv, 0.0, np, nx, nr, nm, ws, ws_bytes, stream);
}

int chm_dep_curr_env(const double *coord, int64_t x_cs, int64_t x_ps, const double *momenta,
                     int64_t p_cs, int64_t p_ps, const double *wghts, int64_t w_ps,
                     chm_c128 *curr, double leftX, const double *rgrid, double dx_inv,
                     double dr_inv, double kx0, int64_t np, int64_t nx, int64_t nr, int64_t nm,
                     void *ws, int64_t ws_bytes, void *stream) {
  return deposit_common(CURR_ENV, coord, x_cs, x_ps, momenta, p_cs, p_ps, wghts, w_ps, curr,
                        nullptr, 0, 0, leftX, rgrid, dx_inv, dr_inv, kx0, np, nx, nr, nm, ws,
                        ws_bytes, stream);
}

int chm_dep_dens_env(const double *coord, int64_t x_cs, int64_t x_ps, const double *wghts,
                     int64_t w_ps, chm_c128 *dens, double leftX, const double *rgrid,
                     double dx_inv, double dr_inv, double kx0, int64_t np, int64_t nx, int64_t nr,
                     int64_t nm, void *ws, int64_t ws_bytes, void *stream) {
  return deposit_common(DENS_ENV, coord, x_cs, x_ps, nullptr, 0, 0, wghts, w_ps, dens, nullptr, 0,
                        0, leftX, rgrid, dx_inv, dr_inv, kx0, np, nx, nr, nm, ws, ws_bytes,
                        stream);
}

int chm_dep_curr_chnk(const double *coord, int64_t x_cs, int64_t x_ps, const double *momenta,
                      int64_t p_cs, int64_t p_ps, const double *wghts, int64_t w_ps,
                      chm_c128 *curr, const int32_t *ind_in_chunk, int64_t nchnk, int64_t guards,
                      double leftX, const double *rgrid, double dx_inv, double dr_inv,
                      int64_t np, int64_t nx, int64_t nr, int64_t nm, void *ws, int64_t ws_bytes,
                      void *stream) {
  CHM_REQUIRE(ind_in_chunk, "dep_curr_chnk: null IndInChunk");
  return deposit_common(CURR, coord, x_cs, x_ps, momenta, p_cs, p_ps, wghts, w_ps, curr,
                        ind_in_chunk, nchnk, guards, leftX, rgrid, dx_inv, dr_inv, 0.0, np, nx,
                        nr, nm, ws, ws_bytes, stream);
}

int chm_dep_dens_chnk(const double *coord, int64_t x_cs, int64_t x_ps, const double *wghts,
                      int64_t w_ps, chm_c128 *dens, const int32_t *ind_in_chunk, int64_t nchnk,
                      int64_t guards, double leftX, const double *rgrid, double dx_inv,
                      double dr_inv, int64_t np, int64_t nx, int64_t nr, int64_t nm, void *ws,
                      int64_t ws_bytes, void *stream) {
  CHM_REQUIRE(ind_in_chunk, "dep_dens_chnk: null IndInChunk");
  return deposit_common(DENS, coord, x_cs, x_ps, nullptr, 0, 0, wghts, w_ps, dens, ind_in_chunk,
                        nchnk, guards, leftX, rgrid, dx_inv, dr_inv, 0.0, np, nx, nr, nm, ws,
                        ws_bytes, stream);
}

int chm_dep_curr_env_chnk(const double *coord, int64_t x_cs, int64_t x_ps, const double *momenta,
                          int64_t p_cs, int64_t p_ps, const double *wghts, int64_t w_ps,
                          chm_c128 *curr, const int32_t *ind_in_chunk, int64_t nchnk,
                          int64_t guards, double leftX, const double *rgrid, double dx_inv,
                          double dr_inv, double kx0, int64_t np, int64_t nx, int64_t nr,
                          int64_t nm, void *ws, int64_t ws_bytes, void *stream) {
  CHM_REQUIRE(ind_in_chunk, "dep_curr_env_chnk: null IndInChunk");
  return deposit_common(CURR_ENV, coord, x_cs, x_ps, momenta, p_cs, p_ps, wghts, w_ps, curr,
                        ind_in_chunk, nchnk, guards, leftX, rgrid, dx_inv, dr_inv, kx0, np, nx,
                        nr, nm, ws, ws_bytes, stream);
}

int chm_dep_dens_env_chnk(const double *coord, int64_t x_cs, int64_t x_ps, const double *wghts,
                          int64_t w_ps, chm_c128 *dens, const int32_t *ind_in_chunk,
                          int64_t nchnk, int64_t guards, double leftX, const double *rgrid,
                          double dx_inv, double dr_inv, double kx0, int64_t np, int64_t nx,
                          int64_t nr, int64_t nm, void *ws, int64_t ws_bytes, void *stream) {
  CHM_REQUIRE(ind_in_chunk, "dep_dens_env_chnk: null IndInChunk");
  return deposit_common(DENS_ENV, coord, x_cs, x_ps, nullptr, 0, 0, wghts, w_ps, dens,
                        ind_in_chunk, nchnk, guards, leftX, rgrid, dx_inv, dr_inv, kx0, np, nx,
                        nr, nm, ws, ws_bytes, stream);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free current deposit
//
// Some callers of this library cannot allocate device memory: a host code
// that reaches the GPU only through this C ABI (an FFI binding with no CUDA
// allocator of its own), or a loop whose device memory budget is fixed at
// start-up and that may not call cudaMalloc mid-run (cudaMalloc can
// synchronise the device and stall other streams).  For them,
// chm_dep_curr_noalloc runs the same deposit as chm_dep_curr with its scratch
// (the 64-bit accumulator, the weight partial sums and the scale) in the
// static device array below instead of a caller-provided workspace.
// ---------------------------------------------------------------------------
#include <mutex>

namespace {

constexpr int64_t kNoAllocScratchBytes = 16LL << 20;  // 16 MiB, held per GPU until exit
static __device__ __align__(256) unsigned char g_dep_scratch[kNoAllocScratchBytes];

std::mutex g_noalloc_mutex;
void *g_noalloc_ptr[128] = {};  // device address of g_dep_scratch, per device

// Resolves (once per device, with that device current) the device address of
// the static scratch; host code cannot pass g_dep_scratch itself, whose name
// on the host is only a stand-in for the symbol.
int noalloc_scratch(void **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 128) {
    set_error("dep_curr_noalloc: cudaGetDevice failed (%s)", cudaGetErrorString(e));
    return CHM_ERR_CUDA;
  }
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ptr[dev]) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_dep_scratch);
    if (e != cudaSuccess || !p) {
      set_error("dep_curr_noalloc: cudaGetSymbolAddress failed (%s)", cudaGetErrorString(e));
      return CHM_ERR_CUDA;
    }
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return CHM_OK;
}

}  // namespace

extern "C" int64_t chm_dep_noalloc_max_bytes(void) { return kNoAllocScratchBytes; }

extern "C" int chm_dep_curr_noalloc(const double *coord, int64_t x_cs, int64_t x_ps,
                                    const double *momenta, int64_t p_cs, int64_t p_ps,
                                    const double *wghts, int64_t w_ps, chm_c128 *curr,
                                    double leftX, const double *rgrid, double dx_inv,
                                    double dr_inv, int64_t np, int64_t nx, int64_t nr, int64_t nm,
                                    void *stream) {
  // the grid's own rules first (as chm_dep_curr checks them), then its size
  // against the static array, without an overflowing product
  if (nx <= 1 || nr <= 1 || nm < 1) {
    set_error("dep_curr_noalloc: bad grid (%lld, %lld, %lld): nx > 1, nr > 1 and nm >= 1 are "
              "required", (long long)nx, (long long)nr, (long long)nm);
    return CHM_ERR_ARG;
  }
  int64_t nodes = 0, need = 0;
  const bool big = __builtin_mul_overflow(nx, nr, &nodes) || __builtin_mul_overflow(nodes, nm, &nodes) ||
                   nodes > (kNoAllocScratchBytes - 8 * kRedBlocks - 256) / 48;
  if (!big) need = chm_dep_ws_bytes(nx, nr, nm, 3, np);
  if (big || need > kNoAllocScratchBytes) {
    set_error("dep_curr_noalloc: a (%lld, %lld, %lld, 3) grid needs more scratch than the "
              "%lld-byte static array; use chm_dep_curr with a workspace",
              (long long)nx, (long long)nr, (long long)nm, (long long)kNoAllocScratchBytes);
    return CHM_ERR_RANGE;
  }
  void *scratch = nullptr;
  int rc = noalloc_scratch(&scratch);
  if (rc) return rc;
  // deposit_common zeroes the accumulator at the start of every call
  return deposit_common(CURR, coord, x_cs, x_ps, momenta, p_cs, p_ps, wghts, w_ps, curr, nullptr, 0,
                        0, leftX, rgrid, dx_inv, dr_inv, 0.0, np, nx, nr, nm, scratch,
                        kNoAllocScratchBytes, stream);
}
