// Batched shared-memory FFT along x (FP64).  See fft.cuh.
#include <math.h>

#include "fft.cuh"
#include "fft_mixed.cuh"

namespace chm {

static constexpr double kPi = 3.14159265358979323846;

bool fft_make_plan(int n, FftPlan *p) {
  if (n < 1 || n > kFftMaxN) return false;
  p->n = n;
  p->nstages = 0;
  int m = n;
  while (m % 4 == 0 && p->nstages < kFftMaxStages) {
    p->radix[p->nstages++] = 4;
    m /= 4;
  }
  const int small[4] = {2, 3, 5, 7};
  for (int s = 0; s < 4; ++s)
    while (m % small[s] == 0 && p->nstages < kFftMaxStages) {
      p->radix[p->nstages++] = small[s];
      m /= small[s];
    }
  for (int f = 11; m > 1 && p->nstages < kFftMaxStages;) {
    if ((i64)f * f > m) f = m;
    if (m % f == 0) {
      p->radix[p->nstages++] = f;
      m /= f;
    } else {
      f += 2;
    }
  }
  return m == 1;
}

// shift[x] = exp(sign i kx[x] leftX) (fb_io.f90:40 / :120) and the twiddles
// tw[x] = exp(-2 pi i x / n), in the first and the second half of the blocks.
// Launched with warp-sized blocks, so that the FP64 trigonometry, a chain of
// dependent operations, spreads over as many SMs as there are warps of work (n =
// 2048: 5.3 us with both in one thread, 4.0 so; with 256-thread blocks and a
// launch for each table 9.8).
__global__ void fft_tables_kernel(double2 *__restrict__ shift, double2 *__restrict__ tw,
                                  const double *__restrict__ kx, double leftX, int sign, int n) {
  const int half = (int)(gridDim.x / 2 * blockDim.x), t = blockIdx.x * blockDim.x + threadIdx.x;
  const int x = t < half ? t : t - half;
  if (x >= n) return;
  double s, c;
  if (t < half) {
    sincos(leftX * kx[x], &s, &c);
    shift[x] = make_double2(c, sign * s);
  } else {
    // sincospi keeps the argument exact
    sincospi(2.0 * (double)x / (double)n, &s, &c);
    tw[x] = make_double2(c, -s);
  }
}

// W^t for the table of the forward transform; sign=+1 conjugates.
__device__ __forceinline__ double2 twid(const double2 *__restrict__ tw, int t, int sign) {
  double2 w = tw[t];
  if (sign > 0) w.y = -w.y;
  return w;
}

// One Stockham pass with radix R over a line in shared memory.
__device__ void stockham_pass(const double2 *__restrict__ src, double2 *__restrict__ dst, int n,
                              int R, int Ns, const double2 *__restrict__ tw, int sign) {
  const int nb = n / R;
  for (int j = threadIdx.x; j < nb; j += blockDim.x) {
    const int k = j % Ns;
    double2 v[16];
    const int tstep = (n / (Ns * R)) * k;  // twiddle index step per r
    if (R <= 16) {
      for (int r = 0; r < R; ++r) {
        double2 a = src[j + r * nb];
        if (r > 0 && k > 0) a = cmul(a, twid(tw, (r * tstep) % n, sign));
        v[r] = a;
      }
      const int base = (j / Ns) * Ns * R + k;
      if (R == 2) {
        dst[base] = cadd(v[0], v[1]);
        dst[base + Ns] = csub(v[0], v[1]);
      } else if (R == 4) {
        double2 a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]);
        double2 a2 = cadd(v[1], v[3]), a3 = csub(v[1], v[3]);
        // multiply a3 by -i (forward) or +i (backward)
        double2 a3r = sign < 0 ? make_double2(a3.y, -a3.x) : make_double2(-a3.y, a3.x);
        dst[base] = cadd(a0, a2);
        dst[base + Ns] = cadd(a1, a3r);
        dst[base + 2 * Ns] = csub(a0, a2);
        dst[base + 3 * Ns] = csub(a1, a3r);
      } else {
        const int step = n / R;
        for (int q = 0; q < R; ++q) {
          double2 acc = v[0];
          for (int r = 1; r < R; ++r) acc = cadd(acc, cmul(v[r], twid(tw, ((r * q) % R) * step, sign)));
          dst[base + q * Ns] = acc;
        }
      }
    } else {
      // large prime radix: direct DFT reading straight from src
      const int base = (j / Ns) * Ns * R + k;
      const int step = n / R;
      for (int q = 0; q < R; ++q) {
        double2 acc = make_double2(0.0, 0.0);
        for (int r = 0; r < R; ++r) {
          double2 a = src[j + r * nb];
          if (r > 0 && k > 0) a = cmul(a, twid(tw, (r * tstep) % n, sign));
          acc = cadd(acc, cmul(a, twid(tw, ((r * q) % R) * step, sign)));
        }
        dst[base + q * Ns] = acc;
      }
    }
  }
}

// Runs all passes; returns the buffer holding the result.
__device__ double2 *run_fft(FftPlan plan, double2 *a, double2 *b, const double2 *__restrict__ tw,
                            int sign) {
  int Ns = 1;
  for (int s = 0; s < plan.nstages; ++s) {
    const int R = plan.radix[s];
    __syncthreads();
    stockham_pass(a, b, plan.n, R, Ns, tw, sign);
    Ns *= R;
    double2 *t = a;
    a = b;
    b = t;
  }
  __syncthreads();
  return a;
}

// MIX: register passes in place (fft_mixed.cuh); else the general passes between
// two buffers, for lengths with a prime factor above 13.  FP64-pipe bound (2
// operations a clock and SM): the 5120 lines of 2048 values of a field step at
// 2048 x 256 x 2 modes, some 44 operations a value, ran 1041 us with the general
// passes and 830 with the register passes, of which the pipe needs 780.
template <bool MIX>
__global__ void __launch_bounds__(512) fft_lines_kernel(FftPlan plan, MixPlan mix, const double2 *__restrict__ tw,
                                                        FftLines L) {
  extern __shared__ __align__(16) double2 sm[];
  const int n = MIX ? mix.n : plan.n;
  double2 *a = sm, *b = sm + (MIX ? 0 : n);
  const i64 line = blockIdx.x;
  const i64 ib = line / L.in_rows, ir = line % L.in_rows;
  const double2 *src = L.in + (ib * L.in_rows_tot + ir + L.in_row_off) * (i64)n;
#pragma unroll 4
  for (int x = threadIdx.x; x < n; x += blockDim.x) {
    double2 v = src[x];
    if (L.pre_shift) v = cmul(v, L.pre_shift[x]);
    a[x] = MIX ? mx_swap(v, L.sign > 0) : v;
  }
  double2 *res = a;
  bool swapped = MIX && L.sign > 0;
  if constexpr (MIX) {
    __syncthreads();
    mx_fft(mix, a, tw);
  } else {
    res = run_fft(plan, a, b, tw, L.sign);
  }
  if (L.filt_mode >= 0) {
    // fb_io.f90:255-304: profile on the first / last nxfilt cells, then the
    // forward FFT and 1/(N shift)
    for (int x = threadIdx.x; x < L.nxfilt; x += blockDim.x) {
      if (L.filt_mode == 0 || L.filt_mode == 2) res[x] = cscale(res[x], L.filtr[x]);
    }
    __syncthreads();
    for (int x = threadIdx.x; x < L.nxfilt; x += blockDim.x) {
      if (L.filt_mode == 1 || L.filt_mode == 2) res[n - 1 - x] = cscale(res[n - 1 - x], L.filtr[x]);
    }
    if constexpr (MIX) {
      __syncthreads();
      for (int x = threadIdx.x; x < n; x += blockDim.x) a[x] = mx_swap(a[x], swapped);
      swapped = false;
      __syncthreads();
      mx_fft(mix, a, tw);
    } else {
      double2 *other = (res == a) ? b : a;
      res = run_fft(plan, res, other, tw, -1);
    }
  }
  const i64 ob = line / L.out_rows, orow = line % L.out_rows;
  double2 *dst = L.out + (ob * L.out_rows_tot + orow + L.out_row_off) * (i64)n;
  double fac = 1.0, sg = 1.0;
  if (L.eb_mode) {
    const int m = (int)(ob % L.nm);
    const double pi_inv = 1.0 / kPi;
    if (L.eb_mode == 1) {
      fac = (m == 0) ? 0.5 * pi_inv : pi_inv;
      sg = (m == 0) ? 1.0 : -1.0;
    } else {
      fac = pi_inv;
      sg = (L.nm == 1) ? 1.0 : -1.0;
    }
  }
  const bool ghost = L.eb_mode && orow == 0;
  double2 *gdst = L.out + (ob * L.out_rows_tot) * (i64)n;
  for (int x = threadIdx.x; x < n; x += blockDim.x) {
    double2 v = MIX ? mx_swap(res[x], swapped) : res[x];
    if (L.filt_mode >= 0) {
      // times 1/(N e^{+i kx leftX}) = conj(shift)/N with |shift| = 1 is not
      // bit-identical; divide as the Fortran does
      double2 s = L.pre_shift[x];
      double d = (double)n * (s.x * s.x + s.y * s.y);
      v = cmul(v, make_double2(s.x / d, -s.y / d));
    }
    if (L.eb_mode) v = cscale(v, fac);
    dst[x] = v;
    if (ghost) gdst[x] = cscale(v, sg);
  }
}

void fft_tables(double2 *shift, double2 *tw, const double *kx, double leftX, int sign, int n, cudaStream_t st) {
  fft_tables_kernel<<<2 * ((n + 31) / 32), 32, 0, st>>>(shift, tw, kx, leftX, sign, n);
  count_launch();
}

int fft_launch(const FftLines &L, int n, i64 nlines, const double2 *tw, cudaStream_t st) {
  FftPlan plan{};
  MixPlan mix{};
  const bool mixed = mix_plan(n, nlines, 128, &mix);
  if (!mixed && !fft_make_plan(n, &plan)) {
    set_error("fft: unsupported length %d (max %d)", n, kFftMaxN);
    return CHM_ERR_RANGE;
  }
  if (nlines <= 0) return CHM_OK;
  const int smem = (mixed ? 1 : 2) * n * (int)sizeof(double2);
  const int threads = mixed ? mix.threads : n >= 1024 ? 512 : (n >= 256 ? 256 : 128);
  auto kern = mixed ? fft_lines_kernel<true> : fft_lines_kernel<false>;
  // (one limit for every length: calls from other threads may have others)
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (mixed ? 1 : 2) * kFftMaxN * (int)sizeof(double2));
  kern<<<(unsigned)nlines, threads, smem, st>>>(plan, mix, tw, L);
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("fft: %s", cudaGetErrorString(e));
    return CHM_ERR_CUDA;
  }
  return CHM_OK;
}

}  // namespace chm
