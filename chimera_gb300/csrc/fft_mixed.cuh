// Mixed-radix FFT of a line in shared memory, in place: Stockham passes whose
// butterflies (radix 2 .. 16) are done in registers, FP64 (fft.cu) and FP32
// (split_spectral.cu).  A pass reads all of a thread's inputs, synchronises and
// writes the outputs, so one buffer serves (half the shared memory of two, and
// twice the resident lines); composite radices (16 = 4 x 4, 15 = 3 x 5, ...)
// take a length of up to 4096 in three passes or four.  Odd primes use the
// symmetric form: X_k and X_(P-k) from the sums and differences of x_j and
// x_(P-j), (P - 1)^2 real multiply-adds for a complex point set instead of 4
// (P - 1)^2.
#pragma once
#include <type_traits>

#include "common.cuh"

namespace chm {

// ----------------------------------------------------------------------
// host side: the passes of a length
// ----------------------------------------------------------------------
constexpr int kMixMaxPasses = 12;
struct MixPlan {
  int n, np, threads;
  bool few;
  int radix[kMixMaxPasses];
  unsigned ns_magic[kMixMaxPasses];  // division by Ns: see mix_div
};

// butterflies a thread holds at once: at most 16 values
__host__ __device__ constexpr int mix_batch(int R) { return R >= 9 ? 1 : 16 / R; }

inline bool mix_search(int m, int left, int from, const int *rad, int nrad, MixPlan *p) {
  if (m == 1) return true;
  if (left == 0) return false;
  for (int i = from; i < nrad; ++i)
    if (m % rad[i] == 0) {
      p->radix[p->np++] = rad[i];
      if (mix_search(m / rad[i], left - 1, i, rad, nrad, p)) return true;
      --p->np;
    }
  return false;
}

// The fewest passes, larger radices first; false for a length with a prime
// factor above 13 (those take the general kernels).  few: while all lines of a
// launch fit the chip's threads (2048 an SM) with a thread for each value, what
// counts is the time of one line, not the SM's throughput.  Then radices up to 5,
// a butterfly to a thread (an SM's four FP64 units share a line) and up to few_threads
// threads to a line (four launches of 384 FP64 lines of 512 values: some 70 us, with
// radix 16 on 32 threads 134).  So the last bits of a line's transform depend on how
// many lines are launched with it (a scalar's and a vector's component differ).
inline bool mix_plan(int n, i64 nlines, int few_threads, MixPlan *p) {
  const bool few = nlines * n <= (i64)sm_count() * 2048;
  static const int rads[] = {16, 15, 14, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};
  static const int few_rads[] = {5, 4, 3, 7, 11, 13, 2};
  const int *rad = few ? few_rads : rads, nrad = few ? 7 : 15;
  if (n < 2 || n > 4096) return false;
  int m = n;
  for (int f : {2, 3, 5, 7, 11, 13})
    while (m % f == 0) m /= f;
  if (m != 1) return false;
  p->n = n;
  p->few = few;
  for (int k = 1; k <= kMixMaxPasses; ++k) {
    p->np = 0;
    if (mix_search(n, k, 0, rad, nrad, p)) {
      int t = few ? (n < few_threads ? n : few_threads) : 1, Ns = 1;
      for (int i = 0; i < p->np; ++i) {
        const int nb = n / p->radix[i];
        int B = mix_batch(p->radix[i]);
        if (few && (nb + few_threads - 1) / few_threads < B) B = (nb + few_threads - 1) / few_threads;
        if ((nb + B - 1) / B > t) t = (nb + B - 1) / B;
        p->ns_magic[i] = Ns > 1 ? 0xffffffffu / (unsigned)Ns + 1u : 0u;
        Ns *= p->radix[i];
      }
      p->threads = (t + 31) / 32 * 32;
      return true;
    }
  }
  return false;
}

#ifdef __CUDACC__
// q = j / Ns for j, Ns < 2^16 (m Ns = 2^32 + e, 0 <= e < Ns, and j e < 2^32)
__device__ __forceinline__ int mix_div(int j, unsigned m) { return m ? (int)__umulhi((unsigned)j, m) : j; }

// ----------------------------------------------------------------------
// cos and sin of 2 pi k / N, evaluated at compile time: the angle is reduced
// exactly to [0, pi / 4], then a Taylor sum in pairs of doubles (Dekker's sums
// and products), so that the constants are rounded once
// ----------------------------------------------------------------------
struct MixDD {
  double h, l;
};
constexpr MixDD mix_sum(double a, double b) {
  const double s = a + b, t = s - a;
  return {s, (a - (s - t)) + (b - t)};
}
constexpr MixDD mix_add(MixDD a, MixDD b) {
  const MixDD s = mix_sum(a.h, b.h);
  return mix_sum(s.h, s.l + a.l + b.l);
}
constexpr MixDD mix_prod(double a, double b) {
  const double ca = 134217729.0 * a, cb = 134217729.0 * b;
  const double ah = ca - (ca - a), al = a - ah, bh = cb - (cb - b), bl = b - bh, p = a * b;
  return {p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
constexpr MixDD mix_mul(MixDD a, MixDD b) {
  const MixDD p = mix_prod(a.h, b.h);
  return mix_sum(p.h, p.l + (a.h * b.l + a.l * b.h));
}
constexpr MixDD mix_quot(MixDD a, double d) {
  const double q = a.h / d;
  const MixDD p = mix_prod(q, -d), r = mix_add(a, p);
  return mix_sum(q, r.h / d);
}
// cos(2 pi k / N) for 0 <= 8 k <= N, or sin
constexpr double mix_octant(int k, int N, bool sine) {
  const MixDD tau = {6.283185307179586, 2.4492935982947064e-16};
  const MixDD x = mix_quot(mix_mul(tau, {(double)k, 0.0}), (double)N), x2 = mix_mul(x, {-x.h, -x.l});
  MixDD term = sine ? x : MixDD{1.0, 0.0}, sum = {0.0, 0.0};
  MixDD t[16] = {};
  for (int i = 0; i < 16; ++i) {
    t[i] = term;
    const int a = 2 * i + (sine ? 2 : 1);
    term = mix_quot(mix_mul(term, x2), (double)a * (a + 1));
  }
  for (int i = 15; i >= 0; --i) sum = mix_add(t[i], sum);  // the small terms first
  return sum.h;
}
constexpr double mix_cos(int k, int N) {
  k %= N;
  if (2 * k > N) k = N - k;                        // cos(2 pi - a)
  if (4 * k > N) {                                 // -cos(pi - a), over 2 N
    const int a = N - 2 * k;                       // pi - a = 2 pi a / (2 N)
    return 8 * a <= 2 * N ? -mix_octant(a, 2 * N, false) : -mix_octant(N - 2 * a, 4 * N, true);
  }
  return 8 * k <= N ? mix_octant(k, N, false) : mix_octant(N - 4 * k, 4 * N, true);
}
constexpr double mix_sin(int k, int N) {           // cos(a - pi / 2), over 4 N
  k %= N;
  return mix_cos(4 * k + 3 * N, 4 * N);
}

constexpr int mix_bitrev(int i, int L) {
  int r = 0;
  for (int b = 0; b < L; ++b) r |= ((i >> b) & 1) << (L - 1 - b);
  return r;
}

template <typename C>
struct MixScalar;
template <>
struct MixScalar<float2> {
  using T = float;
  static __device__ __forceinline__ float2 make(float x, float y) { return make_float2(x, y); }
};
template <>
struct MixScalar<double2> {
  using T = double;
  static __device__ __forceinline__ double2 make(double x, double y) { return make_double2(x, y); }
};

template <typename C>
__device__ __forceinline__ C mx(typename MixScalar<C>::T x, typename MixScalar<C>::T y) {
  return MixScalar<C>::make(x, y);
}
template <typename C>
__device__ __forceinline__ C mx_add(C a, C b) { return mx<C>(a.x + b.x, a.y + b.y); }
template <typename C>
__device__ __forceinline__ C mx_sub(C a, C b) { return mx<C>(a.x - b.x, a.y - b.y); }
template <typename C>
__device__ __forceinline__ C mx_mul(C a, C b) { return mx<C>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
template <typename C>
__device__ __forceinline__ C mx_mi(C a) { return mx<C>(a.y, -a.x); }  // -i a

template <int K, int N, typename C>
__device__ __forceinline__ C mx_const() {  // e^(-2 pi i K / N)
  constexpr double c = mix_cos(K, N), s = mix_sin(K, N);
  return mx<C>((typename MixScalar<C>::T)c, (typename MixScalar<C>::T)(-s));
}

#define MX_INLINE __attribute__((always_inline))
// compile-time loop
template <int I, int E, typename F>
__device__ __forceinline__ void mx_for(F f) {
  if constexpr (I < E) {
    f(std::integral_constant<int, I>{});
    mx_for<I + 1, E>(f);
  }
}

// DFT of the P values v[0], v[S], ... (P = 2, 4 or an odd prime), in place
template <int P, int S, typename C>
__device__ __forceinline__ void mx_dft(C *v) {
  using T = typename MixScalar<C>::T;
  if constexpr (P == 2) {
    const C a = v[0];
    v[0] = mx_add(a, v[S]);
    v[S] = mx_sub(a, v[S]);
  } else if constexpr (P == 4) {
    const C a0 = mx_add(v[0], v[2 * S]), a1 = mx_sub(v[0], v[2 * S]), a2 = mx_add(v[S], v[3 * S]);
    const C a3 = mx_mi(mx_sub(v[S], v[3 * S]));
    v[0] = mx_add(a0, a2);
    v[2 * S] = mx_sub(a0, a2);
    v[S] = mx_add(a1, a3);
    v[3 * S] = mx_sub(a1, a3);
  } else {
    constexpr int H = (P - 1) / 2;
    C s[H], d[H];
    const C x0 = v[0];
    C sum = x0;
    mx_for<0, H>([&](auto j) MX_INLINE {
      s[j()] = mx_add(v[(j() + 1) * S], v[(P - 1 - j()) * S]);
      d[j()] = mx_sub(v[(j() + 1) * S], v[(P - 1 - j()) * S]);
      sum = mx_add(sum, s[j()]);
    });
    v[0] = sum;
    mx_for<1, H + 1>([&](auto k) MX_INLINE {
      C a = x0, b = mx<C>(0, 0);
      mx_for<1, H + 1>([&](auto j) MX_INLINE {
        constexpr double c = mix_cos(j() * k(), P), z = -mix_sin(j() * k(), P);
        const C &sj = s[j() - 1], &dj = d[j() - 1];
        a = mx<C>(a.x + (T)c * sj.x, a.y + (T)c * sj.y);
        b = mx<C>(b.x + (T)z * dj.x, b.y + (T)z * dj.y);
      });
      // X_k = a + i b, X_(P-k) = a - i b
      v[k() * S] = mx<C>(a.x - b.y, a.y + b.x);
      v[(P - k()) * S] = mx<C>(a.x + b.y, a.y - b.x);
    });
  }
}

// radix R = A B: input n = B n1 + n2, output k = k1 + A k2 left in v[B k1 + k2]
template <int A, int B, typename C>
__device__ __forceinline__ void mx_dft2(C *v) {
  if constexpr (B == 1) {
    mx_dft<A, 1>(v);
  } else {
    mx_for<0, B>([&](auto n2) MX_INLINE { mx_dft<A, B>(v + n2()); });
    mx_for<1, A>([&](auto k1) MX_INLINE {
      mx_for<1, B>([&](auto n2) MX_INLINE {
        constexpr int K = n2() * k1();
        C &x = v[B * k1() + n2()];
        if constexpr (4 * K == A * B) x = mx_mi(x);
        else x = mx_mul(x, mx_const<K, A * B, C>());
      });
    });
    mx_for<0, A>([&](auto k1) MX_INLINE { mx_dft<B, 1>(v + B * k1()); });
  }
}

// Radix R = 2^L with the pass's twiddles inside: L levels of radix-2 butterflies
// a +- w b as fused multiply-adds, 8 operations where a product and two sums take
// 10, and R / 2 twiddles instead of R - 1 (the other half are -i times these).
// (a - w b as 2 a - (a + w b) takes 6, but hands the first one's rounding on: the
// error of a transform of 2048 grew by a tenth.)  w^e = tw[e], step = n / (R Ns).
template <int L, typename C>
__device__ __forceinline__ void mx_dft_pow2(C *v, int n, int ke, const C *tw) {
  constexpr int R = 1 << L;
  mx_for<1, L + 1>([&](auto s) MX_INLINE {
    constexpr int h = 1 << (s() - 1), J = h > 1 ? h / 2 : 1;
    mx_for<0, J>([&](auto j) MX_INLINE {
      const C w = tw[ke * (R >> s()) + j() * (n >> s())];
      mx_for<0, R / (2 * h)>([&](auto b) MX_INLINE {
        mx_for<0, (h > 1 ? 2 : 1)>([&](auto half) MX_INLINE {
          constexpr int lo = b() * 2 * h + j() + half() * (h / 2);
          // values of the level stand in bit-reversed order
          constexpr int il = mix_bitrev(lo, L), io = mix_bitrev(lo + h, L);
          const C a = v[il], o = v[io], z = half() ? mx_mi(w) : w;
          const C x = mx<C>(fma(-z.y, o.y, fma(z.x, o.x, a.x)), fma(z.y, o.x, fma(z.x, o.y, a.y)));
          v[il] = x;
          v[io] = mx<C>(fma(z.y, o.y, fma(-z.x, o.x, a.x)), fma(-z.y, o.x, fma(-z.x, o.y, a.y)));
        });
      });
    });
  });
}

// One forward pass over the line in a[0 .. n), T = blockDim threads; tw[t] =
// e^(-2 pi i t / n) in global or shared memory.  LOG: log2 of the radix where it is a power
// of two.
template <int A, int B, int LOG, typename C>
__device__ __forceinline__ void mx_pass(C *a, int n, int Ns, unsigned magic, const C *tw) {
  constexpr int R = A * B, NB = mix_batch(R);
  const int nb = n / R, T = blockDim.x, step = nb / Ns;
  C v[NB * R];
  // set for every thread: values set under a condition alone would be live
  // through the whole switch over the radices
  mx_for<0, NB * R>([&](auto i) MX_INLINE { v[i()] = mx<C>(0, 0); });
  mx_for<0, NB>([&](auto b) MX_INLINE {
    const int j = threadIdx.x + b() * T;
    if (j < nb) mx_for<0, R>([&](auto r) MX_INLINE { v[b() * R + r()] = a[j + r() * nb]; });
  });
  __syncthreads();
  mx_for<0, NB>([&](auto b) MX_INLINE {
    const int j = threadIdx.x + b() * T;
    if (j < nb) {
      const int q = mix_div(j, magic), k = j - q * Ns;
      C *dst = a + q * Ns * R + k, *u = v + b() * R;
      if (LOG > 0 && Ns > 1) {
        mx_dft_pow2<LOG>(u, n, k * step, tw);
        mx_for<0, R>([&](auto i) MX_INLINE { dst[i() * Ns] = u[mix_bitrev(i(), LOG)]; });
      } else {
        if (Ns > 1)
          mx_for<1, R>([&](auto r) MX_INLINE { u[r()] = mx_mul(u[r()], tw[r() * k * step]); });
        mx_dft2<A, B>(u);
        mx_for<0, R>([&](auto i) MX_INLINE { dst[i() * Ns] = u[B * (i() % A) + i() / A]; });
      }
    }
  });
  __syncthreads();
}

// The whole forward transform; the caller has synchronised after filling a.  The
// backward one is this one between two exchanges of the real and imaginary parts
// (mx_swap), which cost nothing where the line is filled and read: one set of
// passes serves both.
template <typename C>
__device__ __forceinline__ C mx_swap(C v, bool yes) { return yes ? mx<C>(v.y, v.x) : v; }

template <typename C>
__device__ __forceinline__ void mx_fft(const MixPlan &P, C *a, const C *tw) {
  const int n = P.n;
  int Ns = 1;
  for (int i = 0; i < P.np; ++i) {
    const int R = P.radix[i];
    const unsigned m = P.ns_magic[i];
    switch (R) {
      case 2: mx_pass<2, 1, 1>(a, n, Ns, m, tw); break;
      case 3: mx_pass<3, 1, 0>(a, n, Ns, m, tw); break;
      case 4: mx_pass<4, 1, 2>(a, n, Ns, m, tw); break;
      case 5: mx_pass<5, 1, 0>(a, n, Ns, m, tw); break;
      case 6: mx_pass<2, 3, 0>(a, n, Ns, m, tw); break;
      case 7: mx_pass<7, 1, 0>(a, n, Ns, m, tw); break;
      case 8: mx_pass<4, 2, 3>(a, n, Ns, m, tw); break;
      case 9: mx_pass<3, 3, 0>(a, n, Ns, m, tw); break;
      case 10: mx_pass<2, 5, 0>(a, n, Ns, m, tw); break;
      case 11: mx_pass<11, 1, 0>(a, n, Ns, m, tw); break;
      case 12: mx_pass<4, 3, 0>(a, n, Ns, m, tw); break;
      case 13: mx_pass<13, 1, 0>(a, n, Ns, m, tw); break;
      case 14: mx_pass<2, 7, 0>(a, n, Ns, m, tw); break;
      case 15: mx_pass<3, 5, 0>(a, n, Ns, m, tw); break;
      default: mx_pass<4, 4, 4>(a, n, Ns, m, tw); break;
    }
    Ns *= R;
  }
}
#endif

}  // namespace chm
