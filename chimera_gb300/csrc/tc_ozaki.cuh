// FP64 products on the BF16 tensor cores: C(M, N) = A(M, K) B(K, N) with the
// operands cut into exact integer slices (tc_ozaki.cu).
#pragma once
#include "common.cuh"

namespace chm {

struct OzProblem {
  const double *A;    // (M, K) column-major, ld = M
  const double *B;    // (K, N) column-major, ld = K
  double *C;          // (M, N) column-major, ld = M
  const double *fac;  // optional real (M / 2, N) factor of the shift epilogue
  // read A as the reflected complex plane: row (x, c) of A is (c ? 1 : -1) *
  // row ((M/2 - x) mod M/2, c) of the stored plane (fb_math.f90:35-36)
  int reflect;
};

constexpr int kOzMaxProblems = 48;

// scratch of a batch with nA distinct A planes and nB distinct B matrices
i64 oz_ws_bytes(i64 M, i64 N, i64 K, i64 nA, i64 nB);

// whether the sliced product takes this shape
bool oz_takes(i64 M, i64 N, i64 K, int count);

// The batch's product, count <= kOzMaxProblems; shift (M / 2 complex) null:
// plain store, else C(x, n) = shift(x) fac(x, n) (A B)(x, n) on complex rows.
// Returns CHM_ERR_WS, with nothing launched, if ws is too small.
int oz_gemm_launch(const OzProblem *p, int count, int M, int N, int K, const double2 *shift,
                   void *ws, i64 ws_bytes, cudaStream_t st);

// nonzero if a product CTA gave up on a bounded wait (then reset)
int oz_status();

}  // namespace chm
