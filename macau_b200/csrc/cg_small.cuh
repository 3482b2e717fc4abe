// Shared pieces of the block-CG solvers (cg_kernels.cu, cg_tiles.cu): the small-matrix workspace and
// the general K x K solve by one CTA.
#pragma once
#include "common.cuh"

namespace mg {

// Small layout (doubles): RtR[64*64] | RtR2[64*64] | M[64*64] | A[64*64] | Psi[64*64] | norms[64]
//                         | inorms[64] | flags[4]
constexpr int kSq = 64 * 64;
struct SmallView {
  double *RtR, *RtR2, *M, *A, *Psi, *norms, *inorms, *flags;
  __host__ __device__ explicit SmallView(double* s)
      : RtR(s), RtR2(s + kSq), M(s + 2 * kSq), A(s + 3 * kSq), Psi(s + 4 * kSq),
        norms(s + 5 * kSq), inorms(s + 5 * kSq + 64), flags(s + 5 * kSq + 128) {}
};

// Left-looking lower Cholesky of the n x n matrix A (leading dimension ld) by one CTA, column by
// column; thread i computes L(i, j).  On a non-positive pivot it stops and leaves column j and
// the columns after it as they were, like the unchecked Eigen llt() the reference uses
// (linop.h:287, 313): the caller's solves then read that partial factor.  Returns false then.
static __device__ bool cta_chol_n(double* A, int n, int ld) {
  __syncthreads();
  for (int j = 0; j < n; j++) {
    double d = A[j + j * ld];
    for (int p = 0; p < j; p++) d -= A[j + p * ld] * A[j + p * ld];
    if (!(d > 0.0)) {
      __syncthreads();
      return false;
    }
    const double ljj = sqrt(d);
    for (int i = j + 1 + threadIdx.x; i < n; i += blockDim.x) {
      double s = A[i + j * ld];
      for (int p = 0; p < j; p++) s -= A[i + p * ld] * A[j + p * ld];
      A[i + j * ld] = s / ljj;
    }
    __syncthreads();
    if (threadIdx.x == 0) A[j + j * ld] = ljj;
    __syncthreads();
  }
  return true;
}

// Out(c, i) = (M^{-T} M^{-1} Rhs)(i, c) for the n columns of Rhs, M the lower Cholesky factor
// in v.M (leading dimension 64): thread c solves column c, forward then backward substitution in
// the order of the reference's llt().solve.  The general path (n > 32, or a failed pivot).
static __device__ void cta_chol_solve_cols(const double* M, const double* Rhs, int n, double* Out) {
  for (int c = threadIdx.x; c < n; c += blockDim.x) {
    double y[64];
    for (int i = 0; i < n; i++) y[i] = Rhs[i + c * 64];
    for (int i = 0; i < n; i++) {
      double s = y[i];
      for (int p = 0; p < i; p++) s -= M[i + p * 64] * y[p];
      y[i] = s / M[i + i * 64];
    }
    for (int i = n - 1; i >= 0; i--) {
      double s = y[i];
      for (int p = i + 1; p < n; p++) s -= M[p + i * 64] * y[p];
      y[i] = s / M[i + i * 64];
    }
    for (int i = 0; i < n; i++) Out[c + i * 64] = y[i];
  }
}

}  // namespace mg
