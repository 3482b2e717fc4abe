// Hyperprior in a fixed order of summation: statistics and Normal-Wishart draw of chains with a
// block-CG link matrix (K <= 64), and of the batched problems (K <= 32).
//
// Why these do not use the kernels of hyper_kernels.cu and hyper_wide.cu:
//   * A link solve stops at a tolerance (1e-6 by default), and its result within that tolerance
//     depends on the last bit of its right-hand side: latents that differ by one unit in the last
//     place give link matrices that differ by 1e-7 to 2e-6 (1,203 to 5,003 rows, 517 to 4,099
//     features, 7 to 64 components), in FP64 too, and mixed latents that differ by 2e-4 a sweep
//     later.  So a chain with side information repeats a recorded one only if everything that
//     reaches the solve is summed in the order it was recorded with: the rows (launch_sample),
//     these, and the SpMMs and solves of cg_kernels.cu.
//   * A batch runs many mixed-precision chains for many sweeps, each rounding Lambda to FP32 and its
//     latents to BF16: of 64 problems over 40 sweeps about one met a Lambda whose last FP64 bit
//     decided its FP32 rounding, and its latents were then 0.04 apart.
//   * A single mixed chain without a link takes those kernels all the same: the same bit costs it its
//     recorded course about once in 6,000 sweeps (6 of 28 chains at K = 8 to 64 within 1,500 sweeps),
//     not in every call.  FP64 chains without a link differ by rounding alone.
//   What bounds them: beside a solve nothing that matters (the draw takes 36 us on one SM at K <= 32);
// in a batch the longest problem's statistics.
#include "common.cuh"
#include "kernels.h"
#include "mma_tiles.cuh"
#include "rng.cuh"
#include "warp_finish.cuh"

namespace mg {
namespace {

constexpr int kStatThreads = 160;  // four warps of products, one of sums

// Column sums of rows r0 .. r1 - 1 of (U - Uhat), row after row, column `lane`; two batches of loads in
// flight.
template <typename T, bool HAT>
__device__ __forceinline__ double ordered_sums(const T* __restrict__ U,
                                               const double* __restrict__ Uhat, long long r0,
                                               long long r1, int K, int stride, int uhat_stride,
                                               int lane) {
  constexpr int B = HAT || sizeof(T) == 8 ? 16 : 32;
  T u[2][B];
  double h[HAT ? 2 : 1][B];
  auto load = [&](int stage, long long row) {
#pragma unroll
    for (int i = 0; i < B; i++) {
      const bool in = row + i < r1 && lane < K;
      u[stage][i] = in ? U[(row + i) * stride + lane] : (T)0;
      if constexpr (HAT) h[stage][i] = in ? Uhat[(row + i) * uhat_stride + lane] : 0.0;
    }
  };
  double s = 0.0;
  load(0, r0);
  for (long long r = r0; r < r1; r += 2 * B) {
#pragma unroll
    for (int v = 0; v < 2; v++) {
      load(v ^ 1, r + (v + 1) * B);
#pragma unroll
      for (int i = 0; i < B; i++) {
        double x = (double)u[v][i];
        if constexpr (HAT) x -= h[v][i];
        s += x;
      }
    }
  }
  return s;
}

// One block's statistics over rows r0 .. r1 - 1 of (U - Uhat) into out[0 .. K + K*K).  The product sum
// of a pair of columns is four sums over every fourth row, added in order; warp w < 4 forms the
// w-th of them for all lower-triangle tiles by m8n8k4.f64, which adds its four products one by
// one in order (bit for bit a chain of fma).
//   What bounds it: 16 cycles of a sub-partition per instruction, 10 of them per 16 rows and warp
//   at K = 32, on one SM per block.  (4 x 4 tiles of fma over rows staged in shared memory: 126 us on
//   average for 64 problems of up to 4,000 rows.)
template <typename T>
__device__ __forceinline__ void ordered_stats(const T* __restrict__ U,
                                             const double* __restrict__ Uhat, long long r0,
                                             long long r1, int K, int stride, int uhat_stride,
                                             double* __restrict__ out) {
  constexpr int R = 4;  // steps of four rows in flight
  __shared__ __align__(16) double red[3][10 * 64];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int nb = (K + 7) / 8;
  double acc[10][2] = {};
  if (warp == 4) {
    const double s =
        Uhat ? ordered_sums<T, true>(U, Uhat, r0, r1, K, stride, uhat_stride, lane)
             : ordered_sums<T, false>(U, Uhat, r0, r1, K, stride, uhat_stride, lane);
    if (lane < K) out[lane] = s;
  } else {
    double f[R][4];
    auto load = [&](int stage, long long row) {
#pragma unroll
      for (int b = 0; b < 4; b++) {
        const int k = 8 * b + g;
        const bool in = row < r1 && k < K;
        f[stage][b] = in ? (double)U[row * stride + k] : 0.0;
        if (Uhat && in) f[stage][b] -= Uhat[row * uhat_stride + k];
      }
    };
    const long long first = r0 + warp + 4 * t;
#pragma unroll
    for (int v = 0; v < R - 1; v++) load(v, first + 16 * v);
    for (long long r = r0; r < r1; r += 16 * R) {
#pragma unroll
      for (int v = 0; v < R; v++) {
        load((v + R - 1) % R, r - r0 + first + 16 * (v + R - 1));
        int q = 0;
#pragma unroll
        for (int bi = 0; bi < 4; bi++)
#pragma unroll
          for (int bj = 0; bj <= bi; bj++) {
            if (bi < nb) mma_f64(acc[q][0], acc[q][1], f[v][bi], f[v][bj]);
            q++;
          }
      }
    }
    if (warp > 0)
#pragma unroll
      for (int q = 0; q < 10; q++)
        *reinterpret_cast<double2*>(&red[warp - 1][q * 64 + g * 8 + 2 * t]) =
            make_double2(acc[q][0], acc[q][1]);
  }
  __syncthreads();
  if (warp > 0) return;
  int q = 0;
#pragma unroll
  for (int bi = 0; bi < 4; bi++)
#pragma unroll
    for (int bj = 0; bj <= bi; bj++) {
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int at = q * 64 + g * 8 + 2 * t + e;
        const double v = ((acc[q][e] + red[0][at]) + red[1][at]) + red[2][at];
        const int i = 8 * bi + g, j = 8 * bj + 2 * t + e;
        if (i < K && j < K) {
          out[K + i + j * K] = v;
          out[K + j + i * K] = v;
        }
      }
      q++;
    }
}

template <typename T>
__global__ void __launch_bounds__(kStatThreads)
    k_link_stats(const T* __restrict__ U, const double* __restrict__ Uhat, long long N, int K,
                 int stride, int uhat_stride, long long rows_per_block,
                 double* __restrict__ partials) {
  const long long r0 = (long long)blockIdx.x * rows_per_block;
  ordered_stats(U, Uhat, r0, min(N, r0 + rows_per_block), K, stride, uhat_stride,
               partials + (size_t)blockIdx.x * (K + K * K));
}

// K > 32: k_stats_wide's products are chains of fma over the rows already (one warp takes a tile
// through all of a block's rows); its column sums, four partial sums each, are replaced by these.
// One warp per 32 columns.
template <typename T>
__global__ void __launch_bounds__(64)
    k_link_sums(const T* __restrict__ U, const double* __restrict__ Uhat, long long N, int K,
                int stride, int uhat_stride, long long rows_per_block,
                double* __restrict__ partials) {
  const long long r0 = (long long)blockIdx.x * rows_per_block, r1 = min(N, r0 + rows_per_block);
  const int c0 = threadIdx.x & ~31, lane = threadIdx.x & 31;
  const double s =
      Uhat ? ordered_sums<T, true>(U + c0, Uhat + c0, r0, r1, K - c0, stride, uhat_stride, lane)
           : ordered_sums<T, false>(U + c0, nullptr, r0, r1, K - c0, stride, uhat_stride, lane);
  if (c0 + lane < K) partials[(size_t)blockIdx.x * (K + K * K) + c0 + lane] = s;
}

// Problem p owns rows row0[p] .. row0[p + 1] - 1 of U (stride 32), K = Kp[p]; one block per problem.
__global__ void __launch_bounds__(kStatThreads)
    k_stats_batch(const float* __restrict__ U, const int* __restrict__ row0,
                  const int* __restrict__ Kp, double* __restrict__ partials) {
  const int p = blockIdx.x;
  ordered_stats<float>(U, nullptr, row0[p], row0[p + 1], Kp[p], 32, 0,
                      partials + (size_t)p * (32 + 32 * 32));
}

// CondNormalWishart -> NormalWishart -> MvNormal_prec (mvnormal.cpp:169-184, 217-287, 314-336)
// for K <= 32 in one CTA of 256 threads, matrices in shared memory (row-major, ld 33), the
// draws of k_nw.  Two identities replace two of the reference's three Cholesky
// factorisations (results agree to FP64 rounding):
//   * chol(X^{-1}) = J M^{-T} J with M = chol(J X J), J the index reversal: one Cholesky of the
//     reversed X (warp 0's registers, warp_factor) and one triangular inverse Y = M^{-1}
//     (lane c solves M y = e_c), L(i, j) = Y(K-1-j, K-1-i);
//   * Lambda = L c^T c L^T = B B^T with B = L c^T lower triangular with positive diagonal, so
//     chol(kappa_c Lambda) = sqrt(kappa_c) B and mu = mu_c + B^{-T} z / sqrt(kappa_c).
// The Bartlett factor c and z are drawn by warps 1-7 while warp 0 factorises.
constexpr int kNwLd = 33;
constexpr int kNwLc = 36;

// mu0 == null stands for zeros, T0 == null for the identity, bb == null for no link matrix.
__device__ __forceinline__ void nw32_run(const double* __restrict__ stats, long long N, int K,
                                         const double* __restrict__ mu0, double kappa,
                                         const double* __restrict__ T0, int nu,
                                         const double* __restrict__ bb,
                                         const double* __restrict__ lambda_beta, Ctl* ctl,
                                         unsigned long long seed, int mode,
                                         double* __restrict__ mu_out,
                                         double* __restrict__ Lambda_out) {
  __shared__ double A[32 * kNwLd], Bm[32 * kNwLd], C[32 * kNwLd], D[32 * kNwLd];
  __shared__ __align__(16) double Lc[32 * kNwLc];
  __shared__ double NU[32], muc[32], m0[32], rl[32], zs[32];
  __shared__ int flag;
  const int t = threadIdx.x, lane = t & 31;
  const int KK = K * K;
  const uint32_t sweep = ctl->sweep;
  // 1. NU = sum x, A = S = sum x x^T; Bm = T = WI + lambda_beta beta beta^T (latentprior.cpp:258-260)
  const double lb = bb ? *lambda_beta : 0.0;
  for (int e = t; e < K; e += 256) NU[e] = stats[e];
  for (int e = t; e < KK; e += 256) {
    A[(e % K) * kNwLd + e / K] = stats[K + e];
    const double w0 = T0 ? T0[e] : (e % K == e / K ? 1.0 : 0.0);
    Bm[(e % K) * kNwLd + e / K] = bb ? w0 + lb * bb[K + e] : w0;
  }
  if (t < K) m0[t] = mu0 ? mu0[t] : 0.0;
  __syncthreads();
  const double kappa_c = kappa + (double)N;
  const int nu_c = nu + (int)N;
  if (t < K) muc[t] = (kappa * m0[t] + NU[t]) / kappa_c;
  __syncthreads();
  // 2. X = T + NS + kappa mu0 mu0^T - kappa_c mu_c mu_c^T   (into A)
  for (int e = t; e < KK; e += blockDim.x) {
    const int i = e % K, j = e / K;
    A[i * kNwLd + j] =
        Bm[i * kNwLd + j] + A[i * kNwLd + j] + kappa * m0[i] * m0[j] - kappa_c * muc[i] * muc[j];
  }
  __syncthreads();
  if (t < 32) {
    // 3a. M = chol(J X J), M^T rows into Lc
    double a[32], d0 = 1.0, rinv = 1.0;
#pragma unroll
    for (int j = 0; j < 32; j++) {
      a[j] = (lane < K && j < K) ? A[(K - 1 - lane) * kNwLd + (K - 1 - j)] : (lane == j ? 1.0 : 0.0);
      if (j == lane) d0 = a[j];
    }
    const bool ok = warp_factor<double, 32>(a, rinv, lane, 0.0, d0, Lc, kNwLc);
    if (lane == 0) flag = ok ? 1 : 0;
    // 3b. Y = M^{-1}: lane c solves M y = e_c; Y(i, c) into D
    if (ok) {
      rl[lane] = rinv;
      __syncwarp();
      double y[32];
#pragma unroll
      for (int i = 0; i < 32; i++) {
        double s = (lane == i) ? 1.0 : 0.0;
#pragma unroll
        for (int q = 0; q < i; q++) s = fma(-Lc[q * kNwLc + i], y[q], s);
        y[i] = s * rl[i];
      }
#pragma unroll
      for (int i = 0; i < 32; i++) D[i * kNwLd + lane] = y[i];
    }
  } else {
    // 3c. Bartlett factor c (upper) into C: c_ii = sqrt(2 Gamma((nu_c - i)/2)), c_ij ~ N(0,1);
    //     z for the mean draw
    for (int e = t - 32; e < KK; e += blockDim.x - 32) {
      const int i = e % K, j = e / K;
      double v = 0.0;
      if (i == j)
        v = sqrt(2.0 * gamma_draw(seed, sweep, stream_id(kWishartDiag, mode), (uint32_t)i,
                                  0.5 * (double)(nu_c - i)));
      else if (j > i)
        v = normal_draw(seed, sweep, stream_id(kWishartOff, mode), (uint32_t)i,
                        (uint32_t)(j - i - 1));
      C[i * kNwLd + j] = v;
    }
    if (t - 32 < K) zs[t - 32] = normal_draw(seed, sweep, stream_id(kMuDraw, mode), 0u, (uint32_t)(t - 32));
  }
  __syncthreads();
  if (!flag) {
    if (t == 0) atomicOr(&ctl->status, kStatHyperFail);
    return;
  }
  // 4. L = chol(T_c) = chol(X^{-1}) into A: L(i, j) = Y(K-1-j, K-1-i), j <= i
  for (int e = t; e < KK; e += blockDim.x) {
    const int i = e % K, j = e / K;
    A[i * kNwLd + j] = (j <= i) ? D[(K - 1 - j) * kNwLd + (K - 1 - i)] : 0.0;
  }
  __syncthreads();
  // 5. B = L c^T (lower triangular): B(i, j) = sum_{q=j..i} L(i, q) c(j, q)
  for (int e = t; e < KK; e += blockDim.x) {
    const int i = e % K, j = e / K;
    double s = 0.0;
    for (int q = j; q <= i; q++) s += A[i * kNwLd + q] * C[j * kNwLd + q];
    Bm[i * kNwLd + j] = (j <= i) ? s : 0.0;
  }
  __syncthreads();
  // 6. Lambda = B B^T
  for (int e = t; e < KK; e += blockDim.x) {
    const int i = e % K, j = e / K;
    const int m = min(i, j);
    double s = 0.0;
    for (int q = 0; q <= m; q++) s += Bm[i * kNwLd + q] * Bm[j * kNwLd + q];
    Lambda_out[e] = s;
  }
  // 7. mu = mu_c + B^{-T} z / sqrt(kappa_c)
  if (t < 32) {
    double x = lane < K ? zs[lane] / sqrt(kappa_c) : 0.0;
    for (int j = K - 1; j >= 0; j--) {
      if (lane == j) x = x / Bm[j * kNwLd + j];
      const double xj = __shfl_sync(0xffffffffu, x, j);
      if (lane < j) x = fma(-Bm[j * kNwLd + lane], xj, x);
    }
    if (lane < K) mu_out[lane] = x + muc[lane];
  }
}
__global__ void __launch_bounds__(256)
    k_link_wishart(const double* __restrict__ stats, long long N, int K,
                   const double* __restrict__ mu0, double kappa, const double* __restrict__ T0,
                   int nu, const double* __restrict__ bb, const double* __restrict__ lambda_beta,
                   Ctl* ctl, unsigned long long seed, int mode, double* __restrict__ mu_out,
                   double* __restrict__ Lambda_out) {
  nw32_run(stats, N, K, mu0, kappa, T0, nu, bb, lambda_beta, ctl, seed, mode, mu_out, Lambda_out);
}

// ---- the draw for 32 < K <= 64 ----
// Matrices in shared memory, column-major with an odd leading dimension, so that the threads of a warp
// touch different banks along a row as along a column.
__host__ __device__ __forceinline__ int odd_ld(int K) { return K | 1; }

// Left-looking lower Cholesky of the K x K matrix A by the block, thread i forming L(i, j); the strict upper triangle is zeroed.  False on a pivot that is not
// positive (the same value in every thread).
__device__ bool block_chol(double* A, int K) {
  const int ld = odd_ld(K);
  __syncthreads();
  for (int j = 0; j < K; j++) {
    double d = A[j + j * ld];
    for (int p = 0; p < j; p++) d = fma(-A[j + p * ld], A[j + p * ld], d);
    if (!(d > 0.0)) {
      __syncthreads();
      return false;
    }
    const double ljj = sqrt(d);
    for (int i = j + 1 + threadIdx.x; i < K; i += blockDim.x) {
      double s = A[i + j * ld];
      for (int p = 0; p < j; p++) s = fma(-A[i + p * ld], A[j + p * ld], s);
      A[i + j * ld] = s / ljj;
    }
    __syncthreads();
    if (threadIdx.x == 0) A[j + j * ld] = ljj;
    __syncthreads();
  }
  for (int q = threadIdx.x; q < K * K; q += blockDim.x)
    if (q % K < q / K) A[q % K + q / K * ld] = 0.0;
  __syncthreads();
  return true;
}

// CondNormalWishart -> NormalWishart -> Wishart -> MvNormal_prec (mvnormal.cpp:169-184, 217-287,
// 314-336) step by step, each matrix element one chain of fma over its index: T_c by the factor of X
// and two substitutions per column, its factor L, Lambda = L (c^T c) L^T, the mean through the
// factor of kappa_c Lambda.  The matrices are in shared memory.
//   What bounds it: the substitutions, a thread per column: 364 us at K = 64 (0.81 ms with the matrices in
// global memory), beside a solve of 3 ms and more.
__global__ void __launch_bounds__(256)
    k_link_wishart_wide(const double* __restrict__ stats, long long N, int K,
                        const double* __restrict__ mu0, double kappa, const double* __restrict__ T0,
                        int nu, const double* __restrict__ bb,
                        const double* __restrict__ lambda_beta, Ctl* ctl, unsigned long long seed,
                        int mode, double* __restrict__ mu_out, double* __restrict__ Lambda_out) {
  extern __shared__ __align__(16) double wsm[];
  __shared__ double muc[64], z[64];
  const int KK = K * K, ld = odd_ld(K);
  const uint32_t sweep = ctl->sweep;
  double *X = wsm, *Tc = X + K * ld, *c = Tc + K * ld, *W = c + K * ld;
  const double lb = bb ? *lambda_beta : 0.0;
  const double kappa_c = kappa + (double)N;
  const int nu_c = nu + (int)N;
  for (int i = threadIdx.x; i < K; i += blockDim.x) muc[i] = fma(kappa, mu0[i], stats[i]) / kappa_c;
  __syncthreads();
  for (int e = threadIdx.x; e < KK; e += blockDim.x) {
    const int i = e % K, j = e / K;
    const double T = bb ? fma(lb, bb[K + e], T0[e]) : T0[e];  // latentprior.cpp:258-260
    X[i + j * ld] = fma(-(kappa_c * muc[i]), muc[j], fma(kappa * mu0[i], mu0[j], T + stats[K + e]));
  }
  bool ok = block_chol(X, K);
  if (ok) {
    for (int q = threadIdx.x; q < K; q += blockDim.x) {  // column q of X^{-1}
      double* x = Tc + q * ld;
      for (int i = 0; i < K; i++) {
        double s = i == q ? 1.0 : 0.0;
        for (int p = 0; p < i; p++) s = fma(-X[i + p * ld], x[p], s);
        x[i] = s / X[i + i * ld];
      }
      for (int i = K - 1; i >= 0; i--) {
        double s = x[i];
        for (int p = i + 1; p < K; p++) s = fma(-X[p + i * ld], x[p], s);
        x[i] = s / X[i + i * ld];
      }
    }
    ok = block_chol(Tc, K);
  }
  if (ok) {
    // Bartlett factor: c_ii = sqrt(2 Gamma((nu_c - i) / 2)), c_ij ~ N(0, 1) for j > i
    for (int e = threadIdx.x; e < KK; e += blockDim.x) {
      const int i = e % K, j = e / K;
      double v = 0.0;
      if (i == j)
        v = sqrt(2.0 * gamma_draw(seed, sweep, stream_id(kWishartDiag, mode), (uint32_t)i,
                                  0.5 * (double)(nu_c - i)));
      else if (j > i)
        v = normal_draw(seed, sweep, stream_id(kWishartOff, mode), (uint32_t)i,
                        (uint32_t)(j - i - 1));
      c[i + j * ld] = v;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < KK; e += blockDim.x) {  // W = c^T c
      const int i = e % K, j = e / K;
      double s = 0.0;
      for (int p = 0; p < K; p++) s = fma(c[p + i * ld], c[p + j * ld], s);
      W[i + j * ld] = s;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < KK; e += blockDim.x) {  // X = L W
      const int i = e % K, j = e / K;
      double s = 0.0;
      for (int p = 0; p < K; p++) s = fma(Tc[i + p * ld], W[p + j * ld], s);
      X[i + j * ld] = s;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < KK; e += blockDim.x) {  // Lambda = X L^T
      const int i = e % K, j = e / K;
      double s = 0.0;
      for (int p = 0; p < K; p++) s = fma(X[i + p * ld], Tc[j + p * ld], s);
      Lambda_out[e] = s;
      c[i + j * ld] = s * kappa_c;
    }
    ok = block_chol(c, K);
  }
  if (!ok) {
    if (threadIdx.x == 0) atomicOr(&ctl->status, kStatHyperFail);
    return;
  }
  // mu = mu_c + chol(kappa_c Lambda)^{-T} z
  for (int i = threadIdx.x; i < K; i += blockDim.x)
    z[i] = normal_draw(seed, sweep, stream_id(kMuDraw, mode), 0u, (uint32_t)i);
  __syncthreads();
  if (threadIdx.x == 0)
    for (int i = K - 1; i >= 0; i--) {
      double s = z[i];
      for (int p = i + 1; p < K; p++) s = fma(-c[p + i * ld], z[p], s);
      z[i] = s / c[i + i * ld];
    }
  __syncthreads();
  for (int i = threadIdx.x; i < K; i += blockDim.x) mu_out[i] = z[i] + muc[i];
}

// BPMFPrior::update_prior per problem with mu0 = 0, b0 = 2, W0 = I, df = K_p
// (latentprior.cpp:79-99), keyed with the problem's seed; then the finish's operands: the FP32
// Lambda (32 x 32, zero beyond K) and Lambda mu (FP64, summed in column order).
__global__ void __launch_bounds__(256)
    k_nw_batch(const double* __restrict__ partials, const int* __restrict__ row0,
               const int* __restrict__ Kp, const unsigned long long* __restrict__ seed, Ctl* ctl,
               int mode, double* __restrict__ mu, double* __restrict__ Lambda,
               float* __restrict__ LamF, double* __restrict__ lmu) {
  const int p = blockIdx.x, K = Kp[p];
  double* L = Lambda + (size_t)p * 1024;
  double* m = mu + (size_t)p * 32;
  nw32_run(partials + (size_t)p * (32 + 32 * 32), row0[p + 1] - row0[p], K, nullptr, 2.0, nullptr, K,
           nullptr, nullptr, ctl, seed[p], mode, m, L);
  __syncthreads();
  for (int e = threadIdx.x; e < 1024; e += blockDim.x) {
    const int i = e >> 5, j = e & 31;
    LamF[(size_t)p * 1024 + e] = (i < K && j < K) ? (float)L[i + j * K] : 0.f;
  }
  if (threadIdx.x < 32) {
    double acc = 0.0;
    if ((int)threadIdx.x < K)
      for (int j = 0; j < K; j++) acc += L[threadIdx.x + j * K] * m[j];
    lmu[(size_t)p * 32 + threadIdx.x] = acc;
  }
}

}  // namespace

void launch_link_stats(const void* U, bool f32, const double* Uhat, long long N, int K, int stride,
                       int uhat_stride, double* partials, int nblocks, cudaStream_t s) {
  const long long rpb = (N + nblocks - 1) / nblocks;
  if (K > 32) {
    launch_stats_wide(U, f32, Uhat, N, K, stride, uhat_stride, partials, nblocks, s);
    if (f32)
      k_link_sums<float><<<nblocks, 64, 0, s>>>((const float*)U, Uhat, N, K, stride, uhat_stride,
                                                rpb, partials);
    else
      k_link_sums<double><<<nblocks, 64, 0, s>>>((const double*)U, Uhat, N, K, stride, uhat_stride,
                                                 rpb, partials);
    MG_CUDA(cudaGetLastError());
    return;
  }
  if (f32)
    k_link_stats<float><<<nblocks, kStatThreads, 0, s>>>((const float*)U, Uhat, N, K, stride,
                                                         uhat_stride, rpb, partials);
  else
    k_link_stats<double><<<nblocks, kStatThreads, 0, s>>>((const double*)U, Uhat, N, K, stride,
                                                          uhat_stride, rpb, partials);
  MG_CUDA(cudaGetLastError());
}

void launch_link_wishart(const double* stats, long long N, int K, const double* mu0, double kappa,
                         const double* T0, int nu, const double* bb, const double* lambda_beta,
                         Ctl* ctl, unsigned long long seed, int mode, double* mu_out,
                         double* Lambda_out, cudaStream_t s) {
  if (K > 32) {
    static bool configured[64] = {false};
    int dev = 0;
    MG_CUDA(cudaGetDevice(&dev));
    if (!configured[dev & 63]) {
      MG_CUDA(cudaFuncSetAttribute(k_link_wishart_wide, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)(4 * 64 * 65 * sizeof(double))));
      configured[dev & 63] = true;
    }
    k_link_wishart_wide<<<1, 256, 4 * sizeof(double) * K * odd_ld(K), s>>>(
        stats, N, K, mu0, kappa, T0, nu, bb, lambda_beta, ctl, seed, mode, mu_out, Lambda_out);
    MG_CUDA(cudaGetLastError());
    return;
  }
  k_link_wishart<<<1, 256, 0, s>>>(stats, N, K, mu0, kappa, T0, nu, bb, lambda_beta, ctl, seed, mode,
                                   mu_out, Lambda_out);
  MG_CUDA(cudaGetLastError());
}

void launch_prior_batch(const float* U, const int* row0, const int* Kp,
                        const unsigned long long* seed, int P, double* partials, Ctl* ctl, int mode,
                        double* mu, double* Lambda, float* LamF, double* lmu, cudaStream_t s) {
  k_stats_batch<<<P, kStatThreads, 0, s>>>(U, row0, Kp, partials);
  MG_CUDA(cudaGetLastError());
  k_nw_batch<<<P, 256, 0, s>>>(partials, row0, Kp, seed, ctl, mode, mu, Lambda, LamF, lmu);
  MG_CUDA(cudaGetLastError());
}

}  // namespace mg
