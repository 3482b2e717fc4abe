// Normal-Wishart hyperprior update on the FP64 matrix instruction m8n8k4.f64.
//
//   k_nw          one block per update, every K <= 128: CondNormalWishart -> NormalWishart -> Wishart
//                 -> MvNormal_prec (mvnormal.cpp:169-184, 217-287, 314-336), all matrices in shared
//                 memory as 8 x 8 tiles of their lower triangles, keyed draws beside the factor.
//   k_stats_wide  32 < K <= 128: per-block partial sums of x and x x^T over the rows of a latent
//                 matrix (x = U, or U - Uhat): the lower-triangle tiles spread over the block's
//                 warps as in the row sampler, rows read straight into fragments.
//
// What bounds k_nw: the chain of the panel factor, about 1,500 to 2,500 cycles per 8 columns; the
// triangular inverse and the three products that follow are matrix instructions on 16 warps.  With
// the matrices in global memory and one thread to a dot product (or a whole substitution) a draw
// took 4.28 ms at K = 128 and 0.81 ms at K = 64; with a matrix row per lane of one warp 25 us at
// K = 32 (450 cycles a column, and 1,024 separate normal draws).
#include "common.cuh"
#include "kernels.h"
#include "rng.cuh"
#include "wide_tiles.cuh"

namespace mg {
namespace {

template <int KP>
struct StatW {
  static constexpr int W = KP == 64 ? 4 : 8, T = 32 * W;
  static constexpr int RB = KP == 64 ? 2 : 4, ND = KP == 64 ? 1 : 2;
};

// What a launch updates: one mode, or both (block rows of mode 0, then of mode 1).
struct StatsArgs {
  const void* U[2];
  const double* Uhat;  // one mode only
  long long N[2], rows_per_block[2];
  int nblocks[2];
  double* partials[2];
};

// A warp's tiles over rows r0 .. r1 - 1.  DIAG: also the column sums of its blocks.
template <typename V, int KP, bool DIAG, bool HAT>
__device__ __forceinline__ void stats_warp(const V* __restrict__ U, const double* __restrict__ Uhat,
                                           long long r0, long long r1, int K, int stride,
                                           int uhat_stride, int br, int bc,
                                           double* __restrict__ out) {
  using C = StatW<KP>;
  constexpr int NR = DIAG ? 4 * C::ND : C::RB, NC = DIAG ? 0 : 4;
  constexpr int NT = DIAG ? 10 * C::ND : 4 * C::RB;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  constexpr int R = 4;  // steps of four rows in flight
  double acc[NT][2], racc[NR], f[R][NR + NC];
#pragma unroll
  for (int q = 0; q < NT; q++) acc[q][0] = acc[q][1] = 0.0;
#pragma unroll
  for (int b = 0; b < NR; b++) racc[b] = 0.0;
  // this lane's components of each block; the loads of a step are independent and unconditional
  // but for the bounds
  int col[NR + NC];
#pragma unroll
  for (int b = 0; b < NR + NC; b++) col[b] = 8 * (b < NR ? br + b : bc + b - NR) + g;
  auto load = [&](int stage, long long row) {
    const V* u = U + row * stride;
    const double* h = HAT ? Uhat + row * uhat_stride : nullptr;
#pragma unroll
    for (int b = 0; b < NR + NC; b++) {
      const bool ok = row < r1 && col[b] < K;
      double x = ok ? (double)__ldg(u + col[b]) : 0.0;
      if constexpr (HAT) x -= ok ? __ldg(h + col[b]) : 0.0;
      f[stage][b] = x;
    }
  };
#pragma unroll
  for (int u = 0; u < R - 1; u++) load(u, r0 + 4 * u + t);
  for (long long r = r0; r < r1; r += 4 * R) {
#pragma unroll
    for (int u = 0; u < R; u++) {
      load((u + R - 1) % R, r + 4 * (u + R - 1) + t);
      int q = 0;
      if constexpr (DIAG) {
#pragma unroll
        for (int s = 0; s < C::ND; s++)
#pragma unroll
          for (int a = 0; a < 4; a++) {
            racc[4 * s + a] += f[u][4 * s + a];
#pragma unroll
            for (int b = 0; b <= a; b++) {
              mma_f64(acc[q][0], acc[q][1], f[u][4 * s + a], f[u][4 * s + b]);
              q++;
            }
          }
      } else {
#pragma unroll
        for (int a = 0; a < NR; a++)
#pragma unroll
          for (int b = 0; b < NC; b++) {
            mma_f64(acc[q][0], acc[q][1], f[u][a], f[u][NR + b]);
            q++;
          }
      }
    }
  }
  auto put = [&](int bi, int bj, const double (&v)[2]) {
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int i = 8 * bi + g, j = 8 * bj + 2 * t + e;
      if (i < K && j < K) {
        out[K + i + (size_t)j * K] = v[e];
        if (bi != bj) out[K + j + (size_t)i * K] = v[e];
      }
    }
  };
  int q = 0;
  if constexpr (DIAG) {
#pragma unroll
    for (int b = 0; b < NR; b++) {
      double s = racc[b];
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      if (t == 0 && 8 * (br + b) + g < K) out[8 * (br + b) + g] = s;
    }
#pragma unroll
    for (int s = 0; s < C::ND; s++)
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b <= a; b++) put(br + 4 * s + a, br + 4 * s + b, acc[q++]);
  } else {
#pragma unroll
    for (int a = 0; a < NR; a++)
#pragma unroll
      for (int b = 0; b < NC; b++) put(br + a, bc + b, acc[q++]);
  }
}

template <typename V, int KP, bool HAT>
__global__ void __launch_bounds__(StatW<KP>::T)
    k_stats_wide(const StatsArgs p, int K, int stride, int uhat_stride) {
  const int m = (int)blockIdx.x < p.nblocks[0] ? 0 : 1;
  const int b = (int)blockIdx.x - (m ? p.nblocks[0] : 0);
  const long long r0 = b * p.rows_per_block[m], r1 = min(p.N[m], r0 + p.rows_per_block[m]);
  const V* U = static_cast<const V*>(p.U[m]);
  double* out = p.partials[m] + (size_t)b * (K + (size_t)K * K);
  const Part64 part = part_of<KP>(threadIdx.x >> 5);
  if (part.diag)
    stats_warp<V, KP, true, HAT>(U, p.Uhat, r0, r1, K, stride, uhat_stride, part.r0, 0, out);
  else
    stats_warp<V, KP, false, HAT>(U, p.Uhat, r0, r1, K, stride, uhat_stride, part.r0, part.c0, out);
}

template <typename V>
void stats_launch(const StatsArgs& a, int K, int stride, int uhat_stride, cudaStream_t s) {
  const int nb = a.nblocks[0] + a.nblocks[1];
  if (K > 64)  // side information needs K <= 64
    k_stats_wide<V, 128, false><<<nb, StatW<128>::T, 0, s>>>(a, K, stride, uhat_stride);
  else if (a.Uhat)
    k_stats_wide<V, 64, true><<<nb, StatW<64>::T, 0, s>>>(a, K, stride, uhat_stride);
  else
    k_stats_wide<V, 64, false><<<nb, StatW<64>::T, 0, s>>>(a, K, stride, uhat_stride);
  MG_CUDA(cudaGetLastError());
}

// ---- the Normal-Wishart draw ----
struct NwArgs {
  const double* stats;  // `nparts` records of sums (K), then x x^T (K x K), added in order
  int nparts;
  const double* mu0;    // null: zero
  const double* T0;     // null: the identity
  double kappa;
  long long N;
  int nu, mode;
  double *mu, *Lambda;
};
struct NwPair {
  NwArgs m[2];
};

constexpr int kNwThreads = 512, kNwHalf = 256;  // warps 0-7: factor, solve; warps 8-15: draws, Lambda

template <int KP>
struct NwW {
  static constexpr int NB = KP / 8, TRI = NB * (NB + 1) / 2;
  // M, then B | Y = M^-1 | the Bartlett factor's transpose | inverses of the diagonal tiles | mu_c,
  // y, x, zeros, z | flag | tile table
  static constexpr size_t kDoubles = (3 * (size_t)TRI + NB) * 64 + 5 * KP + 2 + (TRI + 7) / 8;
};

// Draws of the Bartlett factor c (upper triangular: c_ii = sqrt(2 Gamma((nu_c - i) / 2)), c_ij ~
// N(0, 1) for j > i), stored as its transpose's lower-triangle tiles, the identity beyond K, and
// the mean draw's z, by threads tid < nt.
__device__ __forceinline__ void bartlett(double* Ct, double* z, int K, int n, int nu_c,
                                         unsigned long long seed, uint32_t sweep, uint32_t mode,
                                         int tid, int nt) {
  // the three kinds of draws start at different threads, so that at small K they are different
  // warps' work: gammas from the first, z from the middle, pairs from the last
  for (int i = tid; i < K; i += nt)
    Ct[elem_at(i, i)] = sqrt(2.0 * gamma_draw(seed, sweep, stream_id(kWishartDiag, mode),
                                              (uint32_t)i, 0.5 * (double)(nu_c - i)));
  for (int i = (tid + nt / 2) % nt; i < K; i += nt)
    z[i] = normal_draw(seed, sweep, stream_id(kMuDraw, mode), 0u, (uint32_t)i);
  // off-diagonal draws two to a block: rows i and K - 2 - i together have at most K / 2 + 1 pairs
  const int slots = K / 2 + 1;
  for (int e = nt - 1 - tid; e < slots * (K / 2); e += nt) {
    const int s = e / slots, first = (K - s) / 2;  // pairs of row s
    int i = s, q = e % slots;
    if (q >= first) {
      i = K - 2 - s;
      q -= first;
      if (i <= s || q >= (s + 2) / 2) continue;  // row s alone in the middle, or past the last pair
    }
    const int left = K - 1 - i - 2 * q;  // draws of this pair on: 1 or more
    double z0, z1;
    normal_pair(seed, sweep, stream_id(kWishartOff, mode), (uint32_t)i, (uint32_t)q, &z0, &z1);
    Ct[elem_at(i + 1 + 2 * q, i)] = z0;
    if (left > 1) Ct[elem_at(i + 2 + 2 * q, i)] = z1;
  }
  for (int i = K + tid; i < n; i += nt) {
    for (int j = 0; j < i; j++) Ct[elem_at(i, j)] = 0.0;
    Ct[elem_at(i, i)] = 1.0;
    z[i] = 0.0;
  }
  for (int i = tid; i < n; i += nt)  // the diagonal tiles' upper parts are read too
    for (int j = i + 1; j < (i | 7) + 1; j++) Ct[tile_at(i >> 3, i >> 3) + tile_pos(i & 7, j & 7)] = 0.0;
}

// The update in two identities of the row-reversed matrix (n = K rounded up to 8, the identity
// before the reversed rows, so that both are whole tiles):
//   chol(X^{-1}) = J M^{-T} J with M = chol(J X J), J the index reversal: L(i, j) = Y(n-1-j, n-1-i),
//   Y = M^{-1};
//   Lambda = L c^T c L^T = B B^T with B = L c^T lower triangular, so chol(kappa_c Lambda) =
//   sqrt(kappa_c) B and mu = mu_c + B^{-T} z / sqrt(kappa_c).
template <int KP>
__device__ __forceinline__ void nw_tiles(const NwArgs& p, int K, Ctl* ctl, unsigned long long seed,
                                         double* smem) {
  using C = NwW<KP>;
  double* M = smem;
  double* Y = M + (size_t)C::TRI * 64;
  double* Ct = Y + (size_t)C::TRI * 64;
  double* Di = Ct + (size_t)C::TRI * 64;
  double* muc = Di + (size_t)C::NB * 64;
  double *y = muc + KP, *x = y + KP, *zero = x + KP, *z = zero + KP;
  volatile int* bad = reinterpret_cast<volatile int*>(z + KP);
  unsigned char* tri = reinterpret_cast<unsigned char*>(z + KP + 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int nb = (K + 7) / 8, n = 8 * nb, pad = n - K;
  const uint32_t sweep = ctl->sweep;
  const double kappa_c = p.kappa + (double)p.N;
  const int nu_c = p.nu + (int)p.N;
  if (tid == 0) *bad = 0;
  for (int q = tid; q < C::TRI; q += kNwThreads) {
    int a = 0;
    while (q >= (a + 1) * (a + 2) / 2) a++;
    tri[q] = (unsigned char)((a << 4) | (q - a * (a + 1) / 2));
  }
  const size_t rec = K + (size_t)K * K;
  auto stat = [&](size_t at) {
    double v = p.stats[at];
#pragma unroll 8
    for (int b = 1; b < p.nparts; b++) v += p.stats[b * rec + at];
    return v;
  };
  // x holds mu0 until the mean is solved for
  for (int i = tid; i < n; i += kNwThreads) {
    const double m0 = i < K && p.mu0 ? p.mu0[i] : 0.0;
    muc[i] = i < K ? (p.kappa * m0 + stat(i)) / kappa_c : 0.0;
    x[i] = m0;
    y[i] = zero[i] = 0.0;
  }
  __syncthreads();
  // M = J (T + N S + kappa mu0 mu0^T - kappa_c mu_c mu_c^T) J, a warp per tile; the identity in
  // the first `pad` rows and columns
#pragma unroll 5
  for (int q = warp; q < nb * (nb + 1) / 2; q += kNwThreads / 32) {
    const int a = 8 * (tri[q] >> 4) + g;
    double v[2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int b = 8 * (tri[q] & 15) + 2 * t + e, i = n - 1 - a, j = n - 1 - b;
      v[e] = a == b ? 1.0 : 0.0;
      if (a >= pad && b >= pad) {
        const size_t at = j + (size_t)i * K;
        const double T = p.T0 ? p.T0[at] : (a == b ? 1.0 : 0.0);
        v[e] = T + stat(K + at) + p.kappa * x[i] * x[j] - kappa_c * muc[i] * muc[j];
      }
    }
    *reinterpret_cast<double2*>(M + tile_at(tri[q] >> 4, tri[q] & 15) + tile_pos(g, 2 * t)) =
        make_double2(v[0], v[1]);
  }
  __syncthreads();
  if (warp < 8) {
    wide_factor<kNwHalf>(M, y, Di, nb, tid, 0, bad);
  } else {
    bartlett(Ct, z, K, n, nu_c, seed, sweep, (uint32_t)p.mode, tid - kNwHalf, kNwHalf);
  }
  __syncthreads();
  if (*bad) {
    if (tid == 0) atomicOr(&ctl->status, kStatHyperFail);
    return;
  }
  // Y = M^{-1}.  Its diagonal tiles are the factor's inverses, transposed back.
  for (int e = tid; e < 64 * nb; e += kNwThreads) {
    const int b = e >> 6, r = (e >> 3) & 7, c = e & 7;
    Y[tile_at(b, b) + tile_pos(r, c)] = Di[64 * b + tile_pos(c, r)];
  }
  __syncthreads();
  for (int bj = warp; bj < nb; bj += kNwThreads / 32) inverse_column(M, Y, bj, nb, lane);
  __syncthreads();
  // B = L c^T over M, L(i, j) = Y(n-1-j, n-1-i)
  for (int q = warp; q < nb * (nb + 1) / 2; q += kNwThreads / 32) {
    const int bi = tri[q] >> 4, bj = tri[q] & 15;
    double s[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    for (int k = bj; k <= bi; k++) {
      const double* A = Y + tile_at(nb - 1 - k, nb - 1 - bi);
      const double* B = Ct + tile_at(k, bj);
      mma_f64(s[0][0], s[0][1], A[tile_pos(7 - t, 7 - g)], B[tile_pos(t, g)]);
      mma_f64(s[1][0], s[1][1], A[tile_pos(3 - t, 7 - g)], B[tile_pos(t + 4, g)]);
    }
    *reinterpret_cast<double2*>(M + tile_at(bi, bj) + tile_pos(g, 2 * t)) =
        make_double2(s[0][0] + s[1][0], s[0][1] + s[1][1]);
  }
  __syncthreads();
  if (warp < 8) {
    // mu = mu_c + B^{-T} z / sqrt(kappa_c)
    if (tid < n) {
      // column c of the inverse of diagonal tile b
      const int b = tid >> 3, c = tid & 7;
      const double* D = M + tile_at(b, b);
      double v[8], ri[8];
#pragma unroll
      for (int r = 0; r < 8; r++) {
        ri[r] = 1.0 / D[tile_pos(r, r)];
        v[r] = r == c ? 1.0 : 0.0;
      }
#pragma unroll
      for (int r = 0; r < 8; r++) {
        v[r] *= ri[r];
#pragma unroll
        for (int k = r + 1; k < 8; k++) v[k] = fma(-D[tile_pos(k, r)], v[r], v[k]);
      }
      store_row8(Di + 64 * b, c, v);
      y[tid] = z[tid] / sqrt(kappa_c);
    }
    group_sync<kNwHalf>(0);
    wide_back<kNwHalf>(M, y, Di, x, nb, tid, 0);
    if (tid < K) p.mu[tid] = x[tid] + muc[tid];
  } else {
    // Lambda = B B^T
    for (int q = warp - 8; q < nb * (nb + 1) / 2; q += 8) {
      const int bi = tri[q] >> 4, bj = tri[q] & 15;
      double s[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
      for (int k = 0; k <= bj; k++) {
        const double* A = M + tile_at(bi, k);
        const double* B = M + tile_at(bj, k);
        mma_f64(s[0][0], s[0][1], A[tile_pos(g, t)], B[tile_pos(g, t)]);
        mma_f64(s[1][0], s[1][1], A[tile_pos(g, t + 4)], B[tile_pos(g, t + 4)]);
      }
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int i = 8 * bi + g, j = 8 * bj + 2 * t + e;
        const double v = s[0][e] + s[1][e];
        if (i < K && j < K) {
          p.Lambda[i + (size_t)j * K] = v;
          if (bi != bj) p.Lambda[j + (size_t)i * K] = v;
        }
      }
    }
  }
}

template <int KP>
__global__ void __launch_bounds__(kNwThreads, 1)
    k_nw(const NwPair args, int K, Ctl* ctl, unsigned long long seed) {
  extern __shared__ __align__(16) double nsm[];
  nw_tiles<KP>(args.m[blockIdx.x], K, ctl, seed, nsm);
}

template <int KP>
void nw_launch(const NwPair& a, int count, int K, Ctl* ctl, unsigned long long seed,
               cudaStream_t s) {
  constexpr size_t smem = sizeof(double) * NwW<KP>::kDoubles;
  static_assert(smem <= 227 * 1024, "Normal-Wishart matrices exceed the shared memory of one CTA");
  static bool configured[64] = {false};
  int dev = 0;
  MG_CUDA(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    MG_CUDA(cudaFuncSetAttribute(k_nw<KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured[dev & 63] = true;
  }
  k_nw<KP><<<count, kNwThreads, smem, s>>>(a, K, ctl, seed);
  MG_CUDA(cudaGetLastError());
}

void nw_dispatch(const NwPair& a, int count, int K, Ctl* ctl, unsigned long long seed,
                 cudaStream_t s) {
  if (K <= 32) nw_launch<32>(a, count, K, ctl, seed, s);
  else if (K <= 64) nw_launch<64>(a, count, K, ctl, seed, s);
  else nw_launch<128>(a, count, K, ctl, seed, s);
}

}  // namespace

void launch_stats_wide(const void* U, bool f32, const double* Uhat, long long N, int K, int stride,
                       int uhat_stride, double* partials, int nblocks, cudaStream_t s) {
  const StatsArgs a{{U, nullptr}, Uhat, {N, 0}, {(N + nblocks - 1) / nblocks, 0}, {nblocks, 0},
                    {partials, nullptr}};
  if (Uhat && K > 64) throw MgError(MG_ERR_ARG, "side information supports num_latent <= 64");
  if (f32) stats_launch<float>(a, K, stride, uhat_stride, s);
  else stats_launch<double>(a, K, stride, uhat_stride, s);
}

void launch_stats_wide_pair(const PriorPair& pp, bool f32, int K, int stride, cudaStream_t s) {
  const StatsArgs a{{pp.U[0], pp.U[1]}, nullptr, {pp.N[0], pp.N[1]},
                    {pp.rows_per_block[0], pp.rows_per_block[1]},
                    {pp.nblocks[0], pp.nblocks[1]}, {pp.partials[0], pp.partials[1]}};
  if (f32) stats_launch<float>(a, K, stride, 0, s);
  else stats_launch<double>(a, K, stride, 0, s);
}

void launch_normal_wishart(const double* partials, int nparts, long long N, int K,
                           const double* mu0, double kappa, const double* T0, int nu,
                           Ctl* ctl, unsigned long long seed, int mode, double* mu_out,
                           double* Lambda_out, cudaStream_t s) {
  NwPair a{};
  a.m[0] = NwArgs{partials, nparts, mu0, T0, kappa, N, nu, mode, mu_out, Lambda_out};
  nw_dispatch(a, 1, K, ctl, seed, s);
}

void launch_normal_wishart_pair(const PriorPair& pp, int K, Ctl* ctl, unsigned long long seed,
                                cudaStream_t s) {
  NwPair a{};
  for (int m = 0; m < 2; m++) {
    const bool few = few_parts(pp.nblocks[m], K);
    a.m[m] = NwArgs{few ? pp.partials[m] : pp.final_[m], few ? pp.nblocks[m] : 1, pp.mu0[m], pp.T0[m], pp.kappa[m], pp.N[m], pp.nu[m], m, pp.mu[m],
                    pp.Lambda[m]};
  }
  nw_dispatch(a, 2, K, ctl, seed, s);
}

}  // namespace mg
