// Prior update of the univariate sampler (MacauOnePrior, macauoneprior.cpp:189-290): the link
// matrix, one coefficient at a time, and the per-dimension lambda_beta.  The Normal-Wishart part
// (sample_mu_lambda) and compute_uhat reuse the BPMF statistics kernels and the SpMM.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "rng.cuh"

namespace mg {
namespace {

constexpr int kBetaThreads = 512;
constexpr int kBetaWarps = kBetaThreads / 32;

// One link coefficient per lane d < dc (dimension d0 + d) of feature f, sample_beta's update
// (macauoneprior.cpp:243-252):
//   A = lambda_beta_d + lambda_d colsq_f,   B = lambda_d (zx_d + beta_df colsq_f),
//   beta_df <- B / A + z / sqrt(A),   delta_d = beta_df old - beta_df new.
// zx, lam, lb are this lane's components; the N(0,1) draw of (f, d0 + lane) comes from draws
// (filled by k_beta_draws before the sequential sweep); returns delta (0 for lanes >= dc).
__device__ __forceinline__ double beta_coef(int lane, int dc, int d0, int f, double zx,
                                            double lam, double lb, double cs, double* beta,
                                            int bstride, const double* __restrict__ draws) {
  if (lane >= dc) return 0.0;
  const int dx = d0 + lane;
  double* bp = beta + (size_t)f * bstride + dx;
  const double b = *bp;
  const double A = lb + lam * cs;
  const double B = lam * (zx + b * cs);
  const double Ainv = 1.0 / A;
  const double bn = B * Ainv + sqrt(Ainv) * draws[(size_t)f * bstride + dx];
  *bp = bn;
  return b - bn;
}

// sample_beta (macauoneprior.cpp:216-257) for the dimensions d0 .. d0 + 3 of block blockIdx.x.
// Z = U - mu - Uhat (N x zstride, this block's four columns) is formed first; then the features
// are visited level by level.  lvl_feat lists the features sorted by (level, index), where a
// feature's level is one more than the highest level of an earlier feature sharing a row with
// it, so the features of one level touch disjoint rows of Z and their updates commute: the
// result equals the reference's feature-by-feature order.  A level marked in lvl_warp (many
// features, or none longer than 1024 entries) gives one feature to each warp; the others give
// each feature in turn to the whole block.
template <typename T>
__global__ void __launch_bounds__(kBetaThreads)
    k_beta_one(const long long* __restrict__ tptr, const int* __restrict__ tidx,
               const double* __restrict__ tval, const double* __restrict__ colsq,
               const int* __restrict__ lvl_ptr, const int* __restrict__ lvl_feat,
               const int* __restrict__ lvl_warp, int nlevels, const T* __restrict__ U, int ustride, const double* __restrict__ mu,
               const double* __restrict__ uhat, int hstride, const double* __restrict__ Lambda,
               const double* __restrict__ lambda_beta, int K, long long N,
               double* __restrict__ beta, int bstride, double* __restrict__ Z, int zstride,
               const double* __restrict__ draws) {
  __shared__ double red[kBetaWarps][4];
  __shared__ double dl[4];
  const int d0 = blockIdx.x * 4, dc = min(4, K - d0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // this lane's dimension d0 + lane (lanes 0 .. dc - 1 update the coefficients)
  const double lam = lane < dc ? Lambda[(size_t)(d0 + lane) * (K + 1)] : 0.0;
  const double lb = lane < dc ? lambda_beta[d0 + lane] : 1.0;
  for (long long i = threadIdx.x; i < N; i += kBetaThreads)
    for (int d = 0; d < dc; d++)
      Z[i * zstride + d0 + d] =
          (double)U[i * ustride + d0 + d] - mu[d0 + d] - uhat[i * hstride + d0 + d];
  __syncthreads();
  for (int L = 0; L < nlevels; L++) {
    const int f0 = lvl_ptr[L], f1 = lvl_ptr[L + 1];
    if (lvl_warp[L]) {
      for (int q = f0 + warp; q < f1; q += kBetaWarps) {
        const int f = lvl_feat[q];
        double zx[4] = {0.0, 0.0, 0.0, 0.0};
        for (long long e = tptr[f] + lane; e < tptr[f + 1]; e += 32) {
          const double v = tval ? tval[e] : 1.0;
          const double* zr = Z + (size_t)tidx[e] * zstride + d0;
#pragma unroll
          for (int d = 0; d < 4; d++)
            if (d < dc) zx[d] = fma(v, zr[d], zx[d]);
        }
#pragma unroll
        for (int d = 0; d < 4; d++)
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) zx[d] += __shfl_xor_sync(0xffffffffu, zx[d], o);
        double mine = 0.0;
#pragma unroll
        for (int d = 0; d < 4; d++)
          if (lane == d) mine = zx[d];
        const double my =
            beta_coef(lane, dc, d0, f, mine, lam, lb, colsq[f], beta, bstride, draws);
        double delta[4];
#pragma unroll
        for (int d = 0; d < 4; d++) delta[d] = __shfl_sync(0xffffffffu, my, d);
        for (long long e = tptr[f] + lane; e < tptr[f + 1]; e += 32) {
          const double v = tval ? tval[e] : 1.0;
          double* zr = Z + (size_t)tidx[e] * zstride + d0;
#pragma unroll
          for (int d = 0; d < 4; d++)
            if (d < dc) zr[d] = fma(v, delta[d], zr[d]);
        }
      }
    } else {
      for (int q = f0; q < f1; q++) {
        const int f = lvl_feat[q];
        double zx[4] = {0.0, 0.0, 0.0, 0.0};
        for (long long e = tptr[f] + threadIdx.x; e < tptr[f + 1]; e += kBetaThreads) {
          const double v = tval ? tval[e] : 1.0;
          const double* zr = Z + (size_t)tidx[e] * zstride + d0;
#pragma unroll
          for (int d = 0; d < 4; d++)
            if (d < dc) zx[d] = fma(v, zr[d], zx[d]);
        }
#pragma unroll
        for (int d = 0; d < 4; d++) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) zx[d] += __shfl_xor_sync(0xffffffffu, zx[d], o);
          if (lane == 0) red[warp][d] = zx[d];
        }
        __syncthreads();
        if (warp == 0) {
          double s = 0.0;
          if (lane < dc)
            for (int w = 0; w < kBetaWarps; w++) s += red[w][lane];
          const double my =
              beta_coef(lane, dc, d0, f, s, lam, lb, colsq[f], beta, bstride, draws);
          if (lane < 4) dl[lane] = my;
        }
        __syncthreads();
        const double delta[4] = {dl[0], dl[1], dl[2], dl[3]};
        for (long long e = tptr[f] + threadIdx.x; e < tptr[f + 1]; e += kBetaThreads) {
          const double v = tval ? tval[e] : 1.0;
          double* zr = Z + (size_t)tidx[e] * zstride + d0;
#pragma unroll
          for (int d = 0; d < 4; d++)
            if (d < dc) zr[d] = fma(v, delta[d], zr[d]);
        }
      }
    }
    __syncthreads();
  }
}

// The same link sampler with one block per dimension d and this dimension's column of Z held in
// shared memory (N doubles, N <= kZsMax), so the feature-by-feature chain reads and writes no
// global memory but beta, with 32 warps per block.
//   What bounds it: the chain over the levels.  A level gives each of its features to a warp, or each
// in turn to the whole block (lvl_warp, by the estimate of beta_one_warp_level).  While a feature is
// processed, everything about the next one that no other feature changes is loaded: its entry
// range, the first entries' rows, its coefficient and draw with the reciprocal and the square root
// they are scaled by, and the next level's bounds.  The block's sum takes one barrier: every
// warp adds the 32 warps' sums for itself by a shuffle tree.  (Reading each entry's row twice from
// global memory, a warp for features of up to 1,024 entries and one thread to add the warps' sums,
// 1,294 us for the 8,193 features, 250,000 entries and 32 dimensions of a 5,003-row matrix.)
constexpr int kZsMax = 26 * 1024;
constexpr int kSmemThreads = 1024;
constexpr int kSmemWarps = kSmemThreads / 32;

// A feature's constants for one dimension, and the first NP entries of a thread that takes entries
// first, first + stride, ...
template <bool BINARY, int NP>
struct FeaturePre {
  int f, len;
  long long begin;
  double bcs, b, ainv, sz;
  int i[NP];
  double v[BINARY ? 1 : NP];
};

struct BetaOne {
  const int* tidx;
  const double* tval;
  const double* colsq;
  const int* lvl_feat;
  const longlong2* lvl_range;
  const double* draws;
  double* beta;
  int bstride;
  double lam, lb;
  int d;
};

template <bool BINARY, int NP>
__device__ __forceinline__ FeaturePre<BINARY, NP> fetch_feature(const BetaOne& p, int q, int first,
                                                               int stride) {
  FeaturePre<BINARY, NP> r;
  r.f = p.lvl_feat[q];
  const longlong2 rg = p.lvl_range[q];
  r.begin = rg.x;
  r.len = (int)(rg.y - rg.x);
  const double cs = p.colsq[r.f];
  r.b = p.beta[(size_t)r.f * p.bstride + p.d];
  r.bcs = r.b * cs;
  r.ainv = 1.0 / (p.lb + p.lam * cs);
  r.sz = sqrt(r.ainv) * p.draws[(size_t)r.f * p.bstride + p.d];
#pragma unroll
  for (int k = 0; k < NP; k++) {
    const int e = first + k * stride;
    r.i[k] = e < r.len ? p.tidx[r.begin + e] : -1;
    if constexpr (!BINARY) r.v[k] = e < r.len ? p.tval[r.begin + e] : 0.0;
  }
  return r;
}

// sum of v Z over the thread's entries
template <bool BINARY, int NP>
__device__ __forceinline__ double feature_dot(const BetaOne& p, const FeaturePre<BINARY, NP>& r,
                                              const double* Zs, int first, int stride) {
  double zx = 0.0;
#pragma unroll
  for (int k = 0; k < NP; k++)
    if (r.i[k] >= 0) zx = BINARY ? zx + Zs[r.i[k]] : fma(r.v[BINARY ? 0 : k], Zs[r.i[k]], zx);
#pragma unroll 4
  for (int e = first + NP * stride; e < r.len; e += stride) {
    const double z = Zs[p.tidx[r.begin + e]];
    zx = BINARY ? zx + z : fma(p.tval[r.begin + e], z, zx);
  }
  return zx;
}
// Z += v delta over the thread's entries (one entry per row of Z)
template <bool BINARY, int NP>
__device__ __forceinline__ void feature_add(const BetaOne& p, const FeaturePre<BINARY, NP>& r,
                                            double* Zs, int first, int stride, double delta) {
#pragma unroll
  for (int k = 0; k < NP; k++)
    if (r.i[k] >= 0)
      Zs[r.i[k]] = BINARY ? Zs[r.i[k]] + delta : fma(r.v[BINARY ? 0 : k], delta, Zs[r.i[k]]);
#pragma unroll 4
  for (int e = first + NP * stride; e < r.len; e += stride) {
    const int i = p.tidx[r.begin + e];
    Zs[i] = BINARY ? Zs[i] + delta : fma(p.tval[r.begin + e], delta, Zs[i]);
  }
}
// The new coefficient (macauoneprior.cpp:243-252) from the sum over the feature's entries.
template <bool BINARY, int NP>
__device__ __forceinline__ double new_coef(const BetaOne& p, const FeaturePre<BINARY, NP>& r,
                                           double zx) {
  return p.lam * (zx + r.bcs) * r.ainv + r.sz;
}
__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

template <typename T, bool BINARY>
__global__ void __launch_bounds__(kSmemThreads)
    k_beta_one_smem(const int* __restrict__ tidx, const double* __restrict__ tval,
                    const double* __restrict__ colsq, const int* __restrict__ lvl_ptr,
                    const int* __restrict__ lvl_feat, const longlong2* __restrict__ lvl_range,
                    const int* __restrict__ lvl_warp, int nlevels, const T* __restrict__ U,
                    int ustride, const double* __restrict__ mu,
                    const double* __restrict__ uhat, int hstride,
                    const double* __restrict__ Lambda, const double* __restrict__ lambda_beta,
                    int K, int N, double* __restrict__ beta, int bstride,
                    const double* __restrict__ draws) {
  extern __shared__ double Zs[];
  __shared__ double red[2][kSmemWarps];
  constexpr int NP = BINARY ? 4 : 2;  // entries held ahead per thread
  const int d = blockIdx.x, tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const BetaOne p{tidx, tval, colsq, lvl_feat, lvl_range, draws, beta, bstride,
                  Lambda[(size_t)d * (K + 1)], lambda_beta[d], d};
  for (int i = tid; i < N; i += kSmemThreads)
    Zs[i] = (double)U[(size_t)i * ustride + d] - mu[d] - uhat[(size_t)i * hstride + d];
  FeaturePre<BINARY, NP> cur{};
  int cur_q = -1;  // the feature in `cur`, fetched for this thread's share of it, or -1
  bool cur_block = false;
  int buf = 0;
  int f0 = 0, f1 = nlevels > 0 ? lvl_ptr[1] : 0, mode = nlevels > 0 ? lvl_warp[0] : 0;
  __syncthreads();
  for (int L = 0; L < nlevels; L++) {
    // the next level's bounds and mode
    const bool more = L + 1 < nlevels;
    const int f2 = more ? lvl_ptr[L + 2] : f1, mode2 = more ? lvl_warp[L + 1] : -1;
    // the feature this thread meets first in the next level
    const int q2 = !more ? -1 : mode2 == 0 ? f1 : (f1 + warp < f2 ? f1 + warp : -1);
    const int first2 = mode2 == 0 ? tid : lane, stride2 = mode2 == 0 ? kSmemThreads : 32;
    if (mode != 0) {
      // one feature per warp
      int q = f0 + warp;
      if (q < f1 && (cur_q != q || cur_block)) {
        cur = fetch_feature<BINARY, NP>(p, q, lane, 32);
        cur_q = q;
      }
      if (q >= f1 && q2 >= 0) {  // nothing to do in this level
        cur = fetch_feature<BINARY, NP>(p, q2, first2, stride2);
        cur_q = q2;
        cur_block = mode2 == 0;
      }
      for (; q < f1; q += kSmemWarps) {
        const bool last = q + kSmemWarps >= f1;
        const int qn = last ? q2 : q + kSmemWarps;
        FeaturePre<BINARY, NP> nxt{};
        if (qn >= 0)
          nxt = fetch_feature<BINARY, NP>(p, qn, last ? first2 : lane, last ? stride2 : 32);
        const double bn = new_coef(p, cur, warp_sum(feature_dot(p, cur, Zs, lane, 32)));
        if (lane == 0) beta[(size_t)cur.f * bstride + d] = bn;
        feature_add(p, cur, Zs, lane, 32, cur.b - bn);
        __syncwarp();
        cur = nxt;
        cur_q = qn;
        cur_block = last && mode2 == 0;
      }
    } else {
      // each feature by the whole block
      for (int q = f0; q < f1; q++) {
        if (cur_q != q || !cur_block) cur = fetch_feature<BINARY, NP>(p, q, tid, kSmemThreads);
        const bool last = q + 1 == f1;
        const int qn = last ? q2 : q + 1;
        FeaturePre<BINARY, NP> nxt{};
        if (qn >= 0)
          nxt = fetch_feature<BINARY, NP>(p, qn, last ? first2 : tid,
                                          last ? stride2 : kSmemThreads);
        const double part = warp_sum(feature_dot(p, cur, Zs, tid, kSmemThreads));
        if (lane == 0) red[buf][warp] = part;
        __syncthreads();
        const double bn = new_coef(p, cur, warp_sum(red[buf][lane]));
        buf ^= 1;  // the next sum goes to the other half: one barrier between writes and reads
        if (tid == 0) beta[(size_t)cur.f * bstride + d] = bn;
        feature_add(p, cur, Zs, tid, kSmemThreads, cur.b - bn);
        cur = nxt;
        cur_q = qn;
        cur_block = !last || mode2 == 0;
      }
    }
    __syncthreads();
    f0 = f1;
    f1 = f2;
    mode = mode2;
  }
}

// The link sampler's N(0,1) draws, keyed (kBetaOne, feature f, dimension d) like
// bmrandn_single per feature (macauoneprior.cpp:241): draws[f * stride + d], one Philox block
// per pair of dimensions.
__global__ void k_beta_draws(long long nfeat, int K, int stride, const Ctl* ctl,
                             unsigned long long seed, int mode, double* __restrict__ draws) {
  const int pairs = (K + 1) / 2;
  const uint32_t st = stream_id(kBetaOne, (uint32_t)mode);
  const uint32_t sweep = ctl->sweep;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < nfeat * pairs;
       e += (long long)gridDim.x * blockDim.x) {
    const long long f = e / pairs;
    const int q = (int)(e % pairs);
    double z0, z1;
    normal_pair(seed, sweep, st, (uint32_t)f, (uint32_t)q, &z0, &z1);
    draws[f * stride + 2 * q] = z0;
    if (2 * q + 1 < K) draws[f * stride + 2 * q + 1] = z1;
  }
}

// sample_lambda_beta (macauoneprior.cpp:267-290): lambda_beta_d ~ Gamma(a0 + nfeat / 2,
// 1 / (b0 + sum_f beta_df^2 / 2)), keyed (kLambdaBeta, d).  First the squares' sums per block of
// features, rows read whole (thread (r, d): rows r, r + R, ... of the block), the block's row
// groups added in order.  (One CTA, a warp per dimension reading a column of beta, took 148 us at
// 8,193 features and 32 dimensions.)
constexpr int kSqThreads = 256;
__global__ void __launch_bounds__(kSqThreads)
    k_beta_sq(const double* __restrict__ beta, int bstride, long long nfeat, int K,
              long long rows_per_block, double* __restrict__ parts) {
  __shared__ double s[kSqThreads];
  const int W = K <= 32 ? 32 : 64, R = kSqThreads / W;
  const int d = threadIdx.x % W, rg = threadIdx.x / W;
  const long long r1 = min(nfeat, (blockIdx.x + 1) * rows_per_block);
  double acc = 0.0;
  if (d < K)
#pragma unroll 4
    for (long long f = blockIdx.x * rows_per_block + rg; f < r1; f += R) {
      const double b = beta[f * bstride + d];
      acc = fma(b, b, acc);
    }
  s[threadIdx.x] = acc;
  __syncthreads();
  if (rg == 0 && d < K) {
    for (int q = 1; q < R; q++) acc += s[q * W + d];
    parts[(size_t)blockIdx.x * K + d] = acc;
  }
}
__global__ void k_lambda_beta_one(const double* __restrict__ parts, int nparts, long long nfeat,
                                  int K, double a0, double b0, const Ctl* ctl,
                                  unsigned long long seed, int mode,
                                  double* __restrict__ lambda_beta) {
  const int d = threadIdx.x;
  if (d >= K) return;
  double s = 0.0;
#pragma unroll 8
  for (int b = 0; b < nparts; b++) s += parts[(size_t)b * K + d];
  lambda_beta[d] = gamma_draw(seed, ctl->sweep, stream_id(kLambdaBeta, (uint32_t)mode), (uint32_t)d,
                              a0 + (double)nfeat / 2.0) *
                   (1.0 / (b0 + s / 2.0));
}

template <typename T, bool BINARY>
void beta_smem(const DevCsr& Ft, const double* colsq, const int* lvl_ptr, const int* lvl_feat,
               const longlong2* lvl_range, const int* lvl_warp, int nlevels, const void* U,
               int ustride, const double* mu, const double* uhat, int hstride,
               const double* Lambda, const double* lambda_beta, int K, long long N, double* beta,
               int bstride, const double* draws, cudaStream_t s) {
  static bool configured[64] = {false};
  int dev = 0;
  MG_CUDA(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    MG_CUDA(cudaFuncSetAttribute(k_beta_one_smem<T, BINARY>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double) * kZsMax)));
    configured[dev & 63] = true;
  }
  k_beta_one_smem<T, BINARY><<<K, kSmemThreads, sizeof(double) * (size_t)N, s>>>(
      Ft.idx, Ft.val, colsq, lvl_ptr, lvl_feat, lvl_range, lvl_warp, nlevels, (const T*)U, ustride,
      mu, uhat, hstride, Lambda, lambda_beta, K, (int)N, beta, bstride, draws);
  MG_CUDA(cudaGetLastError());
}

}  // namespace

void launch_beta_one(const DevCsr& Ft, const double* colsq, const int* lvl_ptr,
                     const int* lvl_feat, const longlong2* lvl_range, const int* lvl_warp,
                     int nlevels, const void* U, bool f32, int ustride,
                     const double* mu, const double* uhat, int hstride, const double* Lambda,
                     const double* lambda_beta, int K, long long N, double* beta, int bstride,
                     double* Z, int zstride, double* draws, const Ctl* ctl,
                     unsigned long long seed, int mode, cudaStream_t s) {
  const long long work = Ft.nrow * ((K + 1) / 2);
  k_beta_draws<<<(int)std::min<long long>(4736, (work + 255) / 256), 256, 0, s>>>(
      Ft.nrow, K, bstride, ctl, seed, mode, draws);
  MG_CUDA(cudaGetLastError());
  if (N <= kZsMax) {  // one block per dimension, Z's column in shared memory
    const auto run = f32 ? (Ft.val ? beta_smem<float, false> : beta_smem<float, true>)
                         : (Ft.val ? beta_smem<double, false> : beta_smem<double, true>);
    run(Ft, colsq, lvl_ptr, lvl_feat, lvl_range, lvl_warp, nlevels, U, ustride, mu, uhat, hstride,
        Lambda, lambda_beta, K, N, beta, bstride, draws, s);
    return;
  }
  const int blocks = (K + 3) / 4;
  if (f32)
    k_beta_one<float><<<blocks, kBetaThreads, 0, s>>>(
        Ft.ptr, Ft.idx, Ft.val, colsq, lvl_ptr, lvl_feat, lvl_warp, nlevels, (const float*)U, ustride, mu,
        uhat, hstride, Lambda, lambda_beta, K, N, beta, bstride, Z, zstride, draws);
  else
    k_beta_one<double><<<blocks, kBetaThreads, 0, s>>>(
        Ft.ptr, Ft.idx, Ft.val, colsq, lvl_ptr, lvl_feat, lvl_warp, nlevels, (const double*)U, ustride, mu,
        uhat, hstride, Lambda, lambda_beta, K, N, beta, bstride, Z, zstride, draws);
  MG_CUDA(cudaGetLastError());
}

// Cycles of a level by a warp per feature (32 at a time, a step of 32 entries read, summed and updated
// in about 100 cycles beyond the four held ahead) against each feature by the whole block (about
// 600 with its barrier and the two shuffle trees).
bool beta_one_warp_level(long long N, long long nfeat, long long longest) {
  if (N > kZsMax) return nfeat >= 8 || longest <= 1024;  // k_beta_one
  const long long steps = (longest + 31) / 32;
  const long long warp = (nfeat + kSmemWarps - 1) / kSmemWarps * (400 + 100 * std::max(0LL, steps - 4));
  return warp <= 600 * nfeat;
}

void launch_lambda_beta_one(const double* beta, int bstride, long long nfeat, int K, double a0,
                            double b0, const Ctl* ctl, unsigned long long seed, int mode,
                            double* parts, double* lambda_beta, cudaStream_t s) {
  // `parts` holds nfeat * bstride doubles: at most one record of K per 64 features is written
  const int nb = (int)std::min<long long>(148, (nfeat + 63) / 64);
  k_beta_sq<<<nb, kSqThreads, 0, s>>>(beta, bstride, nfeat, K, (nfeat + nb - 1) / nb, parts);
  MG_CUDA(cudaGetLastError());
  k_lambda_beta_one<<<1, 64, 0, s>>>(parts, nb, nfeat, K, a0, b0, ctl, seed, mode, lambda_beta);
  MG_CUDA(cudaGetLastError());
}

}  // namespace mg
