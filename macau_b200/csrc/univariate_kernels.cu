// Prior update of the univariate sampler (MacauOnePrior, macauoneprior.cpp:189-290): the link
// matrix, one coefficient at a time, and the per-dimension lambda_beta.  The Normal-Wishart part
// (sample_mu_lambda) and compute_uhat reuse the BPMF statistics kernels and the SpMM.
#include <cuda_runtime.h>

#include <algorithm>
#include <numeric>
#include <vector>

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
// are visited level by level.  lvl_feat lists the features sorted by level, where a
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
// global memory but beta, with 16 warps per block (with 32 the idle ones' instructions cost more than
// their share of the work saves, with 8 the long features take longer).
//   What bounds it: the chain over the levels, and in wide levels the instructions per feature.  A
// level gives its features to the block, each in turn, to a warp each or to a lane each (lvl_warp,
// beta_one_levels).  Nothing that a feature needs is more than one memory latency behind when its
// level begins: the bounds of a level are loaded three levels ahead, the id and entry range of the
// feature that a thread takes in it two ahead, its first entries' rows (and values), coefficient, draw
// and squared norm one ahead.  The block's sum takes one barrier: every warp adds the warps' sums for
// itself by a shuffle tree.
//   Microseconds a link draw, with 1,024 threads, one feature ahead and a warp per short feature, then
// as it is: 5,003 rows, 8,193 features, 250,000 entries, K = 32: 1,354 -> 996 (weighted 1,437 -> 996);
// 20,000 rows, 32,768 features, 1M entries: 3,554 -> 2,324; 1,000 rows, 30,000 features, K = 8: 1,197
// -> 393.  Entries held ahead: six made wide levels slower than two (1,718 at the last size before the
// lanes, 1,500) and spilled 260 bytes with weights.
constexpr int kZsMax = 26 * 1024;
constexpr int kSmemThreads = 512;
constexpr int kNp = 2;  // entries held ahead per thread
constexpr int kSmemWarps = kSmemThreads / 32;
// A chain whose other mode has a block-CG link (hyper_ordered.cu): each feature's sum as it was
// recorded, a block's over 1,024 threads and its warps' sums added one after the other.
constexpr int kOrderedThreads = 1024;

// A level: features f0 .. f1 - 1 of the level order, taken by (lvl_warp) the block each in turn, a
// warp each or a lane each.
enum { kByBlock = 0, kByWarp = 1, kByLane = 2 };
struct LevelPre {
  int f0, f1, by;
};
// The id and entry range of the feature a thread takes (f < 0: none).  These and FeaturePre hold what
// the loads return and nothing computed from it: an instruction that used a value here would
// hold the warp until it arrives.
struct FeatureId {
  int f;
  longlong2 rg;
};
// A feature's constants for one dimension, and the first NP entries of a thread that takes entries
// first, first + stride, ...
template <bool BINARY, int NP>
struct FeaturePre {
  int f, len;
  long long begin;
  double b, cs, z;
  int i[NP];
  double v[BINARY ? 1 : NP];
};

struct BetaOne {
  const int* tidx;
  const double* tval;
  const double* colsq;
  const int* lvl_ptr;
  const int* lvl_feat;
  const longlong2* lvl_range;
  const int* lvl_warp;
  const double* draws;
  double* beta;
  int bstride, nlevels;
  double lam, lb;
  int d;
};

__device__ __forceinline__ LevelPre fetch_level(const BetaOne& p, int L) {
  if (L >= p.nlevels) return {0, 0, kByWarp};
  return {p.lvl_ptr[L], p.lvl_ptr[L + 1], p.lvl_warp[L]};
}
__device__ __forceinline__ FeatureId fetch_id(const BetaOne& p, int q, int end) {
  FeatureId id{-1, make_longlong2(0, 0)};
  if (q < end) {
    id.f = p.lvl_feat[q];
    id.rg = p.lvl_range[q];
  }
  return id;
}
template <bool BINARY, int NP>
__device__ __forceinline__ FeaturePre<BINARY, NP> fetch_feature(const BetaOne& p, const FeatureId& id,
                                                               int first, int stride) {
  FeaturePre<BINARY, NP> r;
  r.f = id.f;
  r.begin = id.rg.x;
  r.len = (int)(id.rg.y - id.rg.x);
  r.b = r.cs = r.z = 0.0;
#pragma unroll
  for (int k = 0; k < NP; k++) {
    const int e = first + k * stride;
    r.i[k] = -1;
    if (e < r.len) r.i[k] = p.tidx[r.begin + e];
    if constexpr (!BINARY) {
      r.v[k] = 0.0;
      if (e < r.len) r.v[k] = p.tval[r.begin + e];
    }
  }
  if (id.f >= 0) {
    r.cs = p.colsq[id.f];
    r.b = p.beta[(size_t)id.f * p.bstride + p.d];
    r.z = p.draws[(size_t)id.f * p.bstride + p.d];
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
  const double ainv = 1.0 / (p.lb + p.lam * r.cs);
  return p.lam * (zx + r.b * r.cs) * ainv + sqrt(ainv) * r.z;
}
__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

template <typename T, bool BINARY, int THREADS, int NP>
__global__ void __launch_bounds__(THREADS)
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
  __shared__ double red[2][32];
  constexpr int WARPS = THREADS / 32;
  const int d = blockIdx.x, tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const BetaOne p{tidx, tval, colsq, lvl_ptr, lvl_feat, lvl_range, lvl_warp, draws, beta, bstride,
                  nlevels, Lambda[(size_t)d * (K + 1)], lambda_beta[d], d};
  for (int i = tid; i < N; i += THREADS)
    Zs[i] = (double)U[(size_t)i * ustride + d] - mu[d] - uhat[(size_t)i * hstride + d];
  // this thread's first feature of a level, and its share of the entries
  auto first_id = [&](const LevelPre& l) {
    return fetch_id(p, l.f0 + (l.by == kByLane ? tid : l.by == kByWarp ? warp : 0), l.f1);
  };
  auto share = [&](const LevelPre& l, const FeatureId& id) {
    return fetch_feature<BINARY, NP>(p, id, l.by == kByLane ? 0 : l.by == kByWarp ? lane : tid,
                                     l.by == kByLane ? 1 : l.by == kByWarp ? 32 : THREADS);
  };
  // rings by level: bounds, ids and features; the loop runs four levels at a time so that every
  // ring index is a constant (a register that a load is still to fill is never moved)
  LevelPre lev[4] = {fetch_level(p, 0), fetch_level(p, 1), fetch_level(p, 2), {0, 0, kByWarp}};
  FeatureId id[2] = {{-1, make_longlong2(0, 0)}, first_id(lev[1])};
  FeaturePre<BINARY, NP> pre[2];
  pre[0] = share(lev[0], first_id(lev[0]));
  int buf = 0;
  __syncthreads();
  for (int L0 = 0; L0 < nlevels; L0 += 4) {
#pragma unroll
    for (int u = 0; u < 4; u++) {
      if (L0 + u >= nlevels) break;
      const LevelPre& l = lev[u];
      lev[(u + 3) & 3] = fetch_level(p, L0 + u + 3);
      id[u & 1] = first_id(lev[(u + 2) & 3]);
      pre[(u + 1) & 1] = share(lev[(u + 1) & 3], id[(u + 1) & 1]);
      FeaturePre<BINARY, NP> cur = pre[u & 1];
      if (l.by == kByLane) {
        for (int q = l.f0 + tid; q < l.f1; q += THREADS) {
          FeaturePre<BINARY, NP> next{};
          if (q + THREADS < l.f1) next = share(l, fetch_id(p, q + THREADS, l.f1));
          const double bn = new_coef(p, cur, feature_dot(p, cur, Zs, 0, 1));
          beta[(size_t)cur.f * bstride + d] = bn;
          feature_add(p, cur, Zs, 0, 1, cur.b - bn);
          cur = next;
        }
      } else if (l.by == kByWarp) {
        // one feature per warp
        for (int q = l.f0 + warp; q < l.f1; q += WARPS) {
          FeaturePre<BINARY, NP> next{};
          if (q + WARPS < l.f1) next = share(l, fetch_id(p, q + WARPS, l.f1));
          const double bn = new_coef(p, cur, warp_sum(feature_dot(p, cur, Zs, lane, 32)));
          if (lane == 0) beta[(size_t)cur.f * bstride + d] = bn;
          feature_add(p, cur, Zs, lane, 32, cur.b - bn);
          cur = next;
        }
      } else {
        // each feature by the whole block
        for (int q = l.f0; q < l.f1; q++) {
          FeaturePre<BINARY, NP> next{};
          if (q + 1 < l.f1) next = share(l, fetch_id(p, q + 1, l.f1));
          const double part = warp_sum(feature_dot(p, cur, Zs, tid, THREADS));
          if (lane == 0) red[buf][warp] = part;
          __syncthreads();
          double sum;
          if constexpr (THREADS == kOrderedThreads) {
            sum = 0.0;
            for (int w = 0; w < WARPS; w++) sum += red[buf][w];
          } else {
            sum = warp_sum(lane < WARPS ? red[buf][lane] : 0.0);
          }
          const double bn = new_coef(p, cur, sum);
          buf ^= 1;  // the next sum goes to the other half: one barrier between writes and reads
          if (tid == 0) beta[(size_t)cur.f * bstride + d] = bn;
          feature_add(p, cur, Zs, tid, THREADS, cur.b - bn);
          cur = next;
        }
      }
      __syncthreads();
    }
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

// The same with the squares summed as recorded chains with a block-CG link had them: a warp per
// dimension, a lane's features in order, then a shuffle tree.
__global__ void __launch_bounds__(256)
    k_lambda_beta_ordered(const double* __restrict__ beta, int bstride, long long nfeat, int K,
                          double a0, double b0, const Ctl* ctl, unsigned long long seed, int mode,
                          double* __restrict__ lambda_beta) {
  const int lane = threadIdx.x & 31;
  for (int d = threadIdx.x >> 5; d < K; d += blockDim.x >> 5) {
    double s = 0.0;
#pragma unroll 4
    for (long long f = lane; f < nfeat; f += 32) {
      const double b = beta[f * bstride + d];
      s = fma(b, b, s);
    }
    s = warp_sum(s);
    if (lane == 0)
      lambda_beta[d] = gamma_draw(seed, ctl->sweep, stream_id(kLambdaBeta, (uint32_t)mode),
                                  (uint32_t)d, a0 + (double)nfeat / 2.0) *
                       (1.0 / (b0 + s / 2.0));
  }
}

template <typename T, bool BINARY, int THREADS, int NP>
void beta_smem(const DevCsr& Ft, const double* colsq, const int* lvl_ptr, const int* lvl_feat,
               const longlong2* lvl_range, const int* lvl_warp, int nlevels, const void* U,
               int ustride, const double* mu, const double* uhat, int hstride,
               const double* Lambda, const double* lambda_beta, int K, long long N, double* beta,
               int bstride, const double* draws, cudaStream_t s) {
  static bool configured[64] = {false};
  int dev = 0;
  MG_CUDA(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    MG_CUDA(cudaFuncSetAttribute(k_beta_one_smem<T, BINARY, THREADS, NP>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double) * kZsMax)));
    configured[dev & 63] = true;
  }
  k_beta_one_smem<T, BINARY, THREADS, NP><<<K, THREADS, sizeof(double) * (size_t)N, s>>>(
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
                     double* Z, int zstride, double* draws, bool ordered, const Ctl* ctl,
                     unsigned long long seed, int mode, cudaStream_t s) {
  const long long work = Ft.nrow * ((K + 1) / 2);
  k_beta_draws<<<(int)std::min<long long>(4736, (work + 255) / 256), 256, 0, s>>>(
      Ft.nrow, K, bstride, ctl, seed, mode, draws);
  MG_CUDA(cudaGetLastError());
  if (N <= kZsMax) {  // one block per dimension, Z's column in shared memory
    const auto pick = [&](auto u) {
      using T = decltype(u);
      if (ordered)
        return Ft.val ? beta_smem<T, false, kOrderedThreads, 1>
                      : beta_smem<T, true, kOrderedThreads, 1>;
      return Ft.val ? beta_smem<T, false, kSmemThreads, kNp> : beta_smem<T, true, kSmemThreads, kNp>;
    };
    const auto run = f32 ? pick(0.f) : pick(0.0);
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

// Orders the features by level and splits each level into at most three: the long features, each taken
// by the whole block in turn, the short ones, a lane each, and the others, a warp each.  The features
// of a level touch disjoint rows, so their order does not matter; who takes a feature decides the
// order in which its entries are added.  With Z in shared memory the block's share minimises the
// estimate: 700 cycles per feature of the block (two shuffle trees and a barrier), 600 per 16
// features of the warps plus 60 for every 32 entries of the longest one beyond the first 128.  Lanes
// take the features that have no more entries than a thread holds ahead, where two rounds of the
// warps or more are saved.  k_beta_one, and every chain with a block-CG link (`ordered`), gives a
// level to the warps unless it has few features and a long one.
void beta_one_levels(long long N, bool ordered, const std::vector<int>& level,
                     const std::vector<long long>& ptr, std::vector<int>& lvl_ptr,
                     std::vector<int>& order, std::vector<int>& lvl_warp) {
  const int nfeat = (int)level.size();
  auto len = [&](int f) { return ptr[f + 1] - ptr[f]; };
  order.resize(nfeat);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    return level[a] != level[b] ? level[a] < level[b] : len(a) > len(b);
  });
  lvl_ptr.assign(1, 0);
  lvl_warp.clear();
  for (int s = 0; s < nfeat;) {
    int e = s;
    while (e < nfeat && level[order[e]] == level[order[s]]) e++;
    const long long n = e - s, longest = len(order[s]);
    int cut = s;  // features s .. cut - 1 by the block
    if (ordered || N > kZsMax) {
      if (n < 8 && longest > 1024) cut = e;
    } else {
      long long best = -1;
      for (int c = s; c <= e && c <= s + 64; c++) {
        const long long rest = e - c, steps = rest ? (len(order[c]) + 31) / 32 : 0;
        const long long cost = 700 * (c - s) + (rest + kSmemWarps - 1) / kSmemWarps * 600 +
                               60 * std::max(0LL, steps - 4);
        if (best < 0 || cost < best) {
          best = cost;
          cut = c;
        }
      }
    }
    if (cut > s) {
      lvl_ptr.push_back(cut);
      lvl_warp.push_back(kByBlock);
    }
    // the shortest features of a wide level, whose entries a lane holds ahead
    int lanes = e;
    if (!ordered && N <= kZsMax)
      while (lanes > cut && len(order[lanes - 1]) <= kNp) lanes--;
    if (e - lanes < 2 * kSmemWarps) lanes = e;
    if (lanes > cut) {
      lvl_ptr.push_back(lanes);
      lvl_warp.push_back(kByWarp);
    }
    if (e > lanes) {
      lvl_ptr.push_back(e);
      lvl_warp.push_back(kByLane);
    }
    s = e;
  }
}

void launch_lambda_beta_one(const double* beta, int bstride, long long nfeat, int K, double a0,
                            double b0, const Ctl* ctl, unsigned long long seed, int mode,
                            bool ordered, double* parts, double* lambda_beta, cudaStream_t s) {
  if (ordered) {
    k_lambda_beta_ordered<<<1, 256, 0, s>>>(beta, bstride, nfeat, K, a0, b0, ctl, seed, mode,
                                            lambda_beta);
    MG_CUDA(cudaGetLastError());
    return;
  }
  // `parts` holds nfeat * bstride doubles: at most one record of K per 64 features is written
  const int nb = (int)std::min<long long>(148, (nfeat + 63) / 64);
  k_beta_sq<<<nb, kSqThreads, 0, s>>>(beta, bstride, nfeat, K, (nfeat + nb - 1) / nb, parts);
  MG_CUDA(cudaGetLastError());
  k_lambda_beta_one<<<1, 64, 0, s>>>(parts, nb, nfeat, K, a0, b0, ctl, seed, mode, lambda_beta);
  MG_CUDA(cudaGetLastError());
}

}  // namespace mg
