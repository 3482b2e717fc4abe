// Hyperprior statistics, noise update and test-set evaluation.
//
//   k_stats32         per-block partial sums of x and x x^T over the rows of a latent matrix, K <=
//                     32 (optionally x = U - Uhat, the Macau residual of latentprior.cpp:257);
//                     FP64 accumulation from FP64 or FP32 latents on the FP64 matrix instruction.
//   (K > 32, and the Normal-Wishart draw: hyper_wide.cu)
//   k_lambda_beta     one CTA: posterior_lambda_beta + rgamma (latentprior.cpp:317-331).
//   k_eval / k_eval_finish  eval_rmse (bpmfutils.h:86-114): online posterior mean / variance of
//                     the test predictions and the two RMSEs.
#include "common.cuh"
#include "kernels.h"
#include "mma_tiles.cuh"
#include "rng.cuh"
#include "warp_finish.cuh"

namespace mg {
namespace {

constexpr int kStatThreads = 256;

// lambda_beta ~ Gamma(nux/2, 2 mux/nux), nux = nu + K nfeat,
// mux = mu nux / (nu + mu tr(B B^T Lambda))   (latentprior.cpp:317-331)
__global__ void k_lambda_beta(const double* __restrict__ bb_partials, int nparts, int K,
                              long long nfeat, const double* __restrict__ Lambda, double nu,
                              double mu, const Ctl* ctl, unsigned long long seed, int mode,
                              double* lambda_beta) {
  __shared__ double red[256];
  const int KK = K * K;
  double tr = 0.0;
  for (int e = threadIdx.x; e < KK; e += blockDim.x) {
    double s = 0.0;
    for (int b = 0; b < nparts; b++) s += bb_partials[(size_t)b * (K + KK) + K + e];
    const int i = e % K, j = e / K;
    tr += s * Lambda[j + i * K];
  }
  red[threadIdx.x] = tr;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < (int)blockDim.x; q++) t += red[q];
    const double nux = nu + (double)K * (double)nfeat;
    const double mux = mu * nux / (nu + mu * t);
    const double b = nux / 2, c = 2 * mux / nux;
    *lambda_beta = c * gamma_draw(seed, ctl->sweep, stream_id(kLambdaBeta, mode), 0u, b);
  }
}

constexpr int kEvalThreads = 256;

// Dots of eight consecutive entries by a group of eight lanes: entry j of the group has the rows
// (r, c) of its lane j; the lanes read its two latent rows with vector loads (lane l: elements
// 4l .. 4l + 3, + 32 i), four entries' loads in flight, and the 8 x 8 partial sums are transposed and
// added in three exchange steps (7 shuffles instead of 24).  Returns the dot of the lane's entry.
template <typename T>
__device__ __forceinline__ double dot4(const T* u, const T* v) {
  if constexpr (sizeof(T) == 4) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(u));
    const float4 b = __ldg(reinterpret_cast<const float4*>(v));
    return (double)a.x * (double)b.x + (double)a.y * (double)b.y + (double)a.z * (double)b.z +
           (double)a.w * (double)b.w;
  } else {
    const double2 a0 = __ldg(reinterpret_cast<const double2*>(u));
    const double2 a1 = __ldg(reinterpret_cast<const double2*>(u + 2));
    const double2 b0 = __ldg(reinterpret_cast<const double2*>(v));
    const double2 b1 = __ldg(reinterpret_cast<const double2*>(v + 2));
    return a0.x * b0.x + a0.y * b0.y + a1.x * b1.x + a1.y * b1.y;
  }
}
template <typename T>
__device__ __forceinline__ double group_dots(const T* __restrict__ U, const T* __restrict__ V,
                                             int stride, int K, int r, int c, int l, unsigned mask) {
  double d[8];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const T *u[4], *v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      u[j] = U + (size_t)__shfl_sync(mask, r, 4 * h + j, 8) * stride + 4 * l;
      v[j] = V + (size_t)__shfl_sync(mask, c, 4 * h + j, 8) * stride + 4 * l;
      d[4 * h + j] = 0.0;
    }
    for (int k0 = 4 * l; k0 < K; k0 += 32)
#pragma unroll
      for (int j = 0; j < 4; j++) d[4 * h + j] += dot4<T>(u[j] + (k0 - 4 * l), v[j] + (k0 - 4 * l));
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1)
#pragma unroll
    for (int j = 0; j < o; j++) {
      const bool hi = (l & o) != 0;
      const double keep = hi ? d[j + o] : d[j], send = hi ? d[j] : d[j + o];
      d[j] = keep + __shfl_xor_sync(mask, send, o);
    }
  return d[0];
}

// Online mean / variance update of eval_rmse (bpmfutils.h:86-114): each lane keeps the entry whose
// dot it holds, so the updates and their pred / pvar / value accesses run on all eight lanes.  Per
// block, the squared errors are summed in lane and group order into partials[2 * block .. + 1].
//   What bounds it: the gathers of the latent rows from L2.  The test arrays are read and written
//   once a sweep, past the caches (ld.cs, st.cs): at 2M entries their 96 MB would push the latents
//   and the samplers' entries out of L2, which cost the sweep more (160 us mixed, 257 us FP64 at
//   K = 32) than this kernel takes.
template <typename T>
__global__ void __launch_bounds__(kEvalThreads)
    k_eval(const int* __restrict__ trow, const int* __restrict__ tcol,
           const double* __restrict__ tval, long long ntest, const T* __restrict__ U,
           const T* __restrict__ V, int K, int stride, double mean, int n_fixed, const Ctl* ctl,
           double* __restrict__ pred, double* __restrict__ pvar, double* __restrict__ partials) {
  constexpr int kGroups = kEvalThreads / 8;
  __shared__ double r1[kGroups], r2[kGroups];
  int n = n_fixed;
  if (n < 0) n = ((int)ctl->sweep < ctl->burnin) ? 0 : (int)ctl->sweep - ctl->burnin;
  const int g = threadIdx.x >> 3, l = threadIdx.x & 7;
  const unsigned mask = 0xffu << (8 * ((threadIdx.x & 31) >> 3));
  double se = 0.0, sea = 0.0;
  const long long step = (long long)gridDim.x * kGroups * 8;
  const bool first = n == 0;
  // the next step's entry is loaded while this one's rows are gathered
  int r = 0, c = 0;
  double y = 0.0, old = 0.0, oldv = 0.0;
  auto fetch = [&](long long t) {
    const bool own = t < ntest;
    r = own ? __ldcs(trow + t) : 0;
    c = own ? __ldcs(tcol + t) : 0;
    y = own ? __ldcs(tval + t) : 0.0;
    old = own && !first ? __ldcs(pred + t) : 0.0;
    oldv = own && !first ? __ldcs(pvar + t) : 0.0;
  };
  long long t0 = ((long long)blockIdx.x * kGroups + g) * 8;
  if (t0 < ntest) fetch(t0 + l);
  for (; t0 < ntest; t0 += step) {
    const long long t = t0 + l;  // this lane's entry
    const int r_t = r, c_t = c;
    const double y_t = y, old_t = old, oldv_t = oldv;
    if (t0 + step < ntest) fetch(t + step);
    const double mydot = group_dots<T>(U, V, stride, K, r_t, c_t, l, mask);
    if (t < ntest) {
      const double p = mydot + mean;
      se += (y_t - p) * (y_t - p);
      double pavg;
      if (first) {
        pavg = p;
      } else {
        const double delta = p - old_t;
        pavg = old_t + delta / (n + 1);
        __stcs(pvar + t, oldv_t + delta * (p - pavg));
      }
      sea += (y_t - pavg) * (y_t - pavg);
      __stcs(pred + t, pavg);
    }
  }
  // group sums in lane order
#pragma unroll
  for (int q = 1; q < 8; q++) {
    const double a1 = __shfl_sync(mask, se, q, 8), b1 = __shfl_sync(mask, sea, q, 8);
    if (l == 0) {
      se += a1;
      sea += b1;
    }
  }
  if (l == 0) {
    r1[g] = se;
    r2[g] = sea;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int q = 0; q < kGroups; q++) {
      a += r1[q];
      b += r2[q];
    }
    partials[2 * blockIdx.x] = a;
    partials[2 * blockIdx.x + 1] = b;
  }
}

// One warp: lane q sums partials q, q + 32, ... in order, then a fixed shuffle tree.
__global__ void k_eval_finish(const double* partials, int nparts, long long ntest,
                              double* rmse) {
  const int lane = threadIdx.x & 31;
  double a = 0.0, b = 0.0;
  for (int q = lane; q < nparts; q += 32) {
    a += partials[2 * q];
    b += partials[2 * q + 1];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if (lane == 0) {
    rmse[0] = sqrt(b / (double)ntest);  // posterior-mean RMSE (rmse_test)
    rmse[1] = sqrt(a / (double)ntest);  // single-sample RMSE (rmse_test_onesample)
  }
}

// Row of every CSR entry (the inverse of the row pointers): entry e lies in the row r with
// ptr[r] <= e < ptr[r + 1], found by binary search so that heavy rows cost no more than others.
__global__ void k_entry_rows(const long long* __restrict__ ptr, long long nrows, long long nnz,
                             int* __restrict__ erow) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += stride) {
    long long lo = 0, hi = nrows;  // invariant: ptr[lo] <= e < ptr[hi]
    while (hi - lo > 1) {
      const long long mid = (lo + hi) >> 1;
      if (ptr[mid] <= e) lo = mid;
      else hi = mid;
    }
    erow[e] = (int)lo;
  }
}

// Squared training residuals of AdaptiveGaussianNoise::update (noisemodels.cpp:55-72):
// (U_i . V_j + mean - y)^2 over the entries (i = erow[e], j = col[e], y = val[e]).  Same
// group layout as k_eval, lane l keeps entry t0 + l; the per-block sum goes to partials[block] in lane and
// group order.
template <typename T>
__global__ void __launch_bounds__(kEvalThreads)
    k_noise_sse(const int* __restrict__ erow, const int* __restrict__ col,
                const double* __restrict__ val, long long nnz, const T* __restrict__ U,
                const T* __restrict__ V, int K, int stride, double mean,
                double* __restrict__ partials) {
  constexpr int kGroups = kEvalThreads / 8;
  __shared__ double r1[kGroups];
  const int g = threadIdx.x >> 3, l = threadIdx.x & 7;
  const unsigned mask = 0xffu << (8 * ((threadIdx.x & 31) >> 3));
  double se = 0.0;
  const long long step = (long long)gridDim.x * kGroups * 8;
  // the next step's entry is loaded while this one's rows are gathered
  int r = 0, c = 0;
  double y = 0.0;
  auto fetch = [&](long long t) {
    const bool own = t < nnz;
    r = own ? __ldcs(erow + t) : 0;
    c = own ? __ldcs(col + t) : 0;
    y = own ? __ldcs(val + t) : 0.0;
  };
  long long t0 = ((long long)blockIdx.x * kGroups + g) * 8;
  if (t0 < nnz) fetch(t0 + l);
  for (; t0 < nnz; t0 += step) {
    const int r_t = r, c_t = c;
    const double y_t = y;
    if (t0 + step < nnz) fetch(t0 + step + l);
    const double mydot = group_dots<T>(U, V, stride, K, r_t, c_t, l, mask);
    if (t0 + l < nnz) {
      const double d = (mydot + mean) - y_t;
      se += d * d;
    }
  }
#pragma unroll
  for (int q = 1; q < 8; q++) {
    const double a1 = __shfl_sync(mask, se, q, 8);
    if (l == 0) se += a1;
  }
  if (l == 0) r1[g] = se;
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0;
    for (int q = 0; q < kGroups; q++) a += r1[q];
    partials[blockIdx.x] = a;
  }
}

// The precision draw of AdaptiveGaussianNoise::update (noisemodels.cpp:73-81), one warp: the
// partial sums in a fixed order, then aN = a0 + nnz / 2, bN = b0 + sumsq / 2 with
// (a0, b0) = (1/2, var_total / 2), alpha = Gamma(aN, 1) / bN capped at alpha_max, into ctl->alpha.
__global__ void k_noise_draw(const double* __restrict__ partials, int nparts, long long nnz,
                             double var_total, double alpha_max, Ctl* ctl,
                             unsigned long long seed) {
  const int lane = threadIdx.x & 31;
  double a = 0.0;
  for (int q = lane; q < nparts; q += 32) a += partials[q];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if (lane == 0) {
    const double aN = 0.5 + (double)nnz / 2.0;
    const double bN = 0.5 * var_total + a / 2.0;
    double alpha = gamma_draw(seed, ctl->sweep, stream_id(kNoiseAlpha, 0u), 0u, aN) * (1.0 / bN);
    if (alpha > alpha_max) alpha = alpha_max;
    ctl->alpha = alpha;
  }
}

__global__ void k_set_sweep(Ctl* ctl, uint32_t sweep, int burnin) {
  ctl->sweep = sweep;
  ctl->burnin = burnin;
}

__global__ void k_advance(Ctl* ctl) { ctl->sweep += 1u; }

// One block's statistics (column sums and outer-product sums) over rows r0 .. r1 - 1 of (U - Uhat),
// K <= 8 NB, into out[0 .. K + K*K) (k_stats32 and k_stats32_pair).  Warp
// w takes the four rows 4 (w + 8 i) .. of the block, lane (g, t) = (lane / 4, lane % 4) component
// 8 b + g of row t, which is the operand element of block b on either side of m8n8k4.f64: the
// lower-triangle tiles take NB (NB + 1) / 2 matrix instructions per four rows, on operands loaded
// straight from memory three steps ahead.  The warps' tiles are added in warp order.
//   What bounds it: latency; 4 x 4 DFMA tiles over rows staged in shared memory took 42 us for both
//   modes of 138,000 x 27,000 at K = 32, this 17.
constexpr int kStatWarps = kStatThreads / 32;
template <typename T, int NB>
__device__ __forceinline__ void stats32_blocks(const T* __restrict__ U,
                                               const double* __restrict__ Uhat, long long r0,
                                               long long r1, int K, int stride, int uhat_stride,
                                               double* __restrict__ out, double* buf) {
  constexpr int TILES = NB * (NB + 1) / 2, R = 4, REC = TILES * 64 + 8 * NB;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double acc[TILES][2], su[NB], f[R][NB];
#pragma unroll
  for (int q = 0; q < TILES; q++) acc[q][0] = acc[q][1] = 0.0;
#pragma unroll
  for (int b = 0; b < NB; b++) su[b] = 0.0;
  auto load = [&](int stage, long long row) {
    const T* u = U + row * stride + g;
#pragma unroll
    for (int b = 0; b < NB; b++) {
      const bool ok = row < r1 && 8 * b + g < K;
      double x = ok ? (double)__ldg(u + 8 * b) : 0.0;
      if (Uhat) x -= ok ? __ldg(Uhat + row * uhat_stride + g + 8 * b) : 0.0;
      f[stage][b] = x;
    }
  };
  const long long first = r0 + 4 * warp + t;
  constexpr int STEP = 4 * kStatWarps;
#pragma unroll
  for (int u = 0; u < R - 1; u++) load(u, first + STEP * u);
  for (long long r = first - t; r < r1; r += R * STEP) {
#pragma unroll
    for (int u = 0; u < R; u++) {
      load((u + R - 1) % R, r + t + STEP * (u + R - 1));
      int q = 0;
#pragma unroll
      for (int a = 0; a < NB; a++) {
        su[a] += f[u][a];
#pragma unroll
        for (int b = 0; b <= a; b++) {
          mma_f64(acc[q][0], acc[q][1], f[u][a], f[u][b]);
          q++;
        }
      }
    }
  }
  double* mine = buf + warp * REC;
#pragma unroll
  for (int q = 0; q < TILES; q++)
    *reinterpret_cast<double2*>(mine + q * 64 + g * 8 + 2 * t) = make_double2(acc[q][0], acc[q][1]);
#pragma unroll
  for (int b = 0; b < NB; b++) {
    su[b] += __shfl_xor_sync(0xffffffffu, su[b], 1);
    su[b] += __shfl_xor_sync(0xffffffffu, su[b], 2);
    if (t == 0) mine[TILES * 64 + 8 * b + g] = su[b];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < REC; e += kStatThreads) {
    double v = buf[e];
#pragma unroll
    for (int w = 1; w < kStatWarps; w++) v += buf[w * REC + e];
    if (e >= TILES * 64) {
      if (e - TILES * 64 < K) out[e - TILES * 64] = v;
      continue;
    }
    int a = 0;
    while ((a + 1) * (a + 2) / 2 <= (e >> 6)) a++;
    const int b = (e >> 6) - a * (a + 1) / 2;
    const int i = 8 * a + ((e >> 3) & 7), j = 8 * b + (e & 7);
    if (i < K && j < K) {
      out[K + i + j * K] = v;
      if (a != b) out[K + j + i * K] = v;
    }
  }
}

template <typename T>
__device__ __forceinline__ void stats32_rows(const T* __restrict__ U,
                                             const double* __restrict__ Uhat, long long r0,
                                             long long r1, int K, int stride, int uhat_stride,
                                             double* __restrict__ out) {
  __shared__ __align__(16) double buf[kStatWarps * (10 * 64 + 32)];
  if (K <= 8) stats32_blocks<T, 1>(U, Uhat, r0, r1, K, stride, uhat_stride, out, buf);
  else if (K <= 16) stats32_blocks<T, 2>(U, Uhat, r0, r1, K, stride, uhat_stride, out, buf);
  else if (K <= 24) stats32_blocks<T, 3>(U, Uhat, r0, r1, K, stride, uhat_stride, out, buf);
  else stats32_blocks<T, 4>(U, Uhat, r0, r1, K, stride, uhat_stride, out, buf);
}

template <typename T>
__global__ void __launch_bounds__(kStatThreads)
    k_stats32(const T* __restrict__ U, const double* __restrict__ Uhat, long long N, int K,
              int stride, int uhat_stride, long long rows_per_block, double* __restrict__ partials) {
  const long long r0 = (long long)blockIdx.x * rows_per_block;
  stats32_rows(U, Uhat, r0, min(N, r0 + rows_per_block), K, stride, uhat_stride,
               partials + (size_t)blockIdx.x * (K + K * K));
}

// Sums `nparts` partial records of `len` doubles in a fixed order: CTA c owns elements
// 32 c .. 32 c + 31; warp w adds partials w, w + 8, ... in order, then the 8 warp sums are added
// in warp order.  out = one record.
__global__ void __launch_bounds__(256)
    k_reduce_parts(const double* __restrict__ parts, int nparts, int len, double* __restrict__ out) {
  __shared__ double ws[8][33];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int e = blockIdx.x * 32 + lane;
  double s = 0.0;
  if (e < len) {
#pragma unroll 8
    for (int b = warp; b < nparts; b += 8) s += parts[(size_t)b * len + e];
  }
  ws[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && e < len) {
    double t = ws[0][lane];
#pragma unroll
    for (int w = 1; w < 8; w++) t += ws[w][lane];
    out[e] = t;
  }
}

// ---- both modes' BPMF prior updates in one launch per step: blocks of mode 0, then
// of mode 1, each doing what the single-mode kernel's block does, so the results are the same
// bit for bit; the two modes' steps only overlap ----
template <typename T>
__global__ void __launch_bounds__(kStatThreads)
    k_stats32_pair(PriorPair pp, int K, int stride) {
  const int m = blockIdx.x < pp.nblocks[0] ? 0 : 1;
  const int b = blockIdx.x - (m ? pp.nblocks[0] : 0);
  const long long r0 = (long long)b * pp.rows_per_block[m];
  stats32_rows(static_cast<const T*>(pp.U[m]), nullptr, r0, min(pp.N[m], r0 + pp.rows_per_block[m]),
               K, stride, 0, pp.partials[m] + (size_t)b * (K + K * K));
}

__global__ void __launch_bounds__(256) k_reduce_parts_pair(PriorPair pp, int len) {
  __shared__ double ws[8][33];
  const int nblk = (len + 31) / 32;
  const int m = blockIdx.x < nblk ? 0 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int e = (blockIdx.x - (m ? nblk : 0)) * 32 + lane;
  const double* parts = pp.partials[m];
  const int nparts = pp.nblocks[m];
  double s = 0.0;
  if (e < len) {
#pragma unroll 8
    for (int b = warp; b < nparts; b += 8) s += parts[(size_t)b * len + e];
  }
  ws[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && e < len) {
    double t = ws[0][lane];
#pragma unroll
    for (int w = 1; w < 8; w++) t += ws[w][lane];
    pp.final_[m][e] = t;
  }
}

}  // namespace

int launch_prior_pair(const PriorPair& pp, bool f32, int K, int stride, Ctl* ctl,
                       unsigned long long seed, cudaStream_t s) {
  const int nb = pp.nblocks[0] + pp.nblocks[1];
  if (K > 32)
    launch_stats_wide_pair(pp, f32, K, stride, s);
  else if (f32)
    k_stats32_pair<float><<<nb, kStatThreads, 0, s>>>(pp, K, stride);
  else
    k_stats32_pair<double><<<nb, kStatThreads, 0, s>>>(pp, K, stride);
  MG_CUDA(cudaGetLastError());
  const bool few = few_parts(pp.nblocks[0], K) && few_parts(pp.nblocks[1], K);
  if (!few) {
    const int len = K + K * K;
    k_reduce_parts_pair<<<2 * ((len + 31) / 32), 256, 0, s>>>(pp, len);
    MG_CUDA(cudaGetLastError());
  }
  launch_normal_wishart_pair(pp, K, ctl, seed, s);
  return few ? 2 : 3;
}

// Up to 16 partials are added by the Normal-Wishart block itself: one CTA reads them in less time
// than the reduction's launch takes (2,000 + 1,500 rows, 28 partials in all: a sweep of 47 us lost
// 3 us).  With more its reads cost what the launch does up to about 40 and more beyond (64 partials, a
// call of mg_normal_wishart_noalloc: 50.8 us and 47.3 reduced first at K = 16, 63.5 and 55.3 at K = 32).
bool few_parts(int nblocks, int K) { return K <= 32 && nblocks <= 16; }

int stats_blocks(long long N) {  // at most two blocks per SM: fewer partials to reduce
  long long b = (N + 127) / 128;
  if (b > 296) b = 296;
  return (int)(b < 1 ? 1 : b);
}

void launch_stats(const void* U, bool f32, const double* Uhat, long long N, int K, int stride,
                  int uhat_stride, double* partials, int nblocks, cudaStream_t s) {
  if (K > 128) throw MgError(MG_ERR_ARG, "K > 128 is not supported");
  const long long rpb = (N + nblocks - 1) / nblocks;
  if (K <= 32) {
    if (f32)
      k_stats32<float><<<nblocks, kStatThreads, 0, s>>>((const float*)U, Uhat, N, K, stride,
                                                        uhat_stride, rpb, partials);
    else
      k_stats32<double><<<nblocks, kStatThreads, 0, s>>>((const double*)U, Uhat, N, K, stride,
                                                         uhat_stride, rpb, partials);
    MG_CUDA(cudaGetLastError());
    return;
  }
  launch_stats_wide(U, f32, Uhat, N, K, stride, uhat_stride, partials, nblocks, s);
}

void launch_reduce_parts(const double* parts, int nparts, int len, double* out, cudaStream_t s) {
  k_reduce_parts<<<(len + 31) / 32, 256, 0, s>>>(parts, nparts, len, out);
  MG_CUDA(cudaGetLastError());
}

void launch_lambda_beta(const double* bb_partials, int nparts, int K, long long nfeat,
                        const double* Lambda, double nu, double mu, const Ctl* ctl,
                        unsigned long long seed, int mode, double* lambda_beta, cudaStream_t s) {
  k_lambda_beta<<<1, 256, 0, s>>>(bb_partials, nparts, K, nfeat, Lambda, nu, mu, ctl, seed,
                                  mode, lambda_beta);
  MG_CUDA(cudaGetLastError());
}

int eval_blocks(long long ntest) {
  long long b = (ntest + kEvalThreads - 1) / kEvalThreads;
  if (b > 1184) b = 1184;
  return (int)(b < 1 ? 1 : b);
}

void launch_eval(const int* trow, const int* tcol, const double* tval, long long ntest,
                 const void* U, const void* V, bool f32, int K, int stride, double mean,
                 int n_fixed, const Ctl* ctl, double* pred, double* pvar, double* partials,
                 int nblocks, double* rmse, cudaStream_t s) {
  if (f32)
    k_eval<float><<<nblocks, kEvalThreads, 0, s>>>(trow, tcol, tval, ntest, (const float*)U,
                                                   (const float*)V, K, stride, mean, n_fixed,
                                                   ctl, pred, pvar, partials);
  else
    k_eval<double><<<nblocks, kEvalThreads, 0, s>>>(trow, tcol, tval, ntest, (const double*)U,
                                                    (const double*)V, K, stride, mean, n_fixed,
                                                    ctl, pred, pvar, partials);
  MG_CUDA(cudaGetLastError());
  k_eval_finish<<<1, 32, 0, s>>>(partials, nblocks, ntest, rmse);
  MG_CUDA(cudaGetLastError());
}

void launch_entry_rows(const long long* ptr, long long nrows, long long nnz, int* erow,
                       cudaStream_t s) {
  if (nnz <= 0) return;
  long long b = (nnz + 255) / 256;
  if (b > 4736) b = 4736;
  k_entry_rows<<<(int)b, 256, 0, s>>>(ptr, nrows, nnz, erow);
  MG_CUDA(cudaGetLastError());
}

void launch_noise_update(const int* erow, const int* col, const double* val, long long nnz,
                         const void* U, const void* V, bool f32, int K, int stride, double mean,
                         double var_total, double alpha_max, double* partials, int nblocks,
                         Ctl* ctl, unsigned long long seed, cudaStream_t s) {
  if (f32)
    k_noise_sse<float><<<nblocks, kEvalThreads, 0, s>>>(erow, col, val, nnz, (const float*)U,
                                                        (const float*)V, K, stride, mean,
                                                        partials);
  else
    k_noise_sse<double><<<nblocks, kEvalThreads, 0, s>>>(erow, col, val, nnz, (const double*)U,
                                                         (const double*)V, K, stride, mean,
                                                         partials);
  MG_CUDA(cudaGetLastError());
  k_noise_draw<<<1, 32, 0, s>>>(partials, nblocks, nnz, var_total, alpha_max, ctl, seed);
  MG_CUDA(cudaGetLastError());
}

void launch_set_sweep(Ctl* ctl, uint32_t sweep, int burnin, cudaStream_t s) {
  k_set_sweep<<<1, 1, 0, s>>>(ctl, sweep, burnin);
  MG_CUDA(cudaGetLastError());
}

void launch_advance(Ctl* ctl, cudaStream_t s) {
  k_advance<<<1, 1, 0, s>>>(ctl);
  MG_CUDA(cudaGetLastError());
}

}  // namespace mg
