// Block-CG iteration (solve_blockcg, linop.h:229-343) for up to 32 right-hand sides, its K x K work on
// the FP64 matrix instruction m8n8k4.f64 over 8 x 8 tiles.
//
// Per iteration, after the two SpMMs (cg_kernels.cu):
//   k_cg_outer   partial sums of P KP^T (lower-triangle tiles), rows straight into fragments
//   k_cg_solve   one CTA: A = (chol(P^T K P) \ R^T R)^T
//   k_cg_update  X += A P, R -= A KP, and the partial sums of R R^T of the new R
//   k_cg_solve   convergence test, Psi = (chol(R^T R) \ R2^T R2)^T
//   k_cg_pupdate P = R + Psi P
// The partial sums are reduced over clusters of 8 CTAs through distributed shared memory, in rank
// order, so that a solve reads at most 18 records and no launch only adds records.
//
// What bounds it: the small solves, whose chains run on one SM while the rest of the GPU waits, and
// the memory passes over X, R, P and KP (8.4 MB each at 32,768 features, from L2).  With DFMA
// tiles in shared memory and one warp per right-hand side in the solves an iteration took 28 + 8
// us for the two outer products and their sums, 29 + 31 us for the solves and 25 + 13 us for the row
// updates at 32,768 features and 32 right-hand sides.
#include <cooperative_groups.h>

#include <cmath>

#include "cg_small.cuh"
#include "common.cuh"
#include "kernels.h"
#include "wide_tiles.cuh"

namespace mg {
namespace {

namespace cg = cooperative_groups;

constexpr int kN = 32, kB = kN / 8, kTri = kB * (kB + 1) / 2;  // padded width, blocks, tiles
constexpr int kRecord = kTri * 64;  // lower-triangle tiles, row-major inside a tile
constexpr int kThreads = 256, kWarps = kThreads / 32, kCluster = 8;
constexpr int kMaxClusters = 18;    // 144 of the 148 SMs

// Entry (i, j), i >= j, of a record.
__device__ __forceinline__ int rec_at(int i, int j) {
  return ((i >> 3) * ((i >> 3) + 1) / 2 + (j >> 3)) * 64 + (i & 7) * 8 + (j & 7);
}

// Sum of `n` records' entry e in order.
__device__ __forceinline__ double sum_rec(const double* __restrict__ recs, int n, int e) {
  double s = 0.0;
#pragma unroll 6
  for (int r = 0; r < n; r++) s += __ldcg(recs + (size_t)r * kRecord + e);
  return s;
}

// The block's tiles (acc of each warp) -> one record per cluster: warps in order, then the cluster's
// CTAs in rank order.  buf: kWarps * kRecord doubles of shared memory.
__device__ __forceinline__ void reduce_record(const double (&acc)[kTri][2], double* buf,
                                              double* __restrict__ recs) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int q = 0; q < kTri; q++)
    *reinterpret_cast<double2*>(buf + warp * kRecord + q * 64 + g * 8 + 2 * t) =
        make_double2(acc[q][0], acc[q][1]);
  __syncthreads();
  for (int e = threadIdx.x; e < kRecord; e += kThreads) {
    double s = buf[e];
#pragma unroll
    for (int w = 1; w < kWarps; w++) s += buf[w * kRecord + e];
    buf[e] = s;  // only this thread reads or writes column e
  }
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  constexpr int kSlice = kRecord / kCluster;
  const int rank = (int)cl.block_rank();
  if (threadIdx.x < kSlice) {
    const int e = rank * kSlice + threadIdx.x;
    double s = 0.0;
#pragma unroll
    for (int r = 0; r < kCluster; r++) s += cl.map_shared_rank(buf, r)[e];
    recs[(size_t)(blockIdx.x / kCluster) * kRecord + e] = s;
  }
  cl.sync();  // no CTA leaves while its shared memory is read
}

// Rows of a warp: an equal share of the row groups of `step` rows, contiguous.
__device__ __forceinline__ void warp_rows(long long nrow, int step, long long& r0, long long& r1) {
  const long long nw = (long long)gridDim.x * kWarps;
  const long long w = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
  const long long groups = (nrow + step - 1) / step, per = (groups + nw - 1) / nw;
  r0 = min(nrow, w * per * step);
  r1 = min(nrow, (w + 1) * per * step);
}

// Partial sums of A B^T over the features (rows of kN values): tiles (bi, bj), bj <= bi.
template <typename V>
__global__ void __launch_bounds__(kThreads) __cluster_dims__(kCluster, 1, 1)
    k_cg_outer(const V* __restrict__ A, const V* __restrict__ B, long long nfeat,
               double* __restrict__ recs, const uint32_t* __restrict__ done) {
  if (done && *done) return;
  extern __shared__ __align__(16) double buf[];
  constexpr int R = 4;  // steps of four rows in flight
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  long long r0, r1;
  warp_rows(nfeat, 4, r0, r1);
  double acc[kTri][2], a[R][kB], b[R][kB];
#pragma unroll
  for (int q = 0; q < kTri; q++) acc[q][0] = acc[q][1] = 0.0;
  const bool same = A == B;
  auto load = [&](int stage, long long row) {
    const bool ok = row < r1;
#pragma unroll
    for (int k = 0; k < kB; k++) {
      a[stage][k] = ok ? (double)A[row * kN + 8 * k + g] : 0.0;
      b[stage][k] = same ? a[stage][k] : (ok ? (double)B[row * kN + 8 * k + g] : 0.0);
    }
  };
#pragma unroll
  for (int u = 0; u < R - 1; u++) load(u, r0 + 4 * u + t);
  for (long long r = r0; r < r1; r += 4 * R) {
#pragma unroll
    for (int u = 0; u < R; u++) {
      load((u + R - 1) % R, r + 4 * (u + R - 1) + t);
      int q = 0;
#pragma unroll
      for (int bi = 0; bi < kB; bi++)
#pragma unroll
        for (int bj = 0; bj <= bi; bj++) {
          mma_f64(acc[q][0], acc[q][1], a[u][bi], b[u][bj]);
          q++;
        }
    }
  }
  reduce_record(acc, buf, recs);
}

// B operand fragments of M^T, M the n x n matrix at m (leading dimension 64): fragment (bk, h) of
// column block bn is M(8 bn + g, 8 bk + 2t + h), matching rows read two values a lane.
__device__ __forceinline__ void load_bfrag(double (&f)[kB][kB][2], const double* m, int n, int g,
                                           int t) {
#pragma unroll
  for (int bn = 0; bn < kB; bn++)
#pragma unroll
    for (int bk = 0; bk < kB; bk++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int i = 8 * bn + g, k = 8 * bk + 2 * t + h;
        f[bn][bk][h] = i < n && k < n ? m[i + k * 64] : 0.0;
      }
}
template <typename V>
__device__ __forceinline__ double2 load2(const V* p) {
  if constexpr (sizeof(V) == 8) {
    return *reinterpret_cast<const double2*>(p);
  } else {
    const float2 v = *reinterpret_cast<const float2*>(p);
    return make_double2((double)v.x, (double)v.y);
  }
}
__device__ __forceinline__ void store2(double* p, double2 v) { *reinterpret_cast<double2*>(p) = v; }
__device__ __forceinline__ void store2(float* p, double2 v) {
  *reinterpret_cast<float2*>(p) = make_float2((float)v.x, (float)v.y);
}

// X[f] += A P[f], R[f] -= A KP[f] (linop.h:292-300), eight features a warp at a time, and the
// partial sums of R R^T of the new R unless recs is null.
template <typename V>
__global__ void __launch_bounds__(kThreads) __cluster_dims__(kCluster, 1, 1)
    k_cg_update(long long nfeat, int n, const double* small, const V* __restrict__ P,
                const V* __restrict__ KPm, V* __restrict__ R, double* __restrict__ X,
                double* __restrict__ recs, const uint32_t* __restrict__ done) {
  if (*done) return;
  extern __shared__ __align__(16) double buf[];
  constexpr int LD = kN + 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double* tile = buf + (size_t)warp * 8 * LD;  // the warp's eight new rows of R
  SmallView v(const_cast<double*>(small));
  double f[kB][kB][2], acc[kTri][2];
  load_bfrag(f, v.A, n, g, t);
#pragma unroll
  for (int q = 0; q < kTri; q++) acc[q][0] = acc[q][1] = 0.0;
  long long r0, r1;
  warp_rows(nfeat, 8, r0, r1);
  for (long long r = r0; r < r1; r += 8) {
    const long long row = r + g;
    const bool ok = row < r1;
    const size_t at = (size_t)(ok ? row : r) * kN;
    double2 p[kB], k[kB], x[kB], y[kB];
#pragma unroll
    for (int b = 0; b < kB; b++) {
      p[b] = load2(P + at + 8 * b + 2 * t);
      k[b] = load2(KPm + at + 8 * b + 2 * t);
      x[b] = load2(X + at + 8 * b + 2 * t);
      y[b] = load2(R + at + 8 * b + 2 * t);
      // KP's components from n on are never written; P's are zero
      if (8 * b + 2 * t >= n) k[b].x = 0.0;
      if (8 * b + 2 * t + 1 >= n) k[b].y = 0.0;
    }
#pragma unroll
    for (int bk = 0; bk < kB; bk++)
#pragma unroll
      for (int bn = 0; bn < kB; bn++) {
        mma_f64(x[bn].x, x[bn].y, p[bk].x, f[bn][bk][0]);
        mma_f64(y[bn].x, y[bn].y, -k[bk].x, f[bn][bk][0]);
        mma_f64(x[bn].x, x[bn].y, p[bk].y, f[bn][bk][1]);
        mma_f64(y[bn].x, y[bn].y, -k[bk].y, f[bn][bk][1]);
      }
    __syncwarp();
#pragma unroll
    for (int b = 0; b < kB; b++) {
      if constexpr (sizeof(V) == 4) y[b] = make_double2((double)(float)y[b].x, (double)(float)y[b].y);
      if (ok) {
        store2(X + at + 8 * b + 2 * t, x[b]);
        store2(R + at + 8 * b + 2 * t, y[b]);
      }
      store2(tile + g * LD + 8 * b + 2 * t, ok ? y[b] : make_double2(0.0, 0.0));
    }
    __syncwarp();
    if (recs) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        double a[kB];
#pragma unroll
        for (int b = 0; b < kB; b++) a[b] = tile[(t + 4 * h) * LD + 8 * b + g];
        int q = 0;
#pragma unroll
        for (int bi = 0; bi < kB; bi++)
#pragma unroll
          for (int bj = 0; bj <= bi; bj++) {
            mma_f64(acc[q][0], acc[q][1], a[bi], a[bj]);
            q++;
          }
      }
    }
  }
  if (!recs) return;
  __syncthreads();  // the warps' row tiles share the buffer
  reduce_record(acc, buf, recs);
}

// P[f] = R[f] + Psi P[f] (linop.h:319-326).
template <typename V>
__global__ void __launch_bounds__(kThreads)
    k_cg_pupdate(long long nfeat, int n, const double* small, const V* __restrict__ R,
                 V* __restrict__ P, const uint32_t* __restrict__ done) {
  if (*done) return;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  SmallView v(const_cast<double*>(small));
  double f[kB][kB][2];
  load_bfrag(f, v.Psi, n, g, t);
  long long r0, r1;
  warp_rows(nfeat, 8, r0, r1);
  for (long long r = r0; r < r1; r += 8) {
    const long long row = r + g;
    const bool ok = row < r1;
    const size_t at = (size_t)(ok ? row : r) * kN;
    double2 p[kB], y[kB];
#pragma unroll
    for (int b = 0; b < kB; b++) {
      p[b] = load2(P + at + 8 * b + 2 * t);
      y[b] = load2(R + at + 8 * b + 2 * t);
    }
    __syncwarp();  // every lane has read its rows before one is written
#pragma unroll
    for (int bk = 0; bk < kB; bk++)
#pragma unroll
      for (int bn = 0; bn < kB; bn++) {
        mma_f64(y[bn].x, y[bn].y, p[bk].x, f[bn][bk][0]);
        mma_f64(y[bn].x, y[bn].y, p[bk].y, f[bn][bk][1]);
      }
    if (ok)
#pragma unroll
      for (int b = 0; b < kB; b++) store2(P + at + 8 * b + 2 * t, y[b]);
  }
}

// norms of the right-hand sides from the records of B B^T
__global__ void k_cg_norms32(const double* recs, int nrec, int n, double* small) {
  SmallView v(small);
  const int i = threadIdx.x;
  if (i < n) {
    v.norms[i] = sqrt(sum_rec(recs, nrec, rec_at(i, i)));
    v.inorms[i] = 1.0 / v.norms[i];
  }
}
__global__ void k_cg_rtr32(const double* recs, int nrec, int n, double* small) {
  SmallView v(small);
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int i = e % n, j = e / n;
    v.RtR[i + j * 64] = sum_rec(recs, nrec, rec_at(max(i, j), min(i, j)));
  }
}

struct SolveShared {
  double M[kTri * 64];    // the matrix, then its factor
  double Y[kTri * 64];    // the factor's inverse
  double S[kB * kB * 64]; // right-hand sides, full
  double Z[kB * kB * 64]; // Y S
  double Di[kB * 64];
  double y[kN], zero[kN];
  int bad, conv, broken;
};

// PSI = false: A = (chol(P^T KP) \ R^T R)^T (linop.h:286-289), the matrix summed from `recs`, the
// right-hand side v.RtR.  PSI = true: R2 = R^T R summed from `recs`; converged when all its diagonal
// is below tol^2; Psi = (chol(v.RtR) \ R2)^T; v.RtR <- R2.  A pivot that is not positive takes the
// general path (cg_small.cuh), which leaves the factor partial like the reference's unchecked llt().
template <bool PSI>
__global__ void __launch_bounds__(kThreads, 1)
    k_cg_solve(const double* __restrict__ recs, int nrec, int n, double tolsq, double* small,
               Ctl* ctl, int* flag_out, int iter) {
  if (ctl->cg_done) return;
  __shared__ __align__(16) SolveShared sh;
  SmallView v(small);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int nb = (n + 7) / 8, n8 = 8 * nb;
  if (tid == 0) {
    sh.bad = 0;
    sh.conv = 1;
    sh.broken = 0;
  }
  if (tid < kN) sh.y[tid] = sh.zero[tid] = 0.0;
  // the summed records as a matrix: M (identity beyond n), or the full right-hand side S
  for (int e = tid; e < nb * (nb + 1) / 2 * 64; e += kThreads) {
    int bi = 0;
    while ((bi + 1) * (bi + 2) / 2 <= (e >> 6)) bi++;
    const int bj = (e >> 6) - bi * (bi + 1) / 2, r = (e >> 3) & 7, c = e & 7;
    const int i = 8 * bi + r, j = 8 * bj + c;
    const double x = i < n && j < n ? sum_rec(recs, nrec, e) : (i == j && !PSI ? 1.0 : 0.0);
    if constexpr (PSI) {
      if (i >= j) {
        sh.S[(bi * kB + bj) * 64 + tile_pos(r, c)] = x;
        sh.S[(bj * kB + bi) * 64 + tile_pos(c, r)] = x;
      }
    } else {
      sh.M[(e & ~63) + tile_pos(r, c)] = x;
    }
  }
  for (int e = tid; e < n8 * n8; e += kThreads) {
    const int i = e % n8, j = e / n8;
    const bool in = i < n && j < n;
    const double x = in ? v.RtR[i + j * 64] : 0.0;
    if constexpr (PSI) {
      if (i >= j) sh.M[elem_at(i, j)] = in ? x : (i == j ? 1.0 : 0.0);
    } else {
      sh.S[((i >> 3) * kB + (j >> 3)) * 64 + tile_pos(i & 7, j & 7)] = x;
    }
  }
  __syncthreads();
  if constexpr (PSI) {
    if (tid < n) {
      const double d = sh.S[((tid >> 3) * (kB + 1)) * 64 + tile_pos(tid & 7, tid & 7)];
      if (!(d < tolsq)) atomicAnd(&sh.conv, 0);
      if (!isfinite(d)) atomicOr(&sh.broken, 1);
    }
    __syncthreads();
    // a non-finite residual ends the iteration and reports a breakdown
    const bool conv = sh.conv || sh.broken;
    if (tid == 0) {
      if (sh.broken) atomicOr(&ctl->status, kStatCgFail);
      v.flags[0] = conv;
      ctl->cg_done = (uint32_t)conv;
      if (flag_out && conv) {  // [1]: the iteration that converged, then [0]: done
        flag_out[1] = iter;
        __threadfence_system();
        flag_out[0] = 1;
      }
    }
    if (conv) return;
  }
  const bool ok = wide_factor<double, kN, kThreads>(sh.M, sh.y, sh.Di, sh.zero, nb, 0.0, tid, 0,
                                                    &sh.bad);
  double* Out = PSI ? v.Psi : v.A;
  if (ok) {
    // Y = L^{-1}: diagonal tiles from the factor, a warp per block column below
    for (int e = tid; e < 64 * nb; e += kThreads) {
      const int b = e >> 6, r = (e >> 3) & 7, c = e & 7;
      sh.Y[tile_at(b, b) + tile_pos(r, c)] = sh.Di[64 * b + tile_pos(c, r)];
    }
    __syncthreads();
    if (warp < nb) inverse_column(sh.M, sh.Y, warp, nb, lane);
    __syncthreads();
    // Z = Y S
    for (int q = warp; q < nb * nb; q += kWarps) {
      const int bi = q / nb, bj = q % nb;
      double2 z = make_double2(0.0, 0.0);
      for (int k = 0; k <= bi; k++) {
        const double* A = sh.Y + tile_at(bi, k);
        const double* B = sh.S + (k * kB + bj) * 64;
        mma_f64(z.x, z.y, A[tile_pos(g, t)], B[tile_pos(t, g)]);
        mma_f64(z.x, z.y, A[tile_pos(g, t + 4)], B[tile_pos(t + 4, g)]);
      }
      *reinterpret_cast<double2*>(sh.Z + (bi * kB + bj) * 64 + tile_pos(g, 2 * t)) = z;
    }
    __syncthreads();
    // Y^T Z, column c of the solution to Out(c, .)
    for (int q = warp; q < nb * nb; q += kWarps) {
      const int bi = q / nb, bj = q % nb;
      double z[2] = {0.0, 0.0};
      for (int k = bi; k < nb; k++) {
        const double* A = sh.Y + tile_at(k, bi);
        const double* B = sh.Z + (k * kB + bj) * 64;
        mma_f64(z[0], z[1], A[tile_pos(t, g)], B[tile_pos(t, g)]);
        mma_f64(z[0], z[1], A[tile_pos(t + 4, g)], B[tile_pos(t + 4, g)]);
      }
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int i = 8 * bi + g, c = 8 * bj + 2 * t + e;
        if (i < n && c < n) Out[c + i * 64] = z[e];
      }
    }
  } else {
    // general path over global memory: matrix in v.M, right-hand sides in v.RtR / v.RtR2
    for (int e = tid; e < n * n; e += kThreads) {
      const int i = e % n, j = e / n;
      if constexpr (PSI) {
        v.M[i + j * 64] = v.RtR[i + j * 64];
        v.RtR2[i + j * 64] = sh.S[((i >> 3) * kB + (j >> 3)) * 64 + tile_pos(i & 7, j & 7)];
      } else if (i >= j) {
        v.M[i + j * 64] = sum_rec(recs, nrec, rec_at(i, j));
      }
    }
    cta_chol_n(v.M, n, 64);
    __syncthreads();
    cta_chol_solve_cols(v.M, PSI ? v.RtR2 : v.RtR, n, Out);
  }
  if constexpr (PSI) {
    __syncthreads();
    for (int e = tid; e < n * n; e += kThreads) {
      const int i = e % n, j = e / n;
      v.RtR[i + j * 64] = sh.S[((i >> 3) * kB + (j >> 3)) * 64 + tile_pos(i & 7, j & 7)];
    }
  }
}

// R = P = B * inorms (V), X = 0, Bn = B * inorms (FP64, for residual replacement)
template <typename V>
__global__ void k_cg_init32(const double* __restrict__ B, long long nfeat, int n,
                            const double* small, V* R, V* P, double* X, double* Bn, Ctl* ctl) {
  SmallView v(const_cast<double*>(small));
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl->cg_done = 0u;  // the iterations' skip flag
  const long long total = nfeat * kN;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(e % kN);
    const double r = k < n ? B[e] * v.inorms[k] : 0.0;
    R[e] = (V)r;
    P[e] = (V)r;
    X[e] = 0.0;
    if (Bn) Bn[e] = r;
  }
}

constexpr size_t kReduceSmem = sizeof(double) * kWarps * kRecord;
static_assert(kReduceSmem >= sizeof(double) * kWarps * 8 * (kN + 4), "the update's row tiles");

// Grid of the reducing kernels: whole clusters, one CTA per SM at most, at least four row steps a warp.
int reduce_grid(long long nfeat) {
  const long long ctas = (nfeat + 4 * 8 * kWarps - 1) / (4 * 8 * kWarps);
  const long long clusters = std::min<long long>(kMaxClusters, (ctas + kCluster - 1) / kCluster);
  return (int)std::max(1LL, clusters) * kCluster;
}

template <typename V>
void set_up_kernels() {
  static bool configured[64] = {false};
  int dev = 0;
  MG_CUDA(cudaGetDevice(&dev));
  if (configured[dev & 63]) return;
  MG_CUDA(cudaFuncSetAttribute(k_cg_outer<V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kReduceSmem));
  MG_CUDA(cudaFuncSetAttribute(k_cg_update<V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kReduceSmem));
  configured[dev & 63] = true;
}

}  // namespace

template <typename V>
void Cg32<V>::start(const double* Bn, long long nfeat, int n, V* R, V* P, double* X, double* Bsave,
                    double* small, double* recs, Ctl* ctl, cudaStream_t s) {
  set_up_kernels<V>();
  if constexpr (sizeof(V) == 4) set_up_kernels<double>();
  const int grid = reduce_grid(nfeat), nrec = grid / kCluster;
  k_cg_outer<double><<<grid, kThreads, kReduceSmem, s>>>(Bn, Bn, nfeat, recs, nullptr);
  MG_CUDA(cudaGetLastError());
  k_cg_norms32<<<1, 32, 0, s>>>(recs, nrec, n, small);
  MG_CUDA(cudaGetLastError());
  const int eg = (int)std::min<long long>(148 * 16, (nfeat * kN + 255) / 256);
  k_cg_init32<V><<<eg, 256, 0, s>>>(Bn, nfeat, n, small, R, P, X, Bsave, ctl);
  MG_CUDA(cudaGetLastError());
  k_cg_outer<V><<<grid, kThreads, kReduceSmem, s>>>(R, R, nfeat, recs, nullptr);
  MG_CUDA(cudaGetLastError());
  k_cg_rtr32<<<1, 256, 0, s>>>(recs, nrec, n, small);
  MG_CUDA(cudaGetLastError());
}

template <typename V>
void Cg32<V>::step_a(long long nfeat, int n, const V* P, const V* KP, V* R, double* X, double* small,
                     double* recs, bool with_rr, Ctl* ctl, cudaStream_t s) {
  const int grid = reduce_grid(nfeat), nrec = grid / kCluster;
  const uint32_t* done = &ctl->cg_done;
  k_cg_outer<V><<<grid, kThreads, kReduceSmem, s>>>(P, KP, nfeat, recs, done);
  MG_CUDA(cudaGetLastError());
  k_cg_solve<false><<<1, kThreads, 0, s>>>(recs, nrec, n, 0.0, small, ctl, nullptr, 0);
  MG_CUDA(cudaGetLastError());
  k_cg_update<V><<<grid, kThreads, kReduceSmem, s>>>(nfeat, n, small, P, KP, R, X,
                                                     with_rr ? recs : nullptr, done);
  MG_CUDA(cudaGetLastError());
}

template <typename V>
void Cg32<V>::rr(long long nfeat, const V* R, double* recs, Ctl* ctl, cudaStream_t s) {
  k_cg_outer<V><<<reduce_grid(nfeat), kThreads, kReduceSmem, s>>>(R, R, nfeat, recs, &ctl->cg_done);
  MG_CUDA(cudaGetLastError());
}

template <typename V>
void Cg32<V>::step_psi(long long nfeat, int n, const V* R, V* P, double* small, double* recs,
                       double tolsq, Ctl* ctl, int* flag, int iter, cudaStream_t s) {
  const int nrec = reduce_grid(nfeat) / kCluster;
  k_cg_solve<true><<<1, kThreads, 0, s>>>(recs, nrec, n, tolsq, small, ctl, flag, iter);
  MG_CUDA(cudaGetLastError());
  const long long ctas = (nfeat + 8 * kWarps - 1) / (8 * kWarps);
  k_cg_pupdate<V><<<(int)std::min<long long>(296, ctas), kThreads, 0, s>>>(nfeat, n, small, R, P,
                                                                          &ctl->cg_done);
  MG_CUDA(cudaGetLastError());
}

template struct Cg32<double>;
template struct Cg32<float>;

}  // namespace mg
