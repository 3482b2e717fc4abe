// Per-row latent sampler (sample_latent_blas, latentprior.cpp:361-385) for 32 < K <= 128 in FP64: a
// group of warps samples a row (4 warps at padded width 64, 8 at 128).
//
// Gram.  The lower-triangle tiles of V^T V are spread over the group's warps and formed by the
// warp matrix instruction m8n8k4.f64 on operands gathered straight from global memory into fragment
// registers, the next step's gathers in flight: no staging and no barrier however long the row is.
// Lane (g, t) = (lane / 4, lane % 4) loads component 8b + g of entry t, which is the operand element
// of block b on either side.
// Finish.  MM = Lambda + alpha G in shared memory as 8 x 8 tiles (lower triangle), factorised by
// panels of 8 columns with two barriers each (wide_tiles.cuh): one warp factors the diagonal tile
// while the others bring the tiles below up to date, which are then multiplied by its inverse.
// The right-hand side rides along as one more row, which is the forward substitution.  The backward
// substitution takes one barrier per panel.
//
// What bounds it: short rows, the latency of the panel chain, with 2 (K > 64) or 4 rows in flight
// per SM; long rows, the matrix instructions.  The column-by-column factor this replaces took
// three barriers a column, 78 us a row at K = 64.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "mma_tiles.cuh"
#include "rng.cuh"
#include "warp_finish.cuh"
#include "wide_tiles.cuh"

namespace mg {
namespace {

template <int KP>
struct Wide {
  static constexpr int W = KP == 64 ? 4 : 8;  // warps of a row group
  static constexpr int T = 32 * W;
  static constexpr int NB = KP / 8;                // 8-component blocks
  static constexpr int TRI = NB * (NB + 1) / 2;    // tiles of MM
  // Gram tiles per warp: a warp of the rectangles holds RB x 4 tiles, a warp of the diagonal ND
  // squares of 4 x 4 blocks (10 tiles each)
  static constexpr int RB = KP == 64 ? 2 : 4, ND = KP == 64 ? 1 : 2;
  static constexpr int NT = 10 * ND;
  // gather stages (of 4 entries); at 128 the accumulators leave no registers for a second
  // one, and four warps a sub-partition cover the latency
  static constexpr int R = KP == 64 ? 4 : 1;
  // group's shared memory in doubles: tiles | inverses of the diagonal's | rhs, y | draws | x |
  // flags
  static constexpr size_t kGroupDoubles = (size_t)(TRI + NB) * 64 + 3 * KP + 2;
  static constexpr size_t kCtaDoubles = KP;  // Lambda mu
};

// Accumulates the warp's tiles over the entries of a task; a diagonal warp also its blocks' part
// of the right-hand side (rhs_s, when the task is done).
template <int KP, bool DIAG, int NT>
__device__ __forceinline__ void gram64(const SampleParams& p, const RowTask& tk, double alpha,
                                       int r0, int c0, double (&acc)[NT][2], double* rhs_s) {
  using C = Wide<KP>;
  constexpr int R = C::R, NR = DIAG ? 4 * C::ND : C::RB, NC = DIAG ? 1 : 4;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const double* other = reinterpret_cast<const double*>(p.other) + g;
  double racc[NR];
#pragma unroll
  for (int b = 0; b < NR; b++) racc[b] = 0.0;
  auto load_chunk = [&](int off, int& c, double& w) {
    const bool in = off + lane < tk.len;
    c = in ? p.colidx[tk.begin + off + lane] : 0;
    w = DIAG && in ? (p.vals[tk.begin + off + lane] - p.mean) * alpha : 0.0;
  };
  double fr[R][NR], fc[R][NC];
  auto gather = [&](int stage, int col, bool ok) {
    const double* row = other + (size_t)col * KP;
    gather64<NR>(fr[stage], row + 8 * r0, ok);
    if constexpr (!DIAG) gather64<NC>(fc[stage], row + 8 * c0, ok);
  };
  int c_cur, c_nxt = 0;
  double w_cur, w_nxt = 0.0;
  load_chunk(0, c_cur, w_cur);
#pragma unroll
  for (int u = 0; u < R - 1; u++)
    gather(u, __shfl_sync(0xffffffffu, c_cur, 4 * u + t), 4 * u + t < tk.len);
  for (int off = 0; off < tk.len; off += 32) {
    load_chunk(off + 32, c_nxt, w_nxt);
#pragma unroll
    for (int u = 0; u < 8; u++) {
      if (off + 4 * u < tk.len) {
        const int v = u + R - 1;
        const int cv = __shfl_sync(0xffffffffu, v < 8 ? c_cur : c_nxt, 4 * (v & 7) + t);
        gather(v % R, cv, off + 4 * v + t < tk.len);
        int q = 0;
        if constexpr (DIAG) {
          const double w = __shfl_sync(0xffffffffu, w_cur, 4 * u + t);
#pragma unroll
          for (int s = 0; s < C::ND; s++)
#pragma unroll
            for (int a = 0; a < 4; a++) {
              racc[4 * s + a] = fma(fr[u % R][4 * s + a], w, racc[4 * s + a]);
#pragma unroll
              for (int b = 0; b <= a; b++) {
                mma_f64(acc[q][0], acc[q][1], fr[u % R][4 * s + a], fr[u % R][4 * s + b]);
                q++;
              }
            }
        } else {
#pragma unroll
          for (int a = 0; a < NR; a++)
#pragma unroll
            for (int b = 0; b < NC; b++) {
              mma_f64(acc[q][0], acc[q][1], fr[u % R][a], fc[u % R][b]);
              q++;
            }
        }
      }
    }
    c_cur = c_nxt;
    w_cur = w_nxt;
  }
  if constexpr (DIAG) {
#pragma unroll
    for (int b = 0; b < NR; b++) {
      racc[b] += __shfl_xor_sync(0xffffffffu, racc[b], 1);
      racc[b] += __shfl_xor_sync(0xffffffffu, racc[b], 2);
      if (t == 0) rhs_s[8 * (r0 + b) + g] = racc[b];
    }
  }
}

// ---- MM = Lambda + alpha G, the identity beyond K ----
__device__ __forceinline__ double mm_value(const double* Lambda, int K, double alpha, double gram,
                                           int i, int j) {
  return i < K && j < K ? Lambda[i + (size_t)j * K] + alpha * gram : (i == j ? 1.0 : 0.0);
}

template <int KP, bool DIAG, int NT>
__device__ __forceinline__ void store64(double* M, const double* Lambda, int K, double alpha,
                                        int r0, int c0, const double (&acc)[NT][2]) {
  using C = Wide<KP>;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  auto put = [&](int bi, int bj, const double (&v)[2]) {
    const int i = 8 * bi + g, j = 8 * bj + 2 * t;
    double* d = M + tile_at(bi, bj) + tile_pos(g, 2 * t);
    *reinterpret_cast<double2*>(d) = make_double2(mm_value(Lambda, K, alpha, v[0], i, j),
                                                  mm_value(Lambda, K, alpha, v[1], i, j + 1));
  };
  int q = 0;
  if constexpr (DIAG) {
#pragma unroll
    for (int s = 0; s < C::ND; s++)
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b <= a; b++) put(r0 + 4 * s + a, r0 + 4 * s + b, acc[q++]);
  } else {
#pragma unroll
    for (int a = 0; a < C::RB; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) put(r0 + a, c0 + b, acc[q++]);
  }
}

template <int KP, int G>
__global__ void __launch_bounds__(Wide<KP>::T* G, (KP == 64 ? 4 : 2) / G)
    k_sample_wide(const SampleParams p) {
  using C = Wide<KP>;
  constexpr int T = C::T, NT = C::NT;
  extern __shared__ __align__(16) double smem_w[];
  double* lmu_s = smem_w;
  const int grp = threadIdx.x / T, tid = threadIdx.x % T;
  const int warp = tid >> 5, lane = tid & 31;
  double* M = smem_w + C::kCtaDoubles + (size_t)grp * C::kGroupDoubles;
  double* Di = M + (size_t)C::TRI * 64;
  double* rhs_s = Di + (size_t)C::NB * 64;  // Gram rhs, then the factor's y
  double* z_s = rhs_s + KP;
  double* x_s = z_s + KP;
  volatile int* bad = reinterpret_cast<volatile int*>(x_s + KP);
  volatile int* bcast = bad + 1;  // [0]: task, [1]: whether this part finishes the row
  const int K = p.K, nb = (K + 7) / 8, ntasks = p.ntasks;
  if (tid == 0) bcast[0] = (int)atomicAdd(&p.ctl->queue[p.qslot], 1u);
  for (int i = threadIdx.x; i < KP; i += blockDim.x) {
    double s = 0.0;
    if (i < K)
      for (int j = 0; j < K; j++) s += p.Lambda[i + (size_t)j * K] * p.mu[j];
    lmu_s[i] = s;
  }
  __syncthreads();
  const uint32_t sweep = p.ctl->sweep;
  const double alpha = noise_alpha(p);
  int ti = bcast[0];
  while (ti < ntasks) {
    const RowTask tk = p.tasks[ti];
    int ti_next = 0;  // claimed early: its latency passes behind this row
    if (tid == 0) ti_next = (int)atomicAdd(&p.ctl->queue[p.qslot], 1u);
    double acc[NT][2];
#pragma unroll
    for (int q = 0; q < NT; q++)
#pragma unroll
      for (int e = 0; e < 2; e++) acc[q][e] = 0.0;

    const Part64 part = part_of<KP>(warp);
    if (part.diag) gram64<KP, true>(p, tk, alpha, part.r0, part.c0, acc, rhs_s);
    else gram64<KP, false>(p, tk, alpha, part.r0, part.c0, acc, rhs_s);

    bool finish = true;
    if (tk.nparts > 1) {  // a part of a split row: the last part to arrive adds them in order
      constexpr size_t kSlot = (size_t)KP * KP + KP;
      static_assert((size_t)C::W * NT * 64 <= (size_t)KP * KP, "scratch slot too small");
      const size_t at = ((size_t)warp * NT * 32 + lane) * 2;
      double* sp = p.scratch + (size_t)(tk.slot + tk.part) * kSlot;
#pragma unroll
      for (int q = 0; q < NT; q++)
        *reinterpret_cast<double2*>(sp + at + q * 64) = make_double2(acc[q][0], acc[q][1]);
      group_sync<T>(grp);
      if (tid < KP) sp[KP * KP + tid] = rhs_s[tid];
      __threadfence();
      group_sync<T>(grp);
      if (tid == 0)
        bcast[1] = atomicAdd(&p.split_cnt[tk.split], 1u) == (unsigned)(tk.nparts - 1) ? 1 : 0;
      group_sync<T>(grp);
      finish = bcast[1] != 0;
      if (finish) {
        __threadfence();
        const double* s0 = p.scratch + (size_t)tk.slot * kSlot;
#pragma unroll
        for (int q = 0; q < NT; q++) {
          double a = 0.0, b = 0.0;
          for (int part = 0; part < tk.nparts; part++) {
            const double2 v =
                __ldcg(reinterpret_cast<const double2*>(s0 + (size_t)part * kSlot + at + q * 64));
            a += v.x;
            b += v.y;
          }
          acc[q][0] = a;
          acc[q][1] = b;
        }
        if (tid < KP) {
          double r = 0.0;
          for (int part = 0; part < tk.nparts; part++)
            r += __ldcg(s0 + (size_t)part * kSlot + KP * KP + tid);
          rhs_s[tid] = r;
        }
        if (tid == 0) p.split_cnt[tk.split] = 0u;
      }
    }

    if (finish) {
      const int row = tk.row;
      // the row's draws and the right-hand side Lambda mu + Gram rhs (no Uhat: link chains go through
      // k_sample)
      if (p.znoise) {
        if (tid < KP) z_s[tid] = tid < K ? p.znoise[(size_t)row * K + tid] : 0.0;
      } else if (tid < KP / 2) {
        double z0, z1;
        normal_pair(p.seed, sweep, stream_id(kRowNoise, (uint32_t)p.mode), (uint32_t)row,
                    (uint32_t)tid, &z0, &z1);
        z_s[2 * tid] = 2 * tid < K ? z0 : 0.0;
        z_s[2 * tid + 1] = 2 * tid + 1 < K ? z1 : 0.0;
      }
      group_sync<T>(grp);
      const double rr = tid < KP ? rhs_s[tid] + lmu_s[tid] : 0.0;
      if (tid == 0) *bad = 0;
      if (part.diag) store64<KP, true>(M, p.Lambda, K, alpha, part.r0, part.c0, acc);
      else store64<KP, false>(M, p.Lambda, K, alpha, part.r0, part.c0, acc);
      if (tid < KP) rhs_s[tid] = rr;
      group_sync<T>(grp);
      if (wide_factor<T>(M, rhs_s, Di, nb, tid, grp, bad)) {
        if (tid < 8 * nb) rhs_s[tid] += z_s[tid];
        group_sync<T>(grp);
        wide_back<T>(M, rhs_s, Di, x_s, nb, tid, grp);
        if (tid < K) p.out_f64[(size_t)row * KP + tid] = x_s[tid];
      } else if (tid == 0) {
        atomicOr(&p.ctl->status, kStatCholFail);
        atomicCAS(&p.ctl->bad_row, -1, row);
      }
    }
    if (tid == 0) bcast[0] = ti_next;
    group_sync<T>(grp);
    ti = bcast[0];
  }
}

template <int KP, int G>
void launch_wide(const SampleParams& p, cudaStream_t s, int num_sms) {
  using C = Wide<KP>;
  auto kern = k_sample_wide<KP, G>;
  constexpr size_t smem = sizeof(double) * (C::kCtaDoubles + G * C::kGroupDoubles);
  static int per_sm_cache[64] = {0};
  int dev = 0;
  MG_CUDA(cudaGetDevice(&dev));
  int& per_sm = per_sm_cache[dev & 63];
  if (per_sm == 0) {
    MG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int n = 0;
    MG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, C::T * G, smem));
    per_sm = n < 1 ? 1 : n;
  }
  const int need = std::max(1, (p.ntasks + G - 1) / G);
  kern<<<std::min(num_sms * per_sm, need), C::T * G, smem, s>>>(p);
  MG_CUDA(cudaGetLastError());
}

}  // namespace

void launch_sample_wide(const SampleParams& p, int KP, cudaStream_t s, int num_sms, int groups) {
  if (KP == 128) return launch_wide<128, 1>(p, s, num_sms);
  if (groups == 1) return launch_wide<64, 1>(p, s, num_sms);
  return launch_wide<64, 2>(p, s, num_sms);
}

}  // namespace mg
