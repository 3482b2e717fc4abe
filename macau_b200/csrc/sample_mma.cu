// Per-row latent sampler in FP64 for K <= 32 (sample_latent_blas, latentprior.cpp:361-385): one
// warp samples a row, with the row's Gram V^T V on the FP64 matrix instruction
// mma.sync.m8n8k4.f64 (each accumulation an IEEE FP64 fma).
//
// Why the matrix instruction.  Both Gram operands of an m8n8k4 step are the same four gathered
// rows: lane (g, t) = (lane / 4, lane % 4) holds component g of entry t as A's element (g, t) and
// as B's element (t, g).  So a lane loads each component block once, straight from global memory
// into the fragment, and every lower-triangle tile of the Gram is one instruction on values
// already in registers: no shared-memory staging, no barrier, and 10 tiles of 256 products per
// four entries at K = 32 where 4 x 8 register tiles on DFMA formed all 1,024 products per entry
// from six 16-byte shared-memory loads a lane.
//
// What bounds it: the FP64 pipe (an m8n8k4 takes 16 cycles of a sub-partition, measured, 36.9
// TFLOP/s per GPU) for long rows, and the latency of the row finish for short ones; 16 warps per
// SM at 128 registers keep four rows per sub-partition in flight, and the gathers run three
// steps (12 entries) ahead of the products.  138,000 x 27,000 with 18M entries at K = 32: both
// half-sweeps took 8.5 ms of an 8.97 ms sweep with the DFMA tiles; the sweep takes 2.44 ms now, of
// which the Grams are 1.25 ms of matrix instructions and most of the rest the row finishes.  2,000 x 1,500
// with 54,000 entries at K = 10: a sweep of 112 us became 77 us.
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
struct Warp64 {
  static constexpr int NB = KP / 8;             // component blocks
  static constexpr int TILES = NB * (NB + 1) / 2;
  static constexpr int LD = KP + 1;             // Gram tile in shared memory
  static constexpr int kRing = 4;               // gather stages: loads run three steps ahead
  // MM's tiles and the inverses of the diagonal ones, or the whole Gram of the univariate draws
  // (KP x LD); then the rhs
  static constexpr size_t kTiles = (size_t)(TILES + NB) * 64;
  static constexpr size_t kWork = kTiles > (size_t)KP * LD ? kTiles : (size_t)KP * LD;
  static constexpr size_t kWarpDoubles = kWork + KP;
  static constexpr size_t kCtaDoubles = (size_t)TILES * 64 + KP;  // Lambda's tiles, Lambda mu
};

// Fragment blocks of one entry (component g of each block) of the gathered row `row`, zero when !ok.
template <int KP>
__device__ __forceinline__ void gather_frag(double (&f)[KP / 8], const double* __restrict__ other,
                                            int row, int g, bool ok) {
  const double* src = other + (size_t)row * KP + g;
#pragma unroll
  for (int b = 0; b < KP / 8; b++) f[b] = ok ? __ldg(src + 8 * b) : 0.0;
}

// G warps (row groups) per CTA; 16 warps per SM in every shape.
template <int KP, int G>
__global__ void __launch_bounds__(32 * G, 16 / G) k_sample_f64(const SampleParams p) {
  using C = Warp64<KP>;
  constexpr int NB = C::NB, LD = C::LD, R = C::kRing;
  extern __shared__ __align__(16) double smem_d[];
  double* Lam_s = smem_d;  // Lambda's lower-triangle tiles, the identity beyond K; then Lambda mu
  double* lmu_s = Lam_s + C::TILES * 64;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* Gs = smem_d + C::kCtaDoubles + (size_t)warp * C::kWarpDoubles;
  double* rhs_s = Gs + C::kWork;
  const int g = lane >> 2, t = lane & 3;
  const int K = p.K, ntasks = p.ntasks;
  // the first task is claimed while Lambda is staged
  int ti = 0;
  if (lane == 0) ti = (int)atomicAdd(&p.ctl->queue[p.qslot], 1u);
  ti = __shfl_sync(0xffffffffu, ti, 0);
  for (int e = threadIdx.x; e < KP * KP; e += blockDim.x) {
    const int i = e % KP, j = e / KP;
    if ((i >> 3) >= (j >> 3))
      Lam_s[tile_at(i >> 3, j >> 3) + tile_pos(i & 7, j & 7)] =
          i < K && j < K ? p.Lambda[i + j * K] : (i == j ? 1.0 : 0.0);
  }
  if (threadIdx.x < KP) {
    double s = 0.0;
    if ((int)threadIdx.x < K)
      for (int j = 0; j < K; j++) s += p.Lambda[threadIdx.x + j * K] * p.mu[j];
    lmu_s[threadIdx.x] = s;
  }
  __syncthreads();
  const uint32_t sweep = p.ctl->sweep;
  const double* other = reinterpret_cast<const double*>(p.other);
  const double alpha = noise_alpha(p);

  // entries in chunks of 32 (lane l: entry l of the chunk), steps of four entries
  auto load_chunk = [&](const RowTask& task, int off, int& c, double& w) {
    const bool in = off + lane < task.len;
    c = in ? __ldcs(p.colidx + task.begin + off + lane) : 0;
    w = in ? (__ldcs(p.vals + task.begin + off + lane) - p.mean) * alpha : 0.0;
  };
  RowTask tk{};
  int c_cur = 0, c_nxt = 0, c_nn = 0;  // this chunk's columns, the next one's and the one after's
  double w_cur = 0.0, w_nxt = 0.0, w_nn = 0.0;
  if (ti < ntasks) {
    tk = p.tasks[ti];
    load_chunk(tk, 0, c_cur, w_cur);
  }
  while (ti < ntasks) {
    int ti_next = 0;  // claimed early: its latency passes behind this row
    if (lane == 0) ti_next = (int)atomicAdd(&p.ctl->queue[p.qslot], 1u);
    load_chunk(tk, 32, c_nxt, w_nxt);

    double acc[C::TILES][2];
    double racc[NB];
#pragma unroll
    for (int q = 0; q < C::TILES; q++) acc[q][0] = acc[q][1] = 0.0;
#pragma unroll
    for (int b = 0; b < NB; b++) racc[b] = 0.0;

    double f[R][NB];
#pragma unroll
    for (int u = 0; u < R - 1; u++)
      gather_frag<KP>(f[u], other, __shfl_sync(0xffffffffu, c_cur, 4 * u + t), g,
                      4 * u + t < tk.len);
    for (int off = 0; off < tk.len; off += 32) {
      load_chunk(tk, off + 64, c_nn, w_nn);
#pragma unroll
      for (int u = 0; u < 8; u++) {
        if (off + 4 * u < tk.len) {
          // gathers of step u + R - 1, which may lie in the next chunk
          const int v = u + R - 1;
          const int cv = __shfl_sync(0xffffffffu, v < 8 ? c_cur : c_nxt, 4 * (v & 7) + t);
          gather_frag<KP>(f[v % R], other, cv, g, off + 4 * v + t < tk.len);
          const double w = __shfl_sync(0xffffffffu, w_cur, 4 * u + t);
          int q = 0;
#pragma unroll
          for (int bi = 0; bi < NB; bi++) {
            racc[bi] = fma(f[u % R][bi], w, racc[bi]);
#pragma unroll
            for (int bj = 0; bj <= bi; bj++) {
              mma_f64(acc[q][0], acc[q][1], f[u % R][bi], f[u % R][bj]);
              q++;
            }
          }
        }
      }
      c_cur = c_nxt;
      w_cur = w_nxt;
      c_nxt = c_nn;
      w_nxt = w_nn;
    }
    // the next row's task and first chunk are loaded behind this row's finish
    ti = __shfl_sync(0xffffffffu, ti_next, 0);
    RowTask tk_next{};
    if (ti < ntasks) {
      tk_next = p.tasks[ti];
      load_chunk(tk_next, 0, c_cur, w_cur);
    }
    // the rhs: the four entry lanes of a group hold partial sums
#pragma unroll
    for (int b = 0; b < NB; b++) {
      racc[b] += __shfl_xor_sync(0xffffffffu, racc[b], 1);
      racc[b] += __shfl_xor_sync(0xffffffffu, racc[b], 2);
    }

    bool finish = true;
    if (tk.nparts > 1) {  // a part of a split row: the last part to arrive adds them in order
      constexpr size_t kSlot = (size_t)KP * KP + KP;
      double* sp = p.scratch + (size_t)(tk.slot + tk.part) * kSlot;
#pragma unroll
      for (int q = 0; q < C::TILES; q++)
        *reinterpret_cast<double2*>(sp + (q * 32 + lane) * 2) = make_double2(acc[q][0], acc[q][1]);
      if (t == 0)
#pragma unroll
        for (int b = 0; b < NB; b++) sp[KP * KP + 8 * b + g] = racc[b];
      __threadfence();
      __syncwarp();
      int last = 0;
      if (lane == 0)
        last = atomicAdd(&p.split_cnt[tk.split], 1u) == (unsigned)(tk.nparts - 1) ? 1 : 0;
      finish = __shfl_sync(0xffffffffu, last, 0) != 0;
      if (finish) {
        __threadfence();
#pragma unroll
        for (int q = 0; q < C::TILES; q++) acc[q][0] = acc[q][1] = 0.0;
#pragma unroll
        for (int b = 0; b < NB; b++) racc[b] = 0.0;
        for (int part = 0; part < tk.nparts; part++) {
          const double* s = p.scratch + (size_t)(tk.slot + part) * kSlot;
#pragma unroll
          for (int q = 0; q < C::TILES; q++) {
            const double2 v = __ldcg(reinterpret_cast<const double2*>(s + (q * 32 + lane) * 2));
            acc[q][0] += v.x;
            acc[q][1] += v.y;
          }
#pragma unroll
          for (int b = 0; b < NB; b++) racc[b] += __ldcg(s + KP * KP + 8 * b + g);
        }
        if (lane == 0) p.split_cnt[tk.split] = 0u;
      }
    }

    if (finish) {
      const int row = tk.row;
      if (p.one) {
        // univariate prior: the Gram (both triangles) to shared memory, coordinate draws from it by
        // the lane of its row (warp_finish.cuh)
        int q = 0;
#pragma unroll
        for (int bi = 0; bi < NB; bi++)
#pragma unroll
          for (int bj = 0; bj <= bi; bj++) {
            const int i = 8 * bi + g, j0 = 8 * bj + 2 * t, j1 = j0 + 1;
            Gs[i * LD + j0] = acc[q][0];
            Gs[i * LD + j1] = acc[q][1];
            if (bi != bj) {
              Gs[j0 * LD + i] = acc[q][0];
              Gs[j1 * LD + i] = acc[q][1];
            }
            q++;
          }
        if (t == 0)
#pragma unroll
          for (int b = 0; b < NB; b++) rhs_s[8 * b + g] = racc[b];
        __syncwarp();
        const double rac = lane < KP ? rhs_s[lane] : 0.0;
        double gr[KP];
#pragma unroll
        for (int j = 0; j < KP; j++) gr[j] = lane < K ? Gs[lane * LD + j] : 0.0;
        const double u0 = lane < K ? p.out_f64[(size_t)row * KP + lane] : 0.0;
        const double un = one_gs_warp<KP, double>(gr, rac, u0, p, row, sweep, lane);
        if (lane < K) p.out_f64[(size_t)row * KP + lane] = un;
      } else {
        const double z = row_noise(p, row, K, lane, sweep);
        // MM = Lambda + alpha G as tiles (the Gram is zero beyond K), the rhs by component
        int q = 0;
#pragma unroll
        for (int bi = 0; bi < NB; bi++)
#pragma unroll
          for (int bj = 0; bj <= bi; bj++) {
            const int at = tile_at(bi, bj) + tile_pos(g, 2 * t);
            const double2 lam = *reinterpret_cast<const double2*>(Lam_s + at);
            *reinterpret_cast<double2*>(Gs + at) =
                make_double2(lam.x + alpha * acc[q][0], lam.y + alpha * acc[q][1]);
            q++;
          }
        if (t == 0)
#pragma unroll
          for (int b = 0; b < NB; b++) rhs_s[8 * b + g] = racc[b];
        __syncwarp();
        if (lane < KP) rhs_s[lane] += lmu_s[lane];  // no Uhat: link chains go through k_sample
        __syncwarp();
        if (warp_tiles_solve<NB>(Gs, Gs + C::TILES * 64, rhs_s, (K + 7) / 8, z, lane)) {
          __syncwarp();
          if (lane < K) p.out_f64[(size_t)row * KP + lane] = rhs_s[lane];
        } else if (lane == 0) {
          atomicOr(&p.ctl->status, kStatCholFail);
          atomicCAS(&p.ctl->bad_row, -1, row);
        }
      }
      __syncwarp();
    }
    tk = tk_next;
  }
}

template <int KP, int G>
void launch_f64(const SampleParams& p, cudaStream_t s, int num_sms) {
  using C = Warp64<KP>;
  constexpr size_t smem = sizeof(double) * (C::kCtaDoubles + G * C::kWarpDoubles);
  static bool configured[64] = {false};
  int dev = 0;
  MG_CUDA(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    MG_CUDA(cudaFuncSetAttribute(k_sample_f64<KP, G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
    configured[dev & 63] = true;
  }
  const int need = std::max(1, (p.ntasks + G - 1) / G);
  k_sample_f64<KP, G><<<std::min(num_sms * (16 / G), need), 32 * G, smem, s>>>(p);
  MG_CUDA(cudaGetLastError());
}

}  // namespace

void launch_sample_f64(const SampleParams& p, int KP, cudaStream_t s, int num_sms, int groups) {
  const bool two = groups == 2;
  switch (KP) {
    case 8: return two ? launch_f64<8, 2>(p, s, num_sms) : launch_f64<8, 4>(p, s, num_sms);
    case 16: return two ? launch_f64<16, 2>(p, s, num_sms) : launch_f64<16, 4>(p, s, num_sms);
    case 32: return two ? launch_f64<32, 2>(p, s, num_sms) : launch_f64<32, 4>(p, s, num_sms);
  }
  throw MgError(MG_ERR_ARG, "unsupported latent dimension");
}

}  // namespace mg
