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
// What bounds it: the FP64 pipe (an m8n8k4 takes 16 cycles of a sub-partition, measured, 34
// TFLOP/s per GPU) for long rows, and the latency of the row finish for short ones; 16 warps per
// SM at 128 registers keep four rows per sub-partition in flight, and the gathers run three
// steps (12 entries) ahead of the products.  138,000 x 27,000 with 18M entries at K = 32: both
// half-sweeps took 8.5 ms of an 8.97 ms sweep with the DFMA tiles, 2.5 of 2.98 ms here; 2,000 x
// 1,500 with 54,000 entries at K = 10: a sweep of 112 us became 95 us.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "mma_tiles.cuh"
#include "rng.cuh"
#include "warp_finish.cuh"
#include "wide_tiles.cuh"

namespace mg {
namespace {

// Component of fragment block b held by lane group g.  Two blocks share one 16-byte load, so that
// the eight groups read 128 contiguous bytes of a gathered row: blocks 2c and 2c + 1 hold the
// even and odd components of 16c .. 16c + 15.
template <int KP>
__device__ __forceinline__ int comp_of(int b, int g) {
  return KP == 8 ? g : 16 * (b >> 1) + 2 * g + (b & 1);
}

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
  static constexpr size_t kCtaDoubles = (size_t)KP * (KP + 1) + KP;  // Lambda, Lambda mu
};

// Fragment blocks of one entry (lane's group g) of the gathered row `row`, zero when !ok.
template <int KP>
__device__ __forceinline__ void gather_frag(double (&f)[KP / 8], const double* __restrict__ other,
                                            int row, int g, bool ok) {
  const double* src = other + (size_t)row * KP;
  if constexpr (KP == 8) {
    f[0] = ok ? __ldg(src + g) : 0.0;
  } else {
#pragma unroll
    for (int c = 0; c < KP / 16; c++) {
      const double2 v = ok ? __ldg(reinterpret_cast<const double2*>(src + 16 * c) + g)
                           : make_double2(0.0, 0.0);
      f[2 * c] = v.x;
      f[2 * c + 1] = v.y;
    }
  }
}

// G warps (row groups) per CTA; 16 warps per SM in every shape.
template <int KP, int G>
__global__ void __launch_bounds__(32 * G, 16 / G) k_sample_f64(const SampleParams p) {
  using C = Warp64<KP>;
  constexpr int NB = C::NB, LD = C::LD, R = C::kRing;
  extern __shared__ __align__(16) double smem_d[];
  double* Lam_s = smem_d;  // Lambda (row-major, ld KP + 1), then Lambda mu
  double* lmu_s = Lam_s + KP * (KP + 1);
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
    const int i = e / KP, j = e % KP;
    Lam_s[i * (KP + 1) + j] = (i < K && j < K) ? p.Lambda[i + j * K] : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < KP) {
    double s = 0.0;
    if ((int)threadIdx.x < K)
      for (int j = 0; j < K; j++) s += Lam_s[threadIdx.x * (KP + 1) + j] * p.mu[j];
    lmu_s[threadIdx.x] = s;
  }
  __syncthreads();
  const uint32_t sweep = p.ctl->sweep;
  const double* other = reinterpret_cast<const double*>(p.other);
  const double alpha = noise_alpha(p);

  while (ti < ntasks) {
    const RowTask tk = p.tasks[ti];
    int ti_next = 0;  // claimed early: its latency passes behind this row
    if (lane == 0) ti_next = (int)atomicAdd(&p.ctl->queue[p.qslot], 1u);

    double acc[C::TILES][2];
    double racc[NB];
#pragma unroll
    for (int q = 0; q < C::TILES; q++) acc[q][0] = acc[q][1] = 0.0;
#pragma unroll
    for (int b = 0; b < NB; b++) racc[b] = 0.0;

    // entries in chunks of 32 (lane l: entry l of the chunk), steps of four entries
    auto load_chunk = [&](int off, int& c, double& w) {
      const bool in = off + lane < tk.len;
      c = in ? p.colidx[tk.begin + off + lane] : 0;
      w = in ? (p.vals[tk.begin + off + lane] - p.mean) * alpha : 0.0;
    };
    int c_cur, c_nxt = 0;
    double w_cur, w_nxt = 0.0;
    load_chunk(0, c_cur, w_cur);
    double f[R][NB];
#pragma unroll
    for (int u = 0; u < R - 1; u++)
      gather_frag<KP>(f[u], other, __shfl_sync(0xffffffffu, c_cur, 4 * u + t), g,
                      4 * u + t < tk.len);
    for (int off = 0; off < tk.len; off += 32) {
      load_chunk(off + 32, c_nxt, w_nxt);
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
            const int i = comp_of<KP>(bi, g), j0 = comp_of<KP>(bj, 2 * t),
                      j1 = comp_of<KP>(bj, 2 * t + 1);
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
          for (int b = 0; b < NB; b++) rhs_s[comp_of<KP>(b, g)] = racc[b];
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
        // MM = Lambda + alpha G as tiles, each unordered pair of components once (the blocks hold
        // the components in another order), the identity beyond K; the rhs by component
        auto put = [&](int i, int j, double gram) {
          const int hi = max(i, j), lo = min(i, j);
          Gs[elem_at(hi, lo)] = hi < K ? Lam_s[hi * (KP + 1) + lo] + alpha * gram
                                       : (hi == lo ? 1.0 : 0.0);
        };
        int q = 0;
#pragma unroll
        for (int bi = 0; bi < NB; bi++)
#pragma unroll
          for (int bj = 0; bj <= bi; bj++) {
            const int i = comp_of<KP>(bi, g);
#pragma unroll
            for (int e = 0; e < 2; e++) {
              const int j = comp_of<KP>(bj, 2 * t + e);
              if (bi != bj || i >= j) put(i, j, acc[q][e]);
            }
            q++;
          }
        if (t == 0)
#pragma unroll
          for (int b = 0; b < NB; b++) rhs_s[comp_of<KP>(b, g)] = racc[b];
        __syncwarp();
        double lm;
        if (p.uhat) {  // Macau prior mean mu + Uhat[row]
          const double mun = lane < K ? p.mu[lane] + p.uhat[(size_t)row * KP + lane] : 0.0;
          lm = 0.0;
          for (int j = 0; j < K; j++) {
            const double mj = wshfl(mun, j);
            if (lane < K) lm += Lam_s[lane * (KP + 1) + j] * mj;
          }
        } else {
          lm = lane < KP ? lmu_s[lane] : 0.0;
        }
        if (lane < KP) rhs_s[lane] += lm;
        __syncwarp();
        double x;
        if (warp_tiles_solve<NB>(Gs, Gs + C::TILES * 64, rhs_s, (K + 7) / 8, z, lane, x)) {
          if (lane < K) p.out_f64[(size_t)row * KP + lane] = x;
        } else if (lane == 0) {
          atomicOr(&p.ctl->status, kStatCholFail);
          atomicCAS(&p.ctl->bad_row, -1, row);
        }
      }
      __syncwarp();
    }
    ti = __shfl_sync(0xffffffffu, ti_next, 0);
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
