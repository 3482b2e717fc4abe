// Per-row latent sampler (sample_latent_blas, latentprior.cpp:361-385) for 32 < K <= 128, mixed with BF16
// gathers: a group of warps samples a row (4 warps at padded width 64, 8 at 128), FP32 Gram,
// factor and solves.
//
// Every element is formed by the same operations in the same order as in k_sample (a Gram element
// by one fused multiply-add per entry, a factor element by one per column, IEEE division and
// square root), because a mixed chain rounds each latent to BF16: a difference in the last FP32
// place flips that rounding for a few latents, and two such chains are 2e-5 apart after one
// sweep and 4e-4 after two (667 x 603, 67,033 entries, K = 40).  This rules the tensor cores out
// (their sums of 16 products round otherwise).  The speed comes from what does not change a result:
//   * Gram: only the lower triangle, in register tiles of 8 x 4 (K <= 64) or 8 x 8 per thread, 72
//     or 136 threads of the group, the last warp forming the right-hand side; entries staged 32 at
//     a time as FP32, double-buffered, one barrier a chunk, the next chunk's gathers and the
//     indices of the one after in flight.
//   * Factor: left-looking by panels of 8 columns with two barriers each: one warp factors the
//     diagonal tile while the others bring the tiles below up to date, whose rows are then solved
//     by a thread each; the right-hand side rides along, which is the forward substitution.
//   * Backward substitution: one barrier a panel, each warp forming the panel's eight x for itself.
//
// What bounds it: instruction issue in the Gram of long rows, the chain of divisions and square
// roots (about 100 cycles a column) for short ones, with 6 rows (K <= 64) or 2 in flight per SM.
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "rng.cuh"
#include "warp_finish.cuh"
#include "wide_tiles.cuh"

namespace mg {
namespace {

// FP32 tiles 72 floats apart: threads that hold the same element of neighbouring tiles then touch
// different banks.  The FP64 redo's are packed.
constexpr int kTile = 72;
template <typename F>
constexpr int kLd = sizeof(F) == 4 ? kTile : 64;
template <typename F = float>
__device__ __forceinline__ int ftile(int bi, int bj) { return (bi * (bi + 1) / 2 + bj) * kLd<F>; }

template <int KP>
struct Mixed {
  static constexpr int W = KP == 64 ? 4 : 8;  // warps of a row group
  static constexpr int T = 32 * W;
  static constexpr int NB = KP / 8, TRI = NB * (NB + 1) / 2;
  // register tiles: 8 rows by TC columns, those that reach the lower triangle
  static constexpr int TC = KP == 64 ? 4 : 8, CPR = 8 / TC;
  static constexpr int NTILE = CPR * TRI;
  static constexpr int RC = KP / 32;       // right-hand side components per lane
  static constexpr int kChunk = 32;        // entries per stage
  static constexpr int VPR = KP / 8;       // 16-byte vectors per gathered row
  static constexpr int NV = kChunk * VPR / T;
  // group's shared memory in doubles: tiles (FP64 for the redo; the stages before the finish) |
  // rhs, y | draws | x | diagonal | flags
  static constexpr size_t kGroupDoubles = (size_t)TRI * 64 + 4 * KP + 2;
  static constexpr size_t kCtaDoubles = KP + TRI * kTile / 2;  // Lambda mu | Lambda
  static_assert(2 * kChunk * KP * sizeof(float) <= TRI * 64 * sizeof(double), "stages");
  static_assert(NTILE <= T - 32 && KP * KP >= 8 * TC * T, "tiles, scratch slot");
  static_assert(TRI * kTile * sizeof(float) <= TRI * 64 * sizeof(double), "tiles");
};

// Accumulates the thread's tile (and the last warp's right-hand side) over a task's entries.
// vt: the thread's place in the group for the tiles, rotated from group to group so that the
// sub-partitions share the work.
template <int KP>
__device__ __forceinline__ void gram_mixed(const SampleParams& p, const RowTask& tk, double wscale,
                                           float* stage, int tid, int vt, int rt, int ct, int grp,
                                           float (&acc)[8][Mixed<KP>::TC],
                                           float (&racc)[Mixed<KP>::RC]) {
  using C = Mixed<KP>;
  const int lane = tid & 31;
  const bool tiles = (vt & ~31) < C::NTILE, rhs = vt >= C::T - 32;
  const uint4* other = reinterpret_cast<const uint4*>(p.other);
  const uint2* packed = p.packed + tk.begin;
  int col[C::NV];
  uint4 raw[C::NV];
  float w = 0.f, w_nxt = 0.f;
  auto indices = [&](int off) {
#pragma unroll
    for (int q = 0; q < C::NV; q++) {
      const int r = off + (tid + C::T * q) / C::VPR;
      col[q] = r < tk.len ? (int)packed[r].x : -1;
    }
    if (rhs)
      w_nxt = off + lane < tk.len
                  ? (float)((double)__uint_as_float(packed[off + lane].y) * wscale) : 0.f;
  };
  auto gather = [&]() {
#pragma unroll
    for (int q = 0; q < C::NV; q++)
      raw[q] = col[q] >= 0 ? __ldg(other + (size_t)col[q] * C::VPR + (tid + C::T * q) % C::VPR)
                           : make_uint4(0u, 0u, 0u, 0u);
  };
  auto put = [&](float* buf) {
#pragma unroll
    for (int q = 0; q < C::NV; q++) {
      float4* d = reinterpret_cast<float4*>(buf + 8 * (tid + C::T * q));
      const uint4 v = raw[q];
      d[0] = make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u),
                         __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
      d[1] = make_float4(__uint_as_float(v.z << 16), __uint_as_float(v.z & 0xffff0000u),
                         __uint_as_float(v.w << 16), __uint_as_float(v.w & 0xffff0000u));
    }
  };
  indices(0);
  gather();
  float w_cur = w_nxt;
  indices(C::kChunk);
  put(stage);
  int cur = 0;
  for (int off = 0; off < tk.len; off += C::kChunk) {
    const bool more = off + C::kChunk < tk.len;
    w = w_cur;
    w_cur = w_nxt;
    if (more) {
      gather();
      indices(off + 2 * C::kChunk);
    }
    group_sync<C::T>(grp);
    const float* buf = stage + cur * C::kChunk * KP;
    const int cnt = min(C::kChunk, tk.len - off);
    if (tiles) {
#pragma unroll 2
      for (int r = 0; r < cnt; r++) {
        const float* row = buf + r * KP;
        float a[8], b[C::TC];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const Vec4<float> q = lds4(row + 8 * rt + 4 * h);
#pragma unroll
          for (int u = 0; u < 4; u++) a[4 * h + u] = q.v[u];
        }
#pragma unroll
        for (int h = 0; h < C::TC / 4; h++) {
          const Vec4<float> q = lds4(row + C::TC * ct + 4 * h);
#pragma unroll
          for (int u = 0; u < 4; u++) b[4 * h + u] = q.v[u];
        }
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
          for (int j = 0; j < C::TC; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      }
    } else if (rhs) {
      for (int r = 0; r < cnt; r++) {
        const float wr = __shfl_sync(0xffffffffu, w, r);
#pragma unroll
        for (int c = 0; c < C::RC; c++)
          racc[c] = fmaf(buf[r * KP + lane + 32 * c], wr, racc[c]);
      }
    }
    cur ^= 1;
    if (more) put(stage + cur * C::kChunk * KP);
  }
}

// x[c] -= sum_{k < 8 pn} L(i, k) L(8 pn + c, k) of one row per thread: row = row i of its block's first
// tile; one fused multiply-add per column, in column order.
template <typename F>
__device__ __forceinline__ void update_row(F (&x)[8], const F* row_tile, const F* diag_row, int r,
                                           int pn) {
  for (int k = 0; k < pn; k++) {
    F a[8];
    load_row8(row_tile + k * kLd<F>, r, a);
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int c = 0; c < 8; c++) {
        const Vec4<F> b = lds4(diag_row + k * kLd<F> + c * 8 + 4 * (h ^ ((c >> 1) & 1)));
#pragma unroll
        for (int q = 0; q < 4; q++) x[c] = mfma(-a[4 * h + q], b.v[q], x[c]);
      }
  }
}

// x -> x L^{-T}, L the factored diagonal tile.
template <typename F>
__device__ __forceinline__ void solve_row(F (&x)[8], const F* L) {
#pragma unroll
  for (int c = 0; c < 8; c++) {
    F l[8];
    load_row8(L, c, l);
#pragma unroll
    for (int k = 0; k < c; k++) x[c] = mfma(-x[k], l[k], x[c]);
    x[c] = x[c] / l[c];
  }
}

// Factorises MM (nb blocks) in place, y along with it; df: MM's diagonal.  A pivot that is not
// positive, or in FP32 not above 2^-20 of its original diagonal, fails the group.
//   Per panel: warp 0 subtracts the last panel's product from the diagonal tile and factors it; a
// thread per row below subtracts all earlier panels' products, and the last warp those of the next
// diagonal tile; barrier; the rows below are solved in their threads' registers; barrier.
template <int T, typename F>
__device__ __forceinline__ bool factor_mixed(F* M, F* y, const float* df, int nb, int tid, int grp,
                                             volatile int* bad) {
  constexpr int W = T / 32;
  const int warp = tid >> 5, lane = tid & 31, r = tid & 7;
  for (int pn = 0; pn < nb; pn++) {
    F* D = M + ftile<F>(pn, pn);
    // row of the panel: warp 0 the panel's own, the others those below
    const int j = warp == 0 ? 8 * pn + r : 8 * pn + 8 + tid - 32;
    const bool below = warp > 0 && j < 8 * nb;
    F* tile = M + ftile<F>(below ? j >> 3 : pn, 0);  // the row's block
    F s = (F)0, x[8];
    if (pn > 0 && (warp == 0 || below)) {  // y by the panel before
      F v[8];
      load_row8(tile + (pn - 1) * kLd<F>, r, v);
      s = y[j];
#pragma unroll
      for (int c = 0; c < 8; c++) s = mfma(-v[c], y[8 * pn - 8 + c], s);
    }
    if (warp == 0) {
      if (pn > 0) {
        update_tile(D, M + ftile<F>(pn, 0), M + ftile<F>(pn, 0), pn - 1, pn, kLd<F>, lane);
        if (lane < 8) y[j] = s;
      }
      __syncwarp();
      // lanes 0-7: the tile's rows, 8: y (the others repeat it)
      F* own = lane < 8 ? D : y + 8 * pn;
      const int at = lane < 8 ? r : 0;
      load_row8(own, at, x);
      __syncwarp();
      bool ok = true;
#pragma unroll
      for (int c = 0; c < 8; c++) {
        const F d = wshfl(x[c], c);
        ok = ok & (d > (F)0);
        if constexpr (sizeof(F) == 4) ok = ok & (d > 0x1p-20f * df[8 * pn + c]);
        const F l = msqrt(d), q = (lane > c ? x[c] : d) / l;  // above the diagonal: anything
        x[c] = lane == c ? l : q;
#pragma unroll
        for (int k = c + 1; k < 8; k++) x[k] = mfma(-x[c], wshfl(x[c], k), x[k]);
      }
      if (lane <= 8) store_row8(own, at, x);
      if (!ok && lane == 0) *bad = 1;
    } else {
      if (below) {
        if (pn > 0) y[j] = s;
        load_row8(tile + pn * kLd<F>, r, x);
        update_row(x, tile, M + ftile<F>(pn, 0), r, pn);
      }
      if (warp == W - 1 && pn > 0 && pn + 1 < nb) {
        const F* next = M + ftile<F>(pn + 1, 0);
        update_tile(M + ftile<F>(pn + 1, pn + 1), next, next, 0, pn, kLd<F>, lane);
      }
    }
    group_sync<T>(grp);
    if (*bad) return false;
    if (below) {
      solve_row(x, D);
      store_row8(tile + pn * kLd<F>, r, x);
    }
    group_sync<T>(grp);
  }
  return true;
}

// x = L^{-T} y over the panels from the last (y is overwritten).
template <int T, typename F>
__device__ __forceinline__ void back_mixed(const F* M, F* y, F* x, int nb, int tid, int grp) {
  const int warp = tid >> 5, r = tid & 7;
  for (int pn = nb - 1; pn >= 0; pn--) {
    if (warp == 0 || 32 * warp < 8 * pn) {
      const F* D = M + ftile<F>(pn, pn);
      const bool on = tid < 8 * pn;
      const F* P = M + ftile<F>(pn, on ? tid >> 3 : 0);
      F d[8], l[8], p[8], b = y[8 * pn + r], s = on ? y[tid] : (F)0;
#pragma unroll
      for (int c = 0; c < 8; c++) {
        d[c] = D[tile_pos(c, r)];
        l[c] = D[tile_pos(c, c)];
        p[c] = P[tile_pos(c, r)];
      }
#pragma unroll
      for (int c = 7; c >= 0; c--) {
        const F xc = wshfl(b, c) / l[c];
        if (r < c) b = mfma(-d[c], xc, b);
        if (r == c) b = xc;
        s = mfma(-p[c], xc, s);
      }
      if (on) y[tid] = s;
      if (tid < 8) x[8 * pn + tid] = b;
    }
    group_sync<T>(grp);
  }
}

// The FP64 redo of a row from MM and the right-hand side, in the same order; kept out of line for its
// registers.
template <int T>
__device__ __noinline__ bool redo_solve(double* M, double* y, const double* z, double* x, int nb,
                                        int tid, int grp, volatile int* bad) {
  if (!factor_mixed<T>(M, y, nullptr, nb, tid, grp, bad)) return false;
  if (tid < 8 * nb) y[tid] += z[tid];
  group_sync<T>(grp);
  back_mixed<T>(M, y, x, nb, tid, grp);
  return true;
}

template <int KP, int G>
__global__ void __launch_bounds__(Mixed<KP>::T* G, (KP == 64 ? 6 : 2) / G)
    k_sample_wide_mixed(const SampleParams p, int num_sms) {
  using C = Mixed<KP>;
  constexpr int T = C::T, TC = C::TC;
  extern __shared__ __align__(16) double smem_m[];
  double* lmu_s = smem_m;
  float* lam_s = reinterpret_cast<float*>(smem_m + KP);
  const int grp = threadIdx.x / T, tid = threadIdx.x % T;
  const int lane = tid & 31;
  const int vt = (tid + 32 * (grp + 2 * ((int)blockIdx.x / num_sms))) % T;
  double* M = smem_m + C::kCtaDoubles + (size_t)grp * C::kGroupDoubles;
  double* rhs_s = M + (size_t)C::TRI * 64;
  double* z_s = rhs_s + KP;
  double* x_s = z_s + KP;
  float* df = reinterpret_cast<float*>(x_s + KP);
  volatile int* bad = reinterpret_cast<volatile int*>(df + KP);
  volatile int* bcast = bad + 1;  // [0]: task, then whether this part finishes the row
  float* Mf = reinterpret_cast<float*>(M);
  float* yf = reinterpret_cast<float*>(x_s);  // x_s holds y and x
  float* xf = yf + KP;
  const int K = p.K, nb = (K + 7) / 8, ntasks = p.ntasks;
  if (tid == 0) bcast[0] = (int)atomicAdd(&p.ctl->queue[p.qslot], 1u);
  for (int i = threadIdx.x; i < KP; i += blockDim.x) {
    double s = 0.0;
    if (i < K)
      for (int j = 0; j < K; j++) s += p.Lambda[i + (size_t)j * K] * p.mu[j];
    lmu_s[i] = s;
  }
  for (int e = threadIdx.x; e < KP * KP; e += blockDim.x) {  // both triangles of a diagonal tile
    const int i = e % KP, j = e / KP, hi = max(i, j), lo = min(i, j);
    if (i >> 3 >= j >> 3)
      lam_s[ftile(i >> 3, j >> 3) + tile_pos(i & 7, j & 7)] =
          hi < K ? (float)p.Lambda[hi + (size_t)lo * K] : (i == j ? 1.f : 0.f);
  }
  __syncthreads();
  // the thread's tile: rows 8 rt .., columns TC ct ..
  int rt = 0, ct = vt < C::NTILE ? vt : 0;
  while (ct >= C::CPR * (rt + 1)) {
    ct -= C::CPR * (rt + 1);
    rt++;
  }
  const uint32_t sweep = p.ctl->sweep;
  const double alpha = noise_alpha(p);
  const double wscale = packed_scale(p);
  int ti = bcast[0];
  while (ti < ntasks) {
    const RowTask tk = p.tasks[ti];
    int ti_next = 0;  // claimed early: its latency passes behind this row
    if (tid == 0) ti_next = (int)atomicAdd(&p.ctl->queue[p.qslot], 1u);
    // The second pass is the FP64 redo of a row whose FP32 pivot failed; it forms the Gram again (or
    // adds the parts again), so that the factor need not keep it in registers.
    for (bool redo = false;;) {
      float acc[8][TC], racc[C::RC];
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < TC; j++) acc[i][j] = 0.f;
#pragma unroll
      for (int c = 0; c < C::RC; c++) racc[c] = 0.f;
      if (!redo || tk.nparts == 1) {
        gram_mixed<KP>(p, tk, wscale, Mf, tid, vt, rt, ct, grp, acc, racc);
        if (vt >= T - 32)
#pragma unroll
          for (int c = 0; c < C::RC; c++) rhs_s[lane + 32 * c] = (double)racc[c];
      }
      group_sync<T>(grp);
      if (tk.nparts > 1) {  // a part of a split row: the last part to arrive adds them in order
        constexpr size_t kSlot = (size_t)KP * KP + KP;
        if (!redo) {
          double* sp = p.scratch + (size_t)(tk.slot + tk.part) * kSlot;
          if (vt < C::NTILE)
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
              for (int j = 0; j < TC; j++) sp[(i * TC + j) * T + vt] = (double)acc[i][j];
          if (tid < KP) sp[KP * KP + tid] = rhs_s[tid];
          __threadfence();
          group_sync<T>(grp);
          if (tid == 0)
            bcast[1] = atomicAdd(&p.split_cnt[tk.split], 1u) == (unsigned)(tk.nparts - 1) ? 1 : 0;
          group_sync<T>(grp);
          if (!bcast[1]) break;
          __threadfence();
          if (tid == 0) p.split_cnt[tk.split] = 0u;
        }
        const double* s0 = p.scratch + (size_t)tk.slot * kSlot;
        if (vt < C::NTILE)
#pragma unroll
          for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < TC; j++) {
              double a = 0.0;
              for (int part = 0; part < tk.nparts; part++)
                a += __ldcg(s0 + (size_t)part * kSlot + (i * TC + j) * T + vt);
              acc[i][j] = (float)a;
            }
        if (tid < KP) {
          double r = 0.0;
          for (int part = 0; part < tk.nparts; part++)
            r += __ldcg(s0 + (size_t)part * kSlot + KP * KP + tid);
          rhs_s[tid] = (double)(float)r;
        }
        group_sync<T>(grp);
      }

      const int row = tk.row;
      // MM = Lambda + alpha G, the identity beyond K (FP32: a diagonal tile's upper half mirrors its lower)
      if (vt < C::NTILE && rt < nb) {
        if (!redo) {
          const float af = (float)alpha;
#pragma unroll
          for (int i = 0; i < 8; i++)
#pragma unroll
            for (int h = 0; h < TC / 4; h++) {
              const int half = TC == 4 ? ct & 1 : h;
              const int at = ftile(rt, TC * ct >> 3) + i * 8 + 4 * (half ^ ((i >> 1) & 1));
              Vec4<float> v = lds4(lam_s + at);
              if (8 * rt + i < K)
#pragma unroll
                for (int u = 0; u < 4; u++) v.v[u] = fmaf(af, acc[i][4 * h + u], v.v[u]);
              *reinterpret_cast<float4*>(Mf + at) = make_float4(v.v[0], v.v[1], v.v[2], v.v[3]);
            }
        } else {
#pragma unroll
          for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < TC; j++) {
              const int gi = 8 * rt + i, gj = TC * ct + j;
              if (gi >= gj)
                M[elem_at(gi, gj)] =
                    gi < K ? fma(alpha, (double)acc[i][j], p.Lambda[gi + (size_t)gj * K])
                           : (gi == gj ? 1.0 : 0.0);
            }
        }
      }
      // the row's draws and the right-hand side Lambda (mu + Uhat[row]) + Gram rhs
      if (p.znoise) {
        if (tid < KP) z_s[tid] = tid < K ? p.znoise[(size_t)row * K + tid] : 0.0;
      } else if (tid < KP / 2) {
        double z0, z1;
        normal_pair(p.seed, sweep, stream_id(kRowNoise, (uint32_t)p.mode), (uint32_t)row,
                    (uint32_t)tid, &z0, &z1);
        z_s[2 * tid] = 2 * tid < K ? z0 : 0.0;
        z_s[2 * tid + 1] = 2 * tid + 1 < K ? z1 : 0.0;
      }
      double lm = 0.0;
      if (p.uhat) {
        if (tid < K) x_s[tid] = p.mu[tid] + p.uhat[(size_t)row * KP + tid];
        group_sync<T>(grp);
        if (tid < K)
          for (int j = 0; j < K; j++) lm += p.Lambda[tid + (size_t)j * K] * x_s[j];
        group_sync<T>(grp);
      } else {
        if (tid < KP) lm = lmu_s[tid];
      }
      if (tid < KP) {
        const double rr = rhs_s[tid] + lm;
        if (redo) rhs_s[tid] = rr;
        else yf[tid] = (float)rr;
      }
      if (tid == 0) *bad = 0;
      group_sync<T>(grp);
      if (!redo) {
        if (tid < 8 * nb) df[tid] = Mf[ftile(tid >> 3, tid >> 3) + tile_pos(tid & 7, tid & 7)];
        group_sync<T>(grp);
        if (factor_mixed<T>(Mf, yf, df, nb, tid, grp, bad)) {
          if (tid < 8 * nb) yf[tid] += (float)z_s[tid];
          group_sync<T>(grp);
          back_mixed<T>(Mf, yf, xf, nb, tid, grp);
          if (tid < K) {
            p.out_f32[(size_t)row * KP + tid] = xf[tid];
            store_copy(p, (size_t)row * KP + tid, xf[tid]);
          }
          break;
        }
        if (tid == 0) atomicAdd(&p.ctl->retries[p.mode], 1u);
        redo = true;
        group_sync<T>(grp);  // every thread has seen the flag
      } else {
        if (redo_solve<T>(M, rhs_s, z_s, x_s, nb, tid, grp, bad)) {
          if (tid < K) {
            p.out_f32[(size_t)row * KP + tid] = (float)x_s[tid];
            store_copy(p, (size_t)row * KP + tid, (float)x_s[tid]);
          }
        } else if (tid == 0) {
          atomicOr(&p.ctl->status, kStatCholFail);
          atomicCAS(&p.ctl->bad_row, -1, row);
        }
        break;
      }
    }
    if (tid == 0) bcast[0] = ti_next;
    group_sync<T>(grp);
    ti = bcast[0];
  }
}

template <int KP, int G>
void launch_mixed(const SampleParams& p, cudaStream_t s, int num_sms) {
  using C = Mixed<KP>;
  auto kern = k_sample_wide_mixed<KP, G>;
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
  kern<<<std::min(num_sms * per_sm, need), C::T * G, smem, s>>>(p, num_sms);
  MG_CUDA(cudaGetLastError());
}

}  // namespace

void launch_sample_wide_mixed(const SampleParams& p, int KP, cudaStream_t s, int num_sms,
                              int groups) {
  if (KP == 128) return launch_mixed<128, 2>(p, s, num_sms);
  if (groups == 1) return launch_mixed<64, 1>(p, s, num_sms);
  return launch_mixed<64, 2>(p, s, num_sms);
}

}  // namespace mg
