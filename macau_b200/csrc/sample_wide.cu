// Per-row latent sampler (sample_latent_blas, latentprior.cpp:361-385) for 32 < K <= 128, FP64 or
// mixed with BF16 gathers: a group of warps samples a row (4 warps at padded width 64, 8 at 128).
//
// Gram.  The lower-triangle tiles of V^T V are spread over the group's warps and formed by the
// warp matrix instructions (FP64: m8n8k4.f64; BF16: m16n8k16 with FP32 accumulation) on operands
// gathered straight from global memory into fragment registers, the next step's gathers in
// flight: no staging and no barrier however long the row is.
//   FP64   lane (g, t) = (lane / 4, lane % 4) loads component 8b + g of entry t, which is the
//          operand element of block b on either side.
//   BF16   lane (g, t) loads 16 bytes (components 8g .. 8g + 7 of each 64) of entries 2t, 2t + 1,
//          2t + 8 and 2t + 9 and pairs the entries by byte permutes: component 64h + 8g + b
//          becomes element g of block 8h + b.  The blocks are thus a permutation of the
//          components, undone when the Gram is stored.
// Finish.  MM = Lambda + alpha G in shared memory as 8 x 8 tiles (lower triangle), factorised by
// panels of 8 columns with two barriers each (wide_tiles.cuh): one warp factors the diagonal tile
// while the others bring the tiles below up to date, which are then multiplied by its inverse
// (FP64: m8n8k4.f64; FP32: FMAs).  The right-hand side rides along as one more row, which is the
// forward substitution.  The backward substitution takes one barrier per panel.
//
// What bounds it: short rows, the latency of the panel chain, with 2 (K > 64) or 4 rows in flight
// per SM; long rows, the matrix instructions.  The column-by-column factor this replaces took
// three barriers a column, 78 us a row at K = 64.
#include <cuda_bf16.h>

#include <algorithm>
#include <utility>

#include "common.cuh"
#include "kernels.h"
#include "mma_tiles.cuh"
#include "rng.cuh"
#include "warp_finish.cuh"
#include "wide_tiles.cuh"

namespace mg {
namespace {

template <int KP, bool MIXED>
struct Wide {
  static constexpr int W = KP == 64 ? 4 : 8;  // warps of a row group
  static constexpr int T = 32 * W;
  static constexpr int NB = KP / 8;                // 8-component blocks
  static constexpr int TRI = NB * (NB + 1) / 2;    // tiles of MM
  // Gram tiles per warp and accumulators per lane and tile.  FP64: a warp of the rectangles holds
  // RB x 4 tiles, a warp of the diagonal ND squares of 4 x 4 blocks (10 tiles each).  BF16: see
  // tile16.
  static constexpr int RB = KP == 64 ? 2 : 4, ND = KP == 64 ? 1 : 2;
  static constexpr int NT = MIXED ? (KP == 64 ? 5 : 10) : 10 * ND;
  static constexpr int AE = MIXED ? 4 : 2;
  using Acc = typename std::conditional<MIXED, float, double>::type;
  // FP64 gather stages (of 4 entries); at 128 the accumulators leave no registers for a second
  // one, and four warps a sub-partition cover the latency
  static constexpr int R = KP == 64 ? 4 : 1;
  // group's shared memory in doubles: tiles | inverses of the diagonal's | rhs, y | draws | x |
  // diagonal | flags
  static constexpr size_t kGroupDoubles = (size_t)(TRI + NB) * 64 + 4 * KP + 2;
  static constexpr size_t kCtaDoubles = KP;  // Lambda mu
};

// ---- FP64 Gram ----
// Accumulates the warp's tiles over the entries of a task; a diagonal warp also its blocks' part
// of the right-hand side (rhs_s, when the task is done).
template <int KP, bool DIAG, int NT>
__device__ __forceinline__ void gram64(const SampleParams& p, const RowTask& tk, double alpha,
                                       int r0, int c0, double (&acc)[NT][2], double* rhs_s) {
  using C = Wide<KP, false>;
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

// ---- BF16 Gram ----
// The 16 x 8 tiles of a square of 64 components: (I, j), j <= 2I + 1, in row order, rows the blocks
// 2I and 2I + 1, columns the block j (20 tiles).
constexpr int tile_row16(int t) {
  int I = 0;
  while (t >= (I + 1) * (I + 2)) I++;
  return I;
}
constexpr int tile_col16(int t) { return t - tile_row16(t) * (tile_row16(t) + 1); }

// Tiles of a warp, NT at most.  K <= 64: the square's tiles 5 w .. 5 w + 4.  K <= 128: warps 4 and 5
// share the square of components 0 .. 63, warps 6 and 7 that of 64 .. 127; warp w < 4 has the eight
// tiles of blocks 8 + 2w, 9 + 2w against blocks 0 .. 7.  Returns false past the warp's last tile.
template <int KP>
__device__ __forceinline__ bool tile16(int warp, int q, int& b_row, int& b_col) {
  constexpr int NT = Wide<KP, true>::NT;
  if (KP == 128 && warp < 4) {
    b_row = 8 + 2 * warp;
    b_col = q;
    return q < 8;
  }
  const int half = KP == 128 ? (warp - 4) >> 1 : 0;
  const int lin = (KP == 128 ? (warp & 1) : warp) * NT + q;
  int I = 0;
  while (lin >= (I + 1) * (I + 2)) I++;
  b_row = 8 * half + 2 * I;
  b_col = 8 * half + lin - I * (I + 1);
  return true;
}

// One entry pair's words: blocks 2q (low halves) and 2q + 1 (high halves).
__device__ __forceinline__ uint32_t pair_lo(uint32_t x, uint32_t y) {
  return __byte_perm(x, y, 0x5410);
}
__device__ __forceinline__ uint32_t pair_hi(uint32_t x, uint32_t y) {
  return __byte_perm(x, y, 0x7632);
}
__device__ __forceinline__ float bf_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

template <int FIRST, int NT, size_t... Q>
__device__ __forceinline__ void mma_tiles16(float (&acc)[NT][4], const uint32_t (&f)[8][2],
                                            std::index_sequence<Q...>) {
  (mma_bf16_f32(acc[Q], f[2 * std::integral_constant<int, tile_row16(FIRST + (int)Q)>::value],
                f[2 * std::integral_constant<int, tile_row16(FIRST + (int)Q)>::value + 1],
                f[std::integral_constant<int, tile_col16(FIRST + (int)Q)>::value]),
   ...);
}

// Accumulates a warp's tiles over the entries of a task.  A warp of a square (PART >= 0): its
// tiles PART * NT .. of the square of components 64 half .., and blocks PART * NB .. of the
// right-hand side (rhs_s, by component).  PART = -1: the tiles across, blocks 8 + 2 half and
// 9 + 2 half against 0 .. 7, whose row operand is word `half` of the second 64 components.
template <int KP, int PART>
__device__ __forceinline__ void gram16(const SampleParams& p, const RowTask& tk, float wscale,
                                       int half, float (&acc)[Wide<KP, true>::NT][4],
                                       double* rhs_s) {
  constexpr int NT = Wide<KP, true>::NT, NB = KP == 64 ? 2 : 4;
  constexpr bool ACROSS = PART < 0;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  // 8 components a vector
  const uint4* other = reinterpret_cast<const uint4*>(p.other) + (ACROSS ? 0 : 8 * half) + g;
  const uint32_t* other_row = reinterpret_cast<const uint32_t*>(p.other) + 32 + 4 * g + half;
  float racc[NB] = {};
  auto load_chunk = [&](int off, int& c, float& w) {
    const bool in = off + lane < tk.len;
    const uint2 e = in ? p.packed[tk.begin + off + lane] : make_uint2(0u, 0u);
    c = (int)e.x;
    w = in ? __uint_as_float(e.y) * wscale : 0.f;
  };
  // entries 2t, 2t + 1, 2t + 8, 2t + 9 of a step of 16, two steps
  uint4 raw[2][4];
  uint32_t raw_row[2][4];
  auto gather = [&](int stage, int c_chunk, int upper, int off) {
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int at = 16 * upper + 2 * t + (e & 1) + 8 * (e >> 1);
      const int col = __shfl_sync(0xffffffffu, c_chunk, at);
      const bool ok = off + at < tk.len;
      raw[stage][e] = ok ? __ldg(other + (size_t)col * (KP / 8)) : make_uint4(0u, 0u, 0u, 0u);
      if constexpr (ACROSS) raw_row[stage][e] = ok ? __ldg(other_row + (size_t)col * (KP / 2)) : 0u;
    }
  };
  int c_cur, c_nxt = 0;
  float w_cur, w_nxt = 0.f;
  load_chunk(0, c_cur, w_cur);
  gather(0, c_cur, 0, 0);
  for (int off = 0; off < tk.len; off += 32) {
    load_chunk(off + 32, c_nxt, w_nxt);
#pragma unroll
    for (int u = 0; u < 2; u++) {
      if (off + 16 * u < tk.len) {
        if (u == 0) gather(1, c_cur, 1, off);
        else gather(0, c_nxt, 0, off + 32);
        uint32_t f[8][2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const uint4 x = raw[u][2 * k], y = raw[u][2 * k + 1];
          f[0][k] = pair_lo(x.x, y.x);
          f[1][k] = pair_hi(x.x, y.x);
          f[2][k] = pair_lo(x.y, y.y);
          f[3][k] = pair_hi(x.y, y.y);
          f[4][k] = pair_lo(x.z, y.z);
          f[5][k] = pair_hi(x.z, y.z);
          f[6][k] = pair_lo(x.w, y.w);
          f[7][k] = pair_hi(x.w, y.w);
        }
        if constexpr (ACROSS) {
          uint32_t lo[2], hi[2];
#pragma unroll
          for (int k = 0; k < 2; k++) {
            lo[k] = pair_lo(raw_row[u][2 * k], raw_row[u][2 * k + 1]);
            hi[k] = pair_hi(raw_row[u][2 * k], raw_row[u][2 * k + 1]);
          }
#pragma unroll
          for (int b = 0; b < 8; b++) mma_bf16_f32(acc[b], lo, hi, f[b]);
        } else {
#pragma unroll
          for (int k = 0; k < 2; k++) {
            const float w0 = __shfl_sync(0xffffffffu, w_cur, 16 * u + 8 * k + 2 * t);
            const float w1 = __shfl_sync(0xffffffffu, w_cur, 16 * u + 8 * k + 2 * t + 1);
#pragma unroll
            for (int b = 0; b < NB; b++) {
              racc[b] = fmaf(bf_lo(f[PART * NB + b][k]), w0, racc[b]);
              racc[b] = fmaf(bf_hi(f[PART * NB + b][k]), w1, racc[b]);
            }
          }
          mma_tiles16<PART * NT>(acc, f, std::make_index_sequence<NT>{});
        }
      }
    }
    c_cur = c_nxt;
    w_cur = w_nxt;
  }
  if constexpr (!ACROSS) {
#pragma unroll
    for (int b = 0; b < NB; b++) {
      racc[b] += __shfl_xor_sync(0xffffffffu, racc[b], 1);
      racc[b] += __shfl_xor_sync(0xffffffffu, racc[b], 2);
      if (t == 0) rhs_s[64 * half + 8 * g + PART * NB + b] = (double)racc[b];
    }
  }
}

// ---- MM = Lambda + alpha G in F, the identity beyond K ----
template <typename F>
__device__ __forceinline__ F mm_value(const double* Lambda, int K, F alpha, F gram, int i, int j) {
  return i < K && j < K ? (F)Lambda[i + (size_t)j * K] + alpha * gram : (i == j ? (F)1 : (F)0);
}

template <int KP, bool DIAG, int NT>
__device__ __forceinline__ void store64(double* M, const double* Lambda, int K, double alpha,
                                        int r0, int c0, const double (&acc)[NT][2]) {
  using C = Wide<KP, false>;
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

// Tiles of the BF16 Gram by their linear index; each unordered pair of components is written
// once (the tile rows' two blocks against the tile's block, its own block by lower triangle).
template <typename F, int KP>
__device__ __forceinline__ void store16(F* M, const double* Lambda, int K, F alpha, int warp,
                                        const float (&acc)[Wide<KP, true>::NT][4]) {
  constexpr int NT = Wide<KP, true>::NT;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  auto comp = [](int blk, int e) { return 64 * (blk >> 3) + 8 * e + (blk & 7); };
#pragma unroll
  for (int q = 0; q < NT; q++) {
    int b_row, bj;
    if (!tile16<KP>(warp, q, b_row, bj)) break;
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int bi = b_row + (e >> 1);
      const int i = comp(bi, g), j = comp(bj, 2 * t + (e & 1));
      if (bi > bj || (bi == bj && i >= j)) {
        const int hi = max(i, j), lo = min(i, j);
        M[elem_at(hi, lo)] = mm_value<F>(Lambda, K, alpha, (F)acc[q][e], hi, lo);
      }
    }
  }
}

// The FP64 redo of the mixed path, kept out of line for its registers.
template <int KP, int T>
__device__ __noinline__ bool wide_factor_redo(double* M, double* y, double* Di,
                                              const double* diag0, int nb, int tid, int grp,
                                              volatile int* bad) {
  return wide_factor<double, KP, T>(M, y, Di, diag0, nb, 0.0, tid, grp, bad);
}

template <int KP, int G, bool MIXED>
__global__ void __launch_bounds__(Wide<KP, MIXED>::T* G, (KP == 64 ? 4 : 2) / G)
    k_sample_wide(const SampleParams p) {
  using C = Wide<KP, MIXED>;
  using Acc = typename C::Acc;
  constexpr int T = C::T, NT = C::NT, AE = C::AE;
  extern __shared__ __align__(16) double smem_w[];
  double* lmu_s = smem_w;
  const int grp = threadIdx.x / T, tid = threadIdx.x % T;
  const int warp = tid >> 5, lane = tid & 31;
  double* M = smem_w + C::kCtaDoubles + (size_t)grp * C::kGroupDoubles;
  double* Di = M + (size_t)C::TRI * 64;
  double* rhs_s = Di + (size_t)C::NB * 64;  // Gram rhs, then the factor's y
  double* z_s = rhs_s + KP;
  double* x_s = z_s + KP;
  double* diag_s = x_s + KP;
  volatile int* bad = reinterpret_cast<volatile int*>(diag_s + KP);
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
  const float wscale = (float)packed_scale(p);
  int ti = bcast[0];
  while (ti < ntasks) {
    const RowTask tk = p.tasks[ti];
    int ti_next = 0;  // claimed early: its latency passes behind this row
    if (tid == 0) ti_next = (int)atomicAdd(&p.ctl->queue[p.qslot], 1u);
    Acc acc[NT][AE];
#pragma unroll
    for (int q = 0; q < NT; q++)
#pragma unroll
      for (int e = 0; e < AE; e++) acc[q][e] = (Acc)0;

    if constexpr (MIXED) {
      if constexpr (KP == 64) {
        switch (warp) {
          case 0: gram16<KP, 0>(p, tk, wscale, 0, acc, rhs_s); break;
          case 1: gram16<KP, 1>(p, tk, wscale, 0, acc, rhs_s); break;
          case 2: gram16<KP, 2>(p, tk, wscale, 0, acc, rhs_s); break;
          default: gram16<KP, 3>(p, tk, wscale, 0, acc, rhs_s); break;
        }
      } else {
        if (warp < 4) gram16<KP, -1>(p, tk, wscale, warp, acc, rhs_s);
        else if (warp & 1) gram16<KP, 1>(p, tk, wscale, (warp - 4) >> 1, acc, rhs_s);
        else gram16<KP, 0>(p, tk, wscale, (warp - 4) >> 1, acc, rhs_s);
      }
    } else {
      const Part64 part = part_of<KP>(warp);
      if (part.diag) gram64<KP, true>(p, tk, alpha, part.r0, part.c0, acc, rhs_s);
      else gram64<KP, false>(p, tk, alpha, part.r0, part.c0, acc, rhs_s);
    }

    bool finish = true;
    if (tk.nparts > 1) {  // a part of a split row: the last part to arrive adds them in order
      constexpr size_t kSlot = (size_t)KP * KP + KP;
      static_assert((size_t)C::W * NT * AE * 32 <= (size_t)KP * KP, "scratch slot too small");
      const size_t at = ((size_t)warp * NT * 32 + lane) * AE;
      double* sp = p.scratch + (size_t)(tk.slot + tk.part) * kSlot;
#pragma unroll
      for (int q = 0; q < NT; q++)
#pragma unroll
        for (int e = 0; e < AE; e += 2)
          *reinterpret_cast<double2*>(sp + at + q * 32 * AE + e) =
              make_double2((double)acc[q][e], (double)acc[q][e + 1]);
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
        for (int q = 0; q < NT; q++)
#pragma unroll
          for (int e = 0; e < AE; e += 2) {
            double a = 0.0, b = 0.0;
            for (int part = 0; part < tk.nparts; part++) {
              const double2 v = __ldcg(reinterpret_cast<const double2*>(
                  s0 + (size_t)part * kSlot + at + q * 32 * AE + e));
              a += v.x;
              b += v.y;
            }
            acc[q][e] = (Acc)a;
            acc[q][e + 1] = (Acc)b;
          }
        if (tid < KP) {
          double r = 0.0;
          for (int part = 0; part < tk.nparts; part++)
            r += __ldcg(s0 + (size_t)part * kSlot + KP * KP + tid);
          rhs_s[tid] = (double)(Acc)r;
        }
        if (tid == 0) p.split_cnt[tk.split] = 0u;
      }
    }

    if (finish) {
      const int row = tk.row;
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
      } else {
        group_sync<T>(grp);
        if (tid < KP) lm = lmu_s[tid];
      }
      const double rr = tid < KP ? rhs_s[tid] + lm : 0.0;
      if (tid == 0) *bad = 0;
      bool done = false;
      if constexpr (MIXED) {
        float* Mf = reinterpret_cast<float*>(M);
        float* Dif = reinterpret_cast<float*>(Di);
        float* yf = reinterpret_cast<float*>(x_s);  // x_s holds y and x
        float* xf = yf + KP;
        float* df = reinterpret_cast<float*>(diag_s);
        group_sync<T>(grp);  // x_s was the prior mean
        store16<float, KP>(Mf, p.Lambda, K, (float)alpha, warp, acc);
        if (tid < KP) yf[tid] = (float)rr;
        group_sync<T>(grp);
        if (tid < KP) df[tid] = Mf[elem_at(tid, tid)];
        group_sync<T>(grp);
        done = wide_factor<float, KP, T>(Mf, yf, Dif, df, nb, 0x1p-20f, tid, grp, bad);
        if (done) {
          if (tid < 8 * nb) yf[tid] += (float)z_s[tid];
          group_sync<T>(grp);
          wide_back<float, KP, T>(Mf, yf, Dif, xf, nb, tid, grp);
          if (tid < K) {
            p.out_f32[(size_t)row * KP + tid] = xf[tid];
            store_copy(p, (size_t)row * KP + tid, xf[tid]);
          }
        } else {
          group_sync<T>(grp);  // every thread has seen the flag
          if (tid == 0) {
            atomicAdd(&p.ctl->retries[p.mode], 1u);
            *bad = 0;
          }
        }
      }
      if (!done) {
        group_sync<T>(grp);
        if constexpr (MIXED) {
          store16<double, KP>(M, p.Lambda, K, alpha, warp, acc);
        } else {
          const Part64 part = part_of<KP>(warp);
          if (part.diag) store64<KP, true>(M, p.Lambda, K, alpha, part.r0, part.c0, acc);
          else store64<KP, false>(M, p.Lambda, K, alpha, part.r0, part.c0, acc);
        }
        if (tid < KP) rhs_s[tid] = rr;
        group_sync<T>(grp);
        if (tid < KP) diag_s[tid] = M[elem_at(tid, tid)];
        group_sync<T>(grp);
        bool ok;
        if constexpr (MIXED)
          ok = wide_factor_redo<KP, T>(M, rhs_s, Di, diag_s, nb, tid, grp, bad);
        else
          ok = wide_factor<double, KP, T>(M, rhs_s, Di, diag_s, nb, 0.0, tid, grp, bad);
        if (ok) {
          if (tid < 8 * nb) rhs_s[tid] += z_s[tid];
          group_sync<T>(grp);
          wide_back<double, KP, T>(M, rhs_s, Di, x_s, nb, tid, grp);
          if (tid < K) {
            if constexpr (MIXED) {
              p.out_f32[(size_t)row * KP + tid] = (float)x_s[tid];
              store_copy(p, (size_t)row * KP + tid, (float)x_s[tid]);
            } else {
              p.out_f64[(size_t)row * KP + tid] = x_s[tid];
            }
          }
        } else if (tid == 0) {
          atomicOr(&p.ctl->status, kStatCholFail);
          atomicCAS(&p.ctl->bad_row, -1, row);
        }
      }
    }
    if (tid == 0) bcast[0] = ti_next;
    group_sync<T>(grp);
    ti = bcast[0];
  }
}

template <int KP, int G, bool MIXED>
void launch_wide(const SampleParams& p, cudaStream_t s, int num_sms) {
  using C = Wide<KP, MIXED>;
  auto kern = k_sample_wide<KP, G, MIXED>;
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

void launch_sample_wide(const SampleParams& p, int KP, bool mixed, cudaStream_t s, int num_sms,
                        int groups) {
  if (KP == 128)
    return mixed ? launch_wide<128, 1, true>(p, s, num_sms)
                 : launch_wide<128, 1, false>(p, s, num_sms);
  if (groups == 1)
    return mixed ? launch_wide<64, 1, true>(p, s, num_sms)
                 : launch_wide<64, 1, false>(p, s, num_sms);
  return mixed ? launch_wide<64, 2, true>(p, s, num_sms) : launch_wide<64, 2, false>(p, s, num_sms);
}

}  // namespace mg
