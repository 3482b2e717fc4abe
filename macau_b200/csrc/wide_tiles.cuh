// FP64 and FP32 triangular matrices of 33 to 128 rows in shared memory as 8 x 8 tiles, for a group of
// warps: the panel Cholesky factor with a right-hand side, the backward substitution, and the split
// of a Gram's lower-triangle tiles over the warps (sample_wide.cu, hyper_wide.cu).
#pragma once
#include "common.cuh"
#include "mma_tiles.cuh"
#include "warp_finish.cuh"

namespace mg {

// Barrier of a row group.  bar.sync counts whole warps, so each warp's lanes meet first; every
// thread of the group reaches every call.
template <int T>
__device__ __forceinline__ void group_sync(int g) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(T) : "memory");
}

// Position of element (r, c) inside an 8 x 8 tile: the two halves of rows 2, 3, 6 and 7 swapped,
// so that the eight rows' reads of four columns touch different banks.
__device__ __forceinline__ int tile_pos(int r, int c) { return r * 8 + (c ^ ((r & 2) << 1)); }
__device__ __forceinline__ int tile_at(int bi, int bj) { return (bi * (bi + 1) / 2 + bj) * 64; }
__device__ __forceinline__ int elem_at(int i, int j) {  // i >= j
  return tile_at(i >> 3, j >> 3) + tile_pos(i & 7, j & 7);
}

// The 8 values of row r of a tile.
template <typename F>
__device__ __forceinline__ void load_row8(const F* tile, int r, F (&v)[8]) {
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const Vec4<F> q = lds4(tile + r * 8 + 4 * (h ^ ((r >> 1) & 1)));
#pragma unroll
    for (int u = 0; u < 4; u++) v[4 * h + u] = q.v[u];
  }
}
template <typename F>
__device__ __forceinline__ void store_row8(F* tile, int r, const F (&v)[8]) {
#pragma unroll
  for (int c = 0; c < 8; c++) tile[tile_pos(r, c)] = v[c];
}

// ---- FP64 Grams: lower-triangle tiles by warp (4 warps at 64 components, 8 at 128) ----
// Tiles of a rectangle warp: blocks r0 .. r0 + RB - 1 against c0 .. c0 + 3; of a diagonal warp:
// the lower triangles of the squares of blocks d0 + 4s .. d0 + 4s + 3.
struct Part64 {
  bool diag;
  int r0, c0;
};
template <int KP>
__device__ __forceinline__ Part64 part_of(int warp) {
  if constexpr (KP == 64) {
    if (warp < 2) return {true, 4 * warp, 4 * warp};
    return {false, 4 + 2 * (warp - 2), 0};
  } else {
    if (warp >= 6) return {true, 8 * (warp - 6), 8 * (warp - 6)};
    const int I = warp == 0 ? 1 : (warp < 3 ? 2 : 3);
    return {false, 4 * I, 4 * (warp - I * (I - 1) / 2)};
  }
}

// The n blocks of one entry from their first components at src (component g of each).
template <int N>
__device__ __forceinline__ void gather64(double (&f)[N], const double* src, bool ok) {
#pragma unroll
  for (int b = 0; b < N; b++) f[b] = ok ? __ldg(src + 8 * b) : 0.0;
}

// ---- factor and solves over the tiles ----
// Tile (bi, pn) -= sum_{k < pn} L(bi, k) L(pn, k)^T by one warp (FP64: two accumulators, so that
// consecutive products overlap).
__device__ __forceinline__ void update_tile(double* M, int bi, int pn, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const int p0 = tile_pos(g, t), p1 = tile_pos(g, t + 4);
  const double* A = M + tile_at(bi, 0);
  const double* B = M + tile_at(pn, 0);
  double2* c = reinterpret_cast<double2*>(M + tile_at(bi, pn) + tile_pos(g, 2 * t));
  double2 v = *c, w = make_double2(0.0, 0.0);
  int k = 0;
#pragma unroll 2
  for (; k + 1 < pn; k += 2) {
    const double a0 = -A[64 * k + p0], a1 = -A[64 * k + p1];
    const double a2 = -A[64 * k + 64 + p0], a3 = -A[64 * k + 64 + p1];
    const double b0 = B[64 * k + p0], b1 = B[64 * k + p1];
    const double b2 = B[64 * k + 64 + p0], b3 = B[64 * k + 64 + p1];
    mma_f64(v.x, v.y, a0, b0);
    mma_f64(w.x, w.y, a2, b2);
    mma_f64(v.x, v.y, a1, b1);
    mma_f64(w.x, w.y, a3, b3);
  }
  if (k < pn) {
    mma_f64(v.x, v.y, -A[64 * k + p0], B[64 * k + p0]);
    mma_f64(w.x, w.y, -A[64 * k + p1], B[64 * k + p1]);
  }
  *c = make_double2(v.x + w.x, v.y + w.y);
}
__device__ __forceinline__ void update_tile(float* M, int bi, int pn, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const float* A = M + tile_at(bi, 0);
  const float* B = M + tile_at(pn, 0);
  float2* c = reinterpret_cast<float2*>(M + tile_at(bi, pn) + tile_pos(g, 2 * t));
  float2 v = *c;
#pragma unroll 2
  for (int k = 0; k < pn; k++) {
    float a[8], b0[8], b1[8];
    load_row8(A + 64 * k, g, a);
    load_row8(B + 64 * k, 2 * t, b0);
    load_row8(B + 64 * k, 2 * t + 1, b1);
#pragma unroll
    for (int q = 0; q < 8; q++) {
      v.x = fmaf(-a[q], b0[q], v.x);
      v.y = fmaf(-a[q], b1[q], v.y);
    }
  }
  *c = v;
}

// Factorises MM (nb blocks) in place by panels of 8 columns, left-looking, y (the right-hand side)
// along with it, and leaves the transposed inverse of each diagonal tile in Di (a tile per panel,
// for the backward substitution: eight more rows, those of the identity, go through the panel's
// solve).  A pivot that is not positive, or not above
// rel_floor times its original diagonal, fails the group (all threads return false).
//   Per panel: a warp per tile subtracts the products of the panels before it (a right-looking
//   update of every trailing tile per panel took 1,400 cycles a panel at K = 128, three times
//   this: each product loaded and stored its tile); barrier; every thread that owns a row of the
//   panel factors the diagonal tile for itself and solves its row; barrier.
template <typename F, int KP, int T>
__device__ __forceinline__ bool wide_factor(F* M, F* y, F* Di, const F* diag0, int nb,
                                            F rel_floor, int tid, int grp, volatile int* bad) {
  const int warp = tid >> 5, lane = tid & 31;
  for (int pn = 0; pn < nb; pn++) {
    if (pn > 0) {
      for (int bi = pn + warp; bi < nb; bi += T / 32) update_tile(M, bi, pn, lane);
      // y's components from the panel on, by the panel before
      const int j = 8 * pn + tid;
      if (j < 8 * nb) {
        F v[8], s = y[j];
        load_row8(M + tile_at(j >> 3, pn - 1), j & 7, v);
#pragma unroll
        for (int c = 0; c < 8; c++) s = mfma(-v[c], y[8 * pn - 8 + c], s);
        y[j] = s;
      }
      group_sync<T>(grp);
    }
    // rows 8 pn .. of the panel, the identity's, then y: one thread each
    const int rows = 8 * (nb - pn);
    F* own = tid < rows ? M + tile_at(pn + (tid >> 3), pn) : Di + 64 * pn;
    F x[8];
    if (tid <= rows + 8) {
      const F* D = M + tile_at(pn, pn);
      F l[8][8];
#pragma unroll
      for (int i = 0; i < 8; i++) load_row8(D, i, l[i]);
      if (tid == rows + 8) {
#pragma unroll
        for (int c = 0; c < 8; c++) x[c] = y[8 * pn + c];
      } else if (tid >= rows) {
#pragma unroll
        for (int c = 0; c < 8; c++) x[c] = tid - rows == c ? (F)1 : (F)0;
      } else {
        load_row8(own, tid & 7, x);
      }
      bool ok = true;
#pragma unroll
      for (int c = 0; c < 8; c++) {
        const F d = l[c][c];
        ok = ok && d > (F)0 && d > rel_floor * diag0[8 * pn + c];
        const F r = mrsqrt(d);
#pragma unroll
        for (int i = c + 1; i < 8; i++) l[i][c] *= r;
        x[c] *= r;
#pragma unroll
        for (int j = c + 1; j < 8; j++) {
#pragma unroll
          for (int i = j; i < 8; i++) l[i][j] = mfma(-l[i][c], l[j][c], l[i][j]);
          x[j] = mfma(-x[c], l[j][c], x[j]);
        }
      }
      if (!ok && tid == 0) *bad = 1;
      if (tid == rows + 8) {
#pragma unroll
        for (int c = 0; c < 8; c++) y[8 * pn + c] = x[c];
      } else if (tid >= 8) {
        store_row8(own, tid & 7, x);
      }
    }
    group_sync<T>(grp);
    if (*bad) return false;
    // the factored diagonal tile's rows only now: every owner has read the tile
    if (tid < 8) store_row8(own, tid, x);
  }
  group_sync<T>(grp);
  return true;
}

// x = L^{-T} b over the panels from the last, b in y (overwritten), Di the diagonal tiles'
// transposed inverses; one barrier a panel.  Each warp forms the panel's eight x for itself.
template <typename F, int KP, int T>
__device__ __forceinline__ void wide_back(const F* M, F* y, const F* Di, F* x, int nb, int tid,
                                          int grp) {
  const int warp = tid >> 5, r = tid & 7;
  for (int pn = nb - 1; pn >= 0; pn--) {
    if (warp == 0 || 32 * warp < 8 * pn) {
      F d[8], b[8], p[8];
      load_row8(Di + 64 * pn, r, d);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const Vec4<F> q = lds4(y + 8 * pn + 4 * h);
#pragma unroll
        for (int u = 0; u < 4; u++) b[4 * h + u] = q.v[u];
      }
      const bool on = tid < 8 * pn;
      const F* P = M + tile_at(pn, on ? tid >> 3 : 0);
#pragma unroll
      for (int c = 0; c < 8; c++) p[c] = P[tile_pos(c, r)];
      F s = on ? y[tid] : (F)0, u0 = (F)0, u1 = (F)0, s1 = (F)0;
#pragma unroll
      for (int c = 0; c < 8; c += 2) {
        u0 = mfma(d[c], b[c], u0);
        u1 = mfma(d[c + 1], b[c + 1], u1);
      }
      const F xr = u0 + u1;
#pragma unroll
      for (int c = 0; c < 8; c += 2) {
        s = mfma(-p[c], wshfl(xr, c), s);
        s1 = mfma(-p[c + 1], wshfl(xr, c + 1), s1);
      }
      if (on) y[tid] = s + s1;
      if (tid < 8) x[8 * pn + tid] = xr;
    }
    group_sync<T>(grp);
  }
}

}  // namespace mg
