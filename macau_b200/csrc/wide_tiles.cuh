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
// Trailing tiles (bi, bj) -= P_bi P_bj^T of panel pn, P the panel's tiles: the pairs b <= a of the n1
// block rows below it, the q-th of them to warp q mod W.  The FP64 form takes U tiles at a time,
// so that their loads and products overlap.
template <int W, int U>
__device__ __forceinline__ void trail_tiles(double* M, const unsigned char* tri, int pn, int q0,
                                            int lane) {
  const int g = lane >> 2, t = lane & 3;
  const int p0 = tile_pos(g, t), p1 = tile_pos(g, t + 4), pc = tile_pos(g, 2 * t);
  double2* c[U];
  double2 v[U];
  double a[U][2], b[U][2];
#pragma unroll
  for (int u = 0; u < U; u++) {
    const int ab = tri[q0 + u * W];
    const int bi = pn + 1 + (ab >> 4), bj = pn + 1 + (ab & 15);
    const double* Pi = M + tile_at(bi, pn);
    const double* Pj = M + tile_at(bj, pn);
    c[u] = reinterpret_cast<double2*>(M + tile_at(bi, bj) + pc);
    v[u] = *c[u];
    a[u][0] = -Pi[p0];
    a[u][1] = -Pi[p1];
    b[u][0] = Pj[p0];
    b[u][1] = Pj[p1];
  }
#pragma unroll
  for (int k = 0; k < 2; k++)
#pragma unroll
    for (int u = 0; u < U; u++) mma_f64(v[u].x, v[u].y, a[u][k], b[u][k]);
#pragma unroll
  for (int u = 0; u < U; u++) *c[u] = v[u];
}
template <int W>
__device__ __forceinline__ void trail(double* M, const unsigned char* tri, int pn, int n1, int warp,
                                      int lane) {
  const int n = n1 * (n1 + 1) / 2;
  int q = warp;
  for (; q + 2 * W < n; q += 3 * W) trail_tiles<W, 3>(M, tri, pn, q, lane);
  for (; q < n; q += W) trail_tiles<W, 1>(M, tri, pn, q, lane);
}
template <int W>
__device__ __forceinline__ void trail(float* M, const unsigned char* tri, int pn, int n1, int warp,
                                      int lane) {
  const int g = lane >> 2, t = lane & 3, n = n1 * (n1 + 1) / 2;
  for (int q = warp; q < n; q += W) {
    const int bi = pn + 1 + (tri[q] >> 4), bj = pn + 1 + (tri[q] & 15);
    float a[8], b0[8], b1[8];
    load_row8(M + tile_at(bi, pn), g, a);
    load_row8(M + tile_at(bj, pn), 2 * t, b0);
    load_row8(M + tile_at(bj, pn), 2 * t + 1, b1);
    float2* c = reinterpret_cast<float2*>(M + tile_at(bi, bj) + tile_pos(g, 2 * t));
    float2 v = *c;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      v.x = fmaf(-a[k], b0[k], v.x);
      v.y = fmaf(-a[k], b1[k], v.y);
    }
    *c = v;
  }
}

// Factorises MM (nb blocks) in place by panels, y (the right-hand side) along with it, and leaves
// 1 / L(j, j) in rinv.  A pivot that is not positive, or not above rel_floor times its original
// diagonal, fails the group (all threads return false).  tri[q] = (a << 4) | b, the q-th pair
// b <= a.
template <typename F, int KP, int T>
__device__ __forceinline__ bool wide_factor(F* M, F* y, F* rinv, const F* diag0, int nb,
                                            const unsigned char* tri, F rel_floor, int tid,
                                            int grp, volatile int* bad) {
  const int warp = tid >> 5, lane = tid & 31;
  for (int pn = 0; pn < nb; pn++) {
    // rows 8 pn .. of the panel, then y: one thread each
    const int rows = 8 * (nb - pn);
    F* own = M + tile_at(pn + (tid >> 3), pn);  // the thread's tile when tid < rows
    F x[8];
    if (tid <= rows) {
      const F* D = M + tile_at(pn, pn);
      F l[8][8];
#pragma unroll
      for (int i = 0; i < 8; i++) load_row8(D, i, l[i]);
      if (tid == rows) {
#pragma unroll
        for (int c = 0; c < 8; c++) x[c] = y[8 * pn + c];
      } else {
        load_row8(own, tid & 7, x);
      }
      bool ok = true;
#pragma unroll
      for (int c = 0; c < 8; c++) {
        const F d = l[c][c];
        ok = ok && d > (F)0 && d > rel_floor * diag0[8 * pn + c];
        const F r = mrsqrt(d);
        if (tid == 0) rinv[8 * pn + c] = r;
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
      if (tid == rows) {
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
    // trailing tiles, and y's remaining components
    const int n1 = nb - pn - 1;
    trail<T / 32>(M, tri, pn, n1, warp, lane);
    const int j = 8 * (pn + 1) + tid;
    if (j < 8 * nb) {
      F v[8], s = y[j];
      load_row8(M + tile_at(j >> 3, pn), j & 7, v);
#pragma unroll
      for (int c = 0; c < 8; c++) s = mfma(-v[c], y[8 * pn + c], s);
      y[j] = s;
    }
    group_sync<T>(grp);
  }
  return true;
}

// x = L^{-T} b over the panels from the last, b in y (overwritten), one barrier each.
template <typename F, int KP, int T>
__device__ __forceinline__ void wide_back(const F* M, F* y, const F* rinv, F* x, int nb, int tid,
                                          int grp) {
  for (int pn = nb - 1; pn >= 0; pn--) {
    if (tid < 8 * pn || tid == T - 1) {
      // every thread solves the panel's 8 x 8 system for itself
      F b[8];
#pragma unroll
      for (int c = 0; c < 8; c++) b[c] = y[8 * pn + c];
      const F* D = M + tile_at(pn, pn);
#pragma unroll
      for (int c = 7; c >= 0; c--) {
        F l[8];
        load_row8(D, c, l);
        b[c] *= rinv[8 * pn + c];
#pragma unroll
        for (int d = 0; d < c; d++) b[d] = mfma(-l[d], b[c], b[d]);
      }
      if (tid < 8 * pn) {
        const F* P = M + tile_at(pn, tid >> 3);
        F s = y[tid];
#pragma unroll
        for (int c = 0; c < 8; c++) s = mfma(-P[tile_pos(c, tid & 7)], b[c], s);
        y[tid] = s;
      } else {
#pragma unroll
        for (int c = 0; c < 8; c++) x[8 * pn + c] = b[c];
      }
    }
    group_sync<T>(grp);
  }
}

}  // namespace mg
