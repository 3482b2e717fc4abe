// Triangular matrices in shared memory as 8 x 8 tiles: the panel Cholesky factor with a right-hand
// side and the backward substitution, for a group of warps and up to 128 rows (sample_wide.cu,
// hyper_wide.cu) and for one warp and up to 32 (sample_mma.cu); the tiles' layout and scalar updates
// (sample_wide_mixed.cu); the split of a wide Gram's lower-triangle tiles over the warps.
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
__device__ __forceinline__ void store_row8(double* tile, int r, const double (&v)[8]) {
#pragma unroll
  for (int h = 0; h < 2; h++) {
    double2* d = reinterpret_cast<double2*>(tile + r * 8 + 4 * (h ^ ((r >> 1) & 1)));
    d[0] = make_double2(v[4 * h], v[4 * h + 1]);
    d[1] = make_double2(v[4 * h + 2], v[4 * h + 3]);
  }
}
__device__ __forceinline__ void store_row8(float* tile, int r, const float (&v)[8]) {
#pragma unroll
  for (int h = 0; h < 2; h++)
    *reinterpret_cast<float4*>(tile + r * 8 + 4 * (h ^ ((r >> 1) & 1))) =
        make_float4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
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
// Tile (bi, bj) -= sum_{k0 <= k < k1} L(bi, k) L(bj, k)^T by one warp.  FP64: two accumulators and
// the next pair's operands in flight, so that neither loads nor products wait for one another.
__device__ __forceinline__ void update_tile(double* M, int bi, int bj, int k0, int k1, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const int p0 = tile_pos(g, t), p1 = tile_pos(g, t + 4);
  const double* A = M + tile_at(bi, k0);
  const double* B = M + tile_at(bj, k0);
  double2* c = reinterpret_cast<double2*>(M + tile_at(bi, bj) + tile_pos(g, 2 * t));
  double2 v = *c, w = make_double2(0.0, 0.0);
  const int n = k1 - k0;
  double a[4] = {}, b[4] = {};
  auto fetch = [&](int k) {  // products k and k + 1 (the last one twice when n is odd)
    const int k2 = k + 1 < n ? 64 * (k + 1) : 64 * k;
    a[0] = A[64 * k + p0];
    a[1] = A[64 * k + p1];
    a[2] = A[k2 + p0];
    a[3] = A[k2 + p1];
    b[0] = -B[64 * k + p0];
    b[1] = -B[64 * k + p1];
    b[2] = -B[k2 + p0];
    b[3] = -B[k2 + p1];
  };
  if (n > 0) fetch(0);
  for (int k = 0; k < n; k += 2) {
    const double a0 = a[0], a1 = a[1], a2 = a[2], a3 = a[3];
    const double b0 = b[0], b1 = b[1], b2 = b[2], b3 = b[3];
    if (k + 2 < n) fetch(k + 2);
    mma_f64(v.x, v.y, a0, b0);
    if (k + 1 < n) mma_f64(w.x, w.y, a2, b2);
    mma_f64(v.x, v.y, a1, b1);
    if (k + 1 < n) mma_f64(w.x, w.y, a3, b3);
  }
  *c = make_double2(v.x + w.x, v.y + w.y);
}
// Scalar form (c -= sum over tiles A + k stride, B + k stride): one fused multiply-add per column, in
// column order.
template <typename F>
__device__ __forceinline__ void update_tile(F* tile, const F* A, const F* B, int k0, int k1,
                                            int stride, int lane) {
  const int g = lane >> 2, t = lane & 3;
  F* c = tile + tile_pos(g, 2 * t);
  F v0 = c[0], v1 = c[1];
#pragma unroll 2
  for (int k = k0; k < k1; k++) {
    F a[8], b0[8], b1[8];
    load_row8(A + stride * k, g, a);
    load_row8(B + stride * k, 2 * t, b0);
    load_row8(B + stride * k, 2 * t + 1, b1);
#pragma unroll
    for (int q = 0; q < 8; q++) {
      v0 = mfma(-a[q], b0[q], v0);
      v1 = mfma(-a[q], b1[q], v1);
    }
  }
  c[0] = v0;
  c[1] = v1;
}

// Factor of a diagonal tile by one warp: lanes 0-7 hold its rows (x[j], j <= lane, in; the factor's
// rows out), any other lane a row v that becomes v L^{-T}.  What a column needs of the other rows
// is shuffled before its pivot is known (unscaled), so the chain from pivot to pivot is one
// reciprocal square root, one product and one fma.  False when a pivot is not positive.
__device__ __forceinline__ bool diag_factor(double (&x)[8]) {
  bool ok = true;
  double d = wshfl(x[0], 0);
#pragma unroll
  for (int c = 0; c < 8; c++) {
    double w[8], v = 0.0;
#pragma unroll
    for (int j = c + 1; j < 8; j++) w[j] = wshfl(x[c], j);
    if (c < 7) v = wshfl(x[c + 1], c + 1);
    ok = ok & (d > 0.0);
    const double r = mrsqrt(d);
    if (c < 7) {
      const double l = w[c + 1] * r;
      d = fma(-l, l, v);
    }
    const double s = x[c] * (r * r);
    x[c] *= r;
#pragma unroll
    for (int j = c + 1; j < 8; j++) x[j] = fma(-s, w[j], x[j]);
  }
  return ok;
}

// Tile T <- T L^{-T}, Di the transposed inverse of L, by one warp.
__device__ __forceinline__ void solve_tile(double* T, const double* Di, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const double a0 = T[tile_pos(g, t)], a1 = T[tile_pos(g, t + 4)];
  double2 v = make_double2(0.0, 0.0);
  __syncwarp();
  mma_f64(v.x, v.y, a0, Di[tile_pos(t, g)]);
  mma_f64(v.x, v.y, a1, Di[tile_pos(t + 4, g)]);
  *reinterpret_cast<double2*>(T + tile_pos(g, 2 * t)) = v;
}

// Factorises MM (nb blocks) in place by panels of 8 columns, left-looking, y (the right-hand side)
// along with it, and leaves the transposed inverse of each diagonal tile in Di (a tile per panel).
// A pivot that is not positive fails the group (all threads return false).
//   Per panel: warp 0 subtracts the last panel's product from the diagonal tile and factors it, with
//   the identity's rows and y's among its lanes, while the other warps subtract all earlier
//   panels' from the tiles below and from the next diagonal tile; barrier; the tiles below times the
//   transposed inverse; barrier.  (Every row's owner factoring the diagonal tile for itself,
//   without the second step, took 2,800 cycles a panel at K = 64 in FP64: 244 FP64 instructions
//   a thread, in every warp.)
template <int T>
__device__ __forceinline__ bool wide_factor(double* M, double* y, double* Di, int nb, int tid,
                                            int grp, volatile int* bad) {
  constexpr int W = T / 32;
  const int warp = tid >> 5, lane = tid & 31;
  for (int pn = 0; pn < nb; pn++) {
    // y's components by the panel before: the panel's own by warp 0, the others by warps 1 ..
    const int j = warp == 0 ? 8 * pn + (lane & 7) : 8 * pn + 8 + tid - 32;
    double s = 0.0;
    if (pn > 0 && j < 8 * nb) {
      double v[8];
      load_row8(M + tile_at(j >> 3, pn - 1), j & 7, v);
      s = y[j];
      double s1 = 0.0;
#pragma unroll
      for (int c = 0; c < 8; c += 2) {
        s = fma(-v[c], y[8 * pn - 8 + c], s);
        s1 = fma(-v[c + 1], y[8 * pn - 7 + c], s1);
      }
      s += s1;
    }
    if (warp == 0) {
      if (pn > 0) {
        update_tile(M, pn, pn, pn - 1, pn, lane);
        if (lane < 8) y[j] = s;
      }
      __syncwarp();
      // lanes 0-7: the tile's rows, 8-15: the identity's, 16: y
      double* row = lane < 8 ? M + tile_at(pn, pn) : (lane < 16 ? Di + 64 * pn : y + 8 * pn);
      const int r = lane < 16 ? lane & 7 : 0;
      double x[8];
      if (lane < 8 || lane == 16) {
        load_row8(row, r, x);
      } else {
#pragma unroll
        for (int c = 0; c < 8; c++) x[c] = lane - 8 == c ? 1.0 : 0.0;
      }
      __syncwarp();
      const bool ok = diag_factor(x);
      if (lane <= 16) store_row8(row, r, x);
      if (!ok && lane == 0) *bad = 1;
    } else {
      if (pn > 0) {
        if (j < 8 * nb) y[j] = s;
        for (int bi = pn + warp; bi < nb; bi += W - 1) update_tile(M, bi, pn, 0, pn, lane);
        // the next diagonal tile, by the warp whose turn is next
        if (pn + 1 < nb && warp == 1 + (nb - pn - 1) % (W - 1))
          update_tile(M, pn + 1, pn + 1, 0, pn, lane);
      }
    }
    group_sync<T>(grp);
    if (*bad) return false;
    for (int bi = pn + 1 + warp; bi < nb; bi += W)
      solve_tile(M + tile_at(bi, pn), Di + 64 * pn, lane);
    group_sync<T>(grp);
  }
  return true;
}

// x = L^{-T} b over the panels from the last, b in y (overwritten), Di the diagonal tiles'
// transposed inverses; one barrier a panel.  Each warp forms the panel's eight x for itself.
template <int T>
__device__ __forceinline__ void wide_back(const double* M, double* y, const double* Di, double* x,
                                          int nb, int tid, int grp) {
  const int warp = tid >> 5, r = tid & 7;
  for (int pn = nb - 1; pn >= 0; pn--) {
    if (warp == 0 || 32 * warp < 8 * pn) {
      double d[8], b[8], p[8];
      load_row8(Di + 64 * pn, r, d);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const Vec4<double> q = lds4(y + 8 * pn + 4 * h);
#pragma unroll
        for (int u = 0; u < 4; u++) b[4 * h + u] = q.v[u];
      }
      const bool on = tid < 8 * pn;
      const double* P = M + tile_at(pn, on ? tid >> 3 : 0);
#pragma unroll
      for (int c = 0; c < 8; c++) p[c] = P[tile_pos(c, r)];
      double s = on ? y[tid] : 0.0, u0 = 0.0, u1 = 0.0, s1 = 0.0;
#pragma unroll
      for (int c = 0; c < 8; c += 2) {
        u0 = fma(d[c], b[c], u0);
        u1 = fma(d[c + 1], b[c + 1], u1);
      }
      const double xr = u0 + u1;
#pragma unroll
      for (int c = 0; c < 8; c += 2) {
        s = fma(-p[c], wshfl(xr, c), s);
        s1 = fma(-p[c + 1], wshfl(xr, c + 1), s1);
      }
      if (on) y[tid] = s + s1;
      if (tid < 8) x[8 * pn + tid] = xr;
    }
    group_sync<T>(grp);
  }
}

// Block column bj of Y = L^{-1} below its diagonal tile, by one warp: Y(i, j) = -Y(i, i) sum_k
// L(i, k) Y(k, j).  Y's diagonal tiles are in place.
__device__ __forceinline__ void inverse_column(const double* L, double* Y, int bj, int nb,
                                               int lane) {
  const int g = lane >> 2, t = lane & 3;
  for (int bi = bj + 1; bi < nb; bi++) {
    double s[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    for (int k = bj; k < bi; k++) {
      const double* A = L + tile_at(bi, k);
      const double* B = Y + tile_at(k, bj);
      mma_f64(s[0][0], s[0][1], A[tile_pos(g, t)], B[tile_pos(t, g)]);
      mma_f64(s[1][0], s[1][1], A[tile_pos(g, t + 4)], B[tile_pos(t + 4, g)]);
    }
    double* out = Y + tile_at(bi, bj);
    *reinterpret_cast<double2*>(out + tile_pos(g, 2 * t)) =
        make_double2(s[0][0] + s[1][0], s[0][1] + s[1][1]);
    __syncwarp();
    const double* A = Y + tile_at(bi, bi);
    const double b0 = out[tile_pos(t, g)], b1 = out[tile_pos(t + 4, g)];
    double2 v = make_double2(0.0, 0.0);
    __syncwarp();
    mma_f64(v.x, v.y, -A[tile_pos(g, t)], b0);
    mma_f64(v.x, v.y, -A[tile_pos(g, t + 4)], b1);
    *reinterpret_cast<double2*>(out + tile_pos(g, 2 * t)) = v;
    __syncwarp();
  }
}

// ---- the same for one warp and at most 32 rows (NB <= 4 blocks): factor, forward substitution,
// the draw z added, backward substitution.  y: right-hand side by component, overwritten by x.
// False when a pivot is not positive.
//   What bounds it: the shared-memory pipe (loads, stores and shuffles), so the vectors go through
// the matrix instruction as well, as a row that every lane group repeats: a tile's fragment costs
// two conflict-free loads where a row or a column per lane cost eight conflicting ones.
template <int NB>
__device__ __forceinline__ bool warp_tiles_solve(double* M, double* Di, double* y, int nb, double z,
                                                 int lane) {
  const int g = lane >> 2, t = lane & 3, r8 = lane & 7;
  const int p0 = tile_pos(g, t), p1 = tile_pos(g, t + 4), pc = tile_pos(g, 2 * t);
  const int q0 = tile_pos(t, g), q1 = tile_pos(t + 4, g);
  auto pair_at = [&](double* v, int b) { return reinterpret_cast<double2*>(v + 8 * b + 2 * t); };
#pragma unroll 1
  for (int pn = 0; pn < nb; pn++) {
    if (pn > 0) {
      // the panel's tiles and y's components by all panels before it
      double2 acc[NB], ya = *pair_at(y, pn);
#pragma unroll
      for (int bi = 1; bi < NB; bi++)
        if (bi >= pn && bi < nb) acc[bi] = *reinterpret_cast<double2*>(M + tile_at(bi, pn) + pc);
      for (int k = 0; k < pn; k++) {
        const double* B = M + tile_at(pn, k);
        const double b0 = -B[p0], b1 = -B[p1];
        mma_f64(ya.x, ya.y, y[8 * k + t], b0);
#pragma unroll
        for (int bi = 1; bi < NB; bi++)
          if (bi >= pn && bi < nb) {
            const double* A = M + tile_at(bi, k);
            mma_f64(acc[bi].x, acc[bi].y, A[p0], b0);
            mma_f64(acc[bi].x, acc[bi].y, A[p1], b1);
          }
        mma_f64(ya.x, ya.y, y[8 * k + 4 + t], b1);
      }
      __syncwarp();
      if (g == 0) *pair_at(y, pn) = ya;
#pragma unroll
      for (int bi = 1; bi < NB; bi++)
        if (bi >= pn && bi < nb) *reinterpret_cast<double2*>(M + tile_at(bi, pn) + pc) = acc[bi];
      __syncwarp();
    }
    // lanes 0-7: the diagonal tile's rows, 8-15: the identity's, 16: y
    double* row = lane < 8 ? M + tile_at(pn, pn) : (lane < 16 ? Di + 64 * pn : y + 8 * pn);
    const int r = lane < 16 ? r8 : 0;
    double x[8];
    if (lane < 8 || lane == 16) {
      load_row8(row, r, x);
    } else {
#pragma unroll
      for (int c = 0; c < 8; c++) x[c] = lane - 8 == c ? 1.0 : 0.0;
    }
    if (!diag_factor(x)) return false;
    if (lane >= 8 && lane <= 16) store_row8(row, r, x);
    __syncwarp();
    if (pn + 1 < nb) {
      const double d0 = Di[64 * pn + q0], d1 = Di[64 * pn + q1];
      double2 acc[NB];
#pragma unroll
      for (int bi = 1; bi < NB; bi++)
        if (bi > pn && bi < nb) {
          const double* T = M + tile_at(bi, pn);
          acc[bi] = make_double2(0.0, 0.0);
          mma_f64(acc[bi].x, acc[bi].y, T[p0], d0);
          mma_f64(acc[bi].x, acc[bi].y, T[p1], d1);
        }
      __syncwarp();
#pragma unroll
      for (int bi = 1; bi < NB; bi++)
        if (bi > pn && bi < nb) *reinterpret_cast<double2*>(M + tile_at(bi, pn) + pc) = acc[bi];
      __syncwarp();
    }
  }
  if (lane < 8 * nb) y[lane] += z;
  __syncwarp();
#pragma unroll 1
  for (int pn = nb - 1; pn >= 0; pn--) {
    double2 v = make_double2(0.0, 0.0);
    mma_f64(v.x, v.y, y[8 * pn + t], Di[64 * pn + p0]);
    mma_f64(v.x, v.y, y[8 * pn + 4 + t], Di[64 * pn + p1]);
    __syncwarp();
    if (g == 0) *pair_at(y, pn) = v;
    __syncwarp();
    if (pn > 0) {
      const double x0 = -y[8 * pn + t], x1 = -y[8 * pn + 4 + t];
      double2 acc[NB];
#pragma unroll
      for (int bj = 0; bj < NB - 1; bj++)
        if (bj < pn) {
          const double* P = M + tile_at(pn, bj);
          acc[bj] = *pair_at(y, bj);
          mma_f64(acc[bj].x, acc[bj].y, x0, P[q0]);
          mma_f64(acc[bj].x, acc[bj].y, x1, P[q1]);
        }
      __syncwarp();
#pragma unroll
      for (int bj = 0; bj < NB - 1; bj++)
        if (bj < pn && g == 0) *pair_at(y, bj) = acc[bj];
      __syncwarp();
    }
  }
  return true;
}

}  // namespace mg
