// A posteriori threshold pivoting (APTP) of large indefinite fronts: the
// dense kernel smf's deterministic mode runs on every indefinite front of at
// least 512 rows (solver/src/ldlt_aptp.cpp:1-751, as 2D tile tasks in
// parallel/tile_tasks.cpp:256-351; dispatch multifrontal_serial.cpp:796-821,
// parallel/thread_plan.hpp:43-47). The fully summed columns are taken in
// block columns of 256 (Control::top_tile_nb, control.hpp:638). Per block:
//   - the diagonal tile is factored speculatively by one CTA (an inner sweep
//     of 32-column blocks, complete pivoting on each, then on what failed
//     inside the tile), the rows below it are formed by a triangular solve
//     on many CTAs and checked afterwards against 1/u; the block keeps the
//     leading pivots whose multipliers pass and restores the rest from a
//     backup, in place;
//   - the rest of the front takes a rank-nelim update with those pivots
//     (the eligible columns right of them, and the earlier failed columns)
//     as tiled FP64 GEMMs over the whole GPU.
// At the end the failed columns move behind the pivots (one gather through
// a scratch front) and the non-eligible triangle takes one deferred update.
// Every entry takes the reference's operations in the reference's order and
// rounding: the portable BLAS loops' fused multiply-add chains (a zero
// multiplier skipped), and the fused forms GCC gives ldlt_aptp.cpp's
// a*b + c*d expressions (fma(a, b, c*d), except the first output of
// row_times_d, fma(c, d, a*b)). With the same input the front's L, D, pivot
// order, tags and Schur complement are the reference's, bit for bit.
#pragma once
#include "smfg_aptp_host.h"
#include "smfg_internal.cuh"

namespace smfg {
namespace aptp {

// Threads of the tile kernel: one CTA factors a 256-column tile, a chain of
// pivots; 1,024 threads would spill its rows' solves.
constexpr int kTileNT = 512;

__device__ __forceinline__ size_t ix(int j, int ld) { return (size_t)j * (size_t)ld; }

__device__ __forceinline__ bool l_ok(double l, double inv_u) { return fabs(l) <= inv_u; }

// Stable inverse of the 2x2 pivot (ldlt_aptp.cpp:83-93): a*c - b*b is fused
// as GCC contracts it.
__device__ __forceinline__ void inv2(double d00, double d10, double d11, double &i00, double &i10,
                                     double &i11) {
  const double s = max3_ref(fabs(d00), fabs(d10), fabs(d11));
  const double a = d00 / s, b = d10 / s, c = d11 / s;
  const double inv = 1.0 / __dmul_rn(fma(a, c, -__dmul_rn(b, b)), s);
  i00 = __dmul_rn(c, inv);
  i10 = __dmul_rn(-b, inv);
  i11 = __dmul_rn(a, inv);
}

// (L D) of one row for the pivots [0, k) of a tile (D inline: diagonal at
// T(t, t), 2x2 off-diagonal at T(t + 1, t)) (ldlt_aptp.cpp:270-287).
__device__ __forceinline__ double ld_of(const double *T, int ld, const int8_t *tags, int t, double l0,
                                        double l1) {
  const double d00 = T[ix(t, ld) + t];
  if (tags[t] == 2) return fma(l1, T[ix(t, ld) + t + 1], __dmul_rn(l0, d00));
  if (tags[t] == -1) {  // second of a 2x2: l0 is the first column's value, l1 this one's
    return fma(l0, T[ix(t - 1, ld) + t], __dmul_rn(l1, T[ix(t, ld) + t]));
  }
  return __dmul_rn(l0, d00);
}

// ---------------------------------------------------------------------------
// CTA-level pieces of the diagonal tile's factorization (one CTA of
// kTileNT threads per tile; the tile lives in global memory / L2).

// Complete pivoting runs on a copy of its view in shared memory (the lower
// triangle packed by columns) when it has at most this many columns: the
// inner blocks, and the tile's failed columns at the end of its sweep.
constexpr int kPackCols = 224;
constexpr int kPackDoubles = kPackCols * (kPackCols + 1) / 2;

struct TileShared {
  // the inner block's backup (column t at bk1 + t * kNb, tile rows) and its
  // packed view; at the end of the sweep one packed view over both
  union {
    struct {
      double bk1[kNb * kIb];
      double pk1[kIb * (kIb + 1) / 2];
    };
    double pk[kPackDoubles];
  };
  double dinv1[2 * kIb];
  int q1[kNb];
  int lpc1[kIb];
  int cp_lp[kNb];
  int itmp[kNb];
  double rv[32];
  int ri[32];
  int nq1, nmin, np;
  double lt[kIb][kIb];  // L of an inner block for its rows' solves: column p at lt[p]
};

// The threads that work on a view: the block, or (small views) one warp of it.
template <bool WARP>
struct Group {
  static __device__ __forceinline__ int tid() { return WARP ? (int)(threadIdx.x & 31) : (int)threadIdx.x; }
  static __device__ __forceinline__ int size() { return WARP ? 32 : (int)blockDim.x; }
  static __device__ __forceinline__ void sync() {
    if (WARP) __syncwarp();
    else __syncthreads();
  }
  // (a barrier too: what the threads read before it may be written after it;
  // a warp's vote alone orders no memory)
  static __device__ __forceinline__ bool any(bool b) {
    if (!WARP) return __syncthreads_or(b) != 0;
    const bool r = __any_sync(0xffffffffu, b) != 0;
    __syncwarp();
    return r;
  }
};

// A view of a symmetric block by columns of its lower triangle: entry (i, j)
// at col(j)[i]. In place (leading dimension ld), or packed.
struct FullView {
  double *A;
  int ld;
  __device__ __forceinline__ double *col(int j) const { return A + ix(j, ld); }
};
struct PackView {
  double *A;
  int n;
  __device__ __forceinline__ double *col(int j) const { return A + j * (2 * n - j - 1) / 2; }
};

// Symmetric transposition of view positions p < q (ldlt_aptp.cpp:67-80);
// tags, rows, lp and loc follow. Callers synchronize before.
template <bool WARP, typename View>
static __device__ void cta_swap(const View &V, int m, int p, int q, int8_t *tags, int *rows, int *lp, int *loc) {
  if (p == q) return;
  if (p > q) {
    const int t = p;
    p = q;
    q = t;
  }
  const int items = m - 1;  // p diag pair + (c < p) + (p < c < q) + (r > q)
  for (int t = Group<WARP>::tid(); t < items; t += Group<WARP>::size()) {
    double *e1, *e2;
    if (t == 0) {
      e1 = V.col(p) + p;
      e2 = V.col(q) + q;
    } else if (t <= p) {
      const int c = t - 1;
      e1 = V.col(c) + p;
      e2 = V.col(c) + q;
    } else if (t < q) {
      const int c = t;  // p < c < q
      e1 = V.col(p) + c;
      e2 = V.col(c) + q;
    } else {
      const int r = t + 1;  // r > q
      e1 = V.col(p) + r;
      e2 = V.col(q) + r;
    }
    const double x = *e1;
    *e1 = *e2;
    *e2 = x;
  }
  if (Group<WARP>::tid() == 0) {
    const int8_t tg = tags[p];
    tags[p] = tags[q];
    tags[q] = tg;
    int u = rows[p];
    rows[p] = rows[q];
    rows[q] = u;
    u = lp[p];
    lp[p] = lp[q];
    lp[q] = u;
    if (loc) {
      u = loc[p];
      loc[p] = loc[q];
      loc[q] = u;
    }
  }
  Group<WARP>::sync();
}

template <typename View>
__device__ __forceinline__ double sym_at(const View &V, int i, int j) {
  return (i >= j) ? V.col(j)[i] : V.col(i)[j];
}

// A thread's share of an argmax of |A|: its first maximum in (column, row)
// order, NaNs never chosen (ldlt_aptp.cpp:108-122).
struct ArgMax {
  double v = -1.0;
  unsigned at = 0xffffffffu;  // column << 16 | row
  __device__ __forceinline__ void add(double x, int i, int j) {
    const double a = fabs(x);
    if (a > v) {
      v = a;
      at = (unsigned)j << 16 | (unsigned)i;
    }
  }
};

// The larger value wins; of equal values the lower column, then the lower row.
__device__ __forceinline__ void warp_argmax(double &v, unsigned &at) {
  const double m = warp_max_bits(v >= 0.0 ? v : 0.0);
  at = __reduce_min_sync(0xffffffffu, v == m ? at : 0xffffffffu);
  v = at == 0xffffffffu ? -1.0 : m;
}

// The group's argmax; ends with every thread holding it (a block: two
// barriers).
template <bool WARP>
static __device__ void cta_argmax(ArgMax t, TileShared &sh, double &amax, int &bi, int &bj) {
  if (WARP) {
    warp_argmax(t.v, t.at);
    __syncwarp();
    amax = t.v;
    bi = (int)(t.at & 0xffffu);
    bj = (int)(t.at >> 16);
    return;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  warp_argmax(t.v, t.at);
  if (lane == 0) {
    sh.rv[wid] = t.v;
    sh.ri[wid] = (int)t.at;
  }
  __syncthreads();
  double v = lane < nw ? sh.rv[lane] : -1.0;
  unsigned at = lane < nw ? (unsigned)sh.ri[lane] : 0xffffffffu;
  warp_argmax(v, at);
  __syncthreads();
  amax = v;
  bi = (int)(at & 0xffffu);
  bj = (int)(at >> 16);
}

// Complete pivoting on an n x n view (ldlt_aptp.cpp:101-210); returns the
// pivots taken. lp: the view's permutation record.
template <bool WARP, typename View>
static __device__ int cta_complete_on(const View &V, int n, int8_t *tags, int *rows, int *lp, int *loc, double inv_u,
                                      double small, TileShared &sh) {
  using GR = Group<WARP>;
  for (int t = GR::tid(); t < n; t += GR::size()) {
    lp[t] = t;
    tags[t] = 0;
  }
  GR::sync();
  int k = 0;
  const int lane = threadIdx.x & 31, wid = WARP ? 0 : threadIdx.x >> 5, nw = GR::size() >> 5;
  // the largest entry of the view, then with each pivot's update that of what
  // is left: a warp per column, its lanes down the rows, four in flight
  ArgMax best;
  for (int j = wid; j < n; j += nw)
    for (int i = j + lane; i < n; i += 32) best.add(V.col(j)[i], i, j);
  while (k < n) {
    double amax;
    int bi, bj;
    cta_argmax<WARP>(best, sh, amax, bi, bj);
    if (!(amax >= small) || !isfinite(amax)) break;
    // every thread takes the decision
    int kind = 1, a = bj, b = -1;
    if (bi != bj) {
      const double amm = V.col(bj)[bj], att = V.col(bi)[bi], amt = V.col(bj)[bi];
      const double delta = fma(amm, att, -__dmul_rn(amt, amt));
      if (fabs(delta) >= __dmul_rn(__dmul_rn(0.5, amt), amt)) {
        kind = 2;
        b = bi;
      } else {
        a = (fabs(att) > fabs(amm)) ? bi : bj;
      }
    }
    // a posteriori bound inside the view
    bool bad = false;
    if (kind == 1) {
      const double lim = __dmul_rn(inv_u, fabs(V.col(a)[a]));
      for (int r = k + GR::tid(); r < n; r += GR::size())
        if (r != a && !(fabs(sym_at(V, r, a)) <= lim)) bad = true;
    } else {
      double i00, i10, i11;
      inv2(V.col(a)[a], V.col(a)[b], V.col(b)[b], i00, i10, i11);
      for (int r = k + GR::tid(); r < n; r += GR::size()) {
        if (r == a || r == b) continue;
        const double x0 = sym_at(V, r, a), x1 = sym_at(V, r, b);
        if (!l_ok(fma(i00, x0, __dmul_rn(i10, x1)), inv_u) || !l_ok(fma(i10, x0, __dmul_rn(i11, x1)), inv_u))
          bad = true;
      }
    }
    if (GR::any(bad)) break;
    if (kind == 1) {
      cta_swap<WARP>(V, n, k, a, tags, rows, lp, loc);
      const double *ck = V.col(k);
      const double inv_d = 1.0 / ck[k];
      // entries (i, j), k < j <= i < n: one fused step each (a warp per
      // column)
      best = ArgMax{};
      if (WARP) {  // (n <= 32: a row a lane, four columns in flight)
        const double y = lane < n ? ck[lane > k ? lane : k] : 0.0;
        for (int j0 = k + 1; j0 < n; j0 += 4) {
          double x[4], l[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int jj = min(j0 + u, n - 1);
            l[u] = __dmul_rn(ck[jj], inv_d);
            x[u] = (lane >= jj && lane < n) ? V.col(jj)[lane] : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (j0 + u < n && lane >= j0 + u && lane < n) {
              if (l[u] != 0.0) {
                x[u] = fma(-y, l[u], x[u]);
                V.col(j0 + u)[lane] = x[u];
              }
              best.add(x[u], lane, j0 + u);
            }
        }
      } else
      for (int jj = k + 1 + wid; jj < n; jj += nw) {
        const double lj = __dmul_rn(ck[jj], inv_d);
        double *cj = V.col(jj);
        for (int i0 = jj + lane; i0 < n; i0 += 4 * 32) {
          double x[4], y[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            x[u] = i0 + 32 * u < n ? cj[i0 + 32 * u] : 0.0;
            y[u] = i0 + 32 * u < n ? ck[i0 + 32 * u] : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (i0 + 32 * u < n) {
              if (lj != 0.0) {
                x[u] = fma(-y[u], lj, x[u]);
                cj[i0 + 32 * u] = x[u];
              }
              best.add(x[u], i0 + 32 * u, jj);
            }
        }
      }
      GR::sync();
      double *ckw = V.col(k);
      for (int i = k + 1 + GR::tid(); i < n; i += GR::size()) ckw[i] = __dmul_rn(ckw[i], inv_d);
      if (GR::tid() == 0) tags[k] = 1;
      GR::sync();
      k += 1;
    } else {
      int partner = b;
      if (a != k) {
        cta_swap<WARP>(V, n, k, a, tags, rows, lp, loc);
        if (partner == k) partner = a;
      }
      if (partner != k + 1) cta_swap<WARP>(V, n, k + 1, partner, tags, rows, lp, loc);
      double *c0 = V.col(k), *c1 = V.col(k + 1);
      double i00, i10, i11;
      inv2(c0[k], c0[k + 1], c1[k + 1], i00, i10, i11);
      best = ArgMax{};
      if (WARP) {
        const int lr = lane > k + 1 && lane < n ? lane : k + 1;
        const double y0 = c0[lr], y1 = c1[lr];
        for (int j0 = k + 2; j0 < n; j0 += 4) {
          double x[4], l0[4], l1[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int jj = min(j0 + u, n - 1);
            const double a0 = c0[jj], a1 = c1[jj];
            l0[u] = fma(i00, a0, __dmul_rn(i10, a1));
            l1[u] = fma(i10, a0, __dmul_rn(i11, a1));
            x[u] = (lane >= jj && lane < n) ? V.col(jj)[lane] : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (j0 + u < n && lane >= j0 + u && lane < n) {
              if (!(l0[u] == 0.0 && l1[u] == 0.0)) {
                x[u] = __dsub_rn(x[u], fma(y0, l0[u], __dmul_rn(y1, l1[u])));
                V.col(j0 + u)[lane] = x[u];
              }
              best.add(x[u], lane, j0 + u);
            }
        }
      } else
      for (int jj = k + 2 + wid; jj < n; jj += nw) {
        const double a0 = c0[jj], a1 = c1[jj];
        const double l0 = fma(i00, a0, __dmul_rn(i10, a1)), l1 = fma(i10, a0, __dmul_rn(i11, a1));
        const bool upd = !(l0 == 0.0 && l1 == 0.0);
        double *cj = V.col(jj);
        for (int i0 = jj + lane; i0 < n; i0 += 4 * 32) {
          double x[4], y0[4], y1[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            x[u] = i0 + 32 * u < n ? cj[i0 + 32 * u] : 0.0;
            y0[u] = i0 + 32 * u < n ? c0[i0 + 32 * u] : 0.0;
            y1[u] = i0 + 32 * u < n ? c1[i0 + 32 * u] : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (i0 + 32 * u < n) {
              if (upd) {
                x[u] = __dsub_rn(x[u], fma(y0[u], l0, __dmul_rn(y1[u], l1)));
                cj[i0 + 32 * u] = x[u];
              }
              best.add(x[u], i0 + 32 * u, jj);
            }
        }
      }
      GR::sync();
      for (int i = k + 2 + GR::tid(); i < n; i += GR::size()) {
        const double a0 = c0[i], a1 = c1[i];
        c0[i] = fma(i00, a0, __dmul_rn(i10, a1));
        c1[i] = fma(i10, a0, __dmul_rn(i11, a1));
      }
      if (GR::tid() == 0) {
        tags[k] = 2;
        tags[k + 1] = -1;
      }
      GR::sync();
      k += 2;
    }
  }
  GR::sync();
  return k;
}

// The same in place at A (leading dimension ld), through a packed copy at pk
// when there is one: a pivot's pass over the view is then bound by its
// barriers, not by L2's latency.
static __device__ int cta_complete(double *A, int ld, int n, int8_t *tags, int *rows, int *lp, int *loc, double inv_u,
                                   double small, TileShared &sh, double *pk) {
  const FullView G{A, ld};
  if (!pk) return cta_complete_on<false>(G, n, tags, rows, lp, loc, inv_u, small, sh);
  const PackView S{pk, n};
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  for (int j = threadIdx.x >> 5; j < n; j += nw)
    for (int i = j + lane; i < n; i += 32) S.col(j)[i] = G.col(j)[i];
  __syncthreads();
  int p;
  if (n <= 32) {
    // one warp: no block barriers in the chain
    if (threadIdx.x < 32) {
      p = cta_complete_on<true>(S, n, tags, rows, lp, loc, inv_u, small, sh);
      if (lane == 0) sh.np = p;
    }
    __syncthreads();
    p = sh.np;
  } else {
    p = cta_complete_on<false>(S, n, tags, rows, lp, loc, inv_u, small, sh);
  }
  for (int j = threadIdx.x >> 5; j < n; j += nw)
    for (int i = j + lane; i < n; i += 32) G.col(j)[i] = S.col(j)[i];
  __syncthreads();
  return p;
}

// Rows [r0, r0 + w) of columns [0, ncols): new row r0 + t takes old row
// r0 + perm[t] (ldlt_aptp.cpp:214-221); w <= 256.
static __device__ void cta_permute_rows(double *A, int ld, int ncols, int r0, int w, const int *perm) {
  const int lane = threadIdx.x & 31;
  int src[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) src[u] = lane + 32 * u < w ? perm[lane + 32 * u] : 0;
  for (int c = threadIdx.x >> 5; c < ncols; c += blockDim.x >> 5) {  // a warp per column
    double v[8], *col = A + ix(c, ld) + r0;
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = lane + 32 * u < w ? col[src[u]] : 0.0;
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (lane + 32 * u < w) col[lane + 32 * u] = v[u];
  }
  __syncthreads();
}

static __device__ bool cta_identity(const int *perm, int w) {
  bool diff = false;
  for (int t = threadIdx.x; t < w; t += blockDim.x) diff = diff || perm[t] != t;
  return !__syncthreads_or(diff);
}

// x := x L^-T for one row (x holds its first k entries, k <= KMAX), L the
// unit lower triangle, column p at lt[p] (2x2 off-diagonals zero): per
// entry one fused chain over the earlier columns in order, a zero L entry
// skipped; then the D^-1 scaling, returning the first pivot whose
// multipliers exceed 1/u, or k (ldlt_aptp.cpp:232-265, :292-304).
template <int KMAX>
__device__ __forceinline__ int row_solve_scale(double (&x)[KMAX], int k, const double (*lt)[KMAX], const int8_t *tags,
                                               const double *dinv, double inv_u) {
#pragma unroll
  for (int j = 1; j < KMAX; ++j) {
    if (j < k) {
      double xj = x[j];
#pragma unroll
      for (int p = 0; p < j; ++p) {
        const double l = lt[p][j];
        const double y = fma(-x[p], l, xj);
        xj = l != 0.0 ? y : xj;
      }
      x[j] = xj;
    }
  }
  int fail = k;
#pragma unroll
  for (int t = 0; t < KMAX; ++t) {
    if (t < k) {
      if (tags[t] == 2) {
        const double i00 = dinv[2 * t], i10 = dinv[2 * t + 1], i11 = dinv[2 * (t + 1)];
        const double a0 = x[t], a1 = x[t + 1 < KMAX ? t + 1 : t];
        const double l0 = fma(i00, a0, __dmul_rn(i10, a1)), l1 = fma(i10, a0, __dmul_rn(i11, a1));
        x[t] = l0;
        if (t + 1 < KMAX) x[t + 1] = l1;
        if (fail == k && (!l_ok(l0, inv_u) || !l_ok(l1, inv_u))) fail = t;
      } else if (tags[t] == 1) {
        const double l = __dmul_rn(x[t], dinv[2 * t]);
        x[t] = l;
        if (fail == k && !l_ok(l, inv_u)) fail = t;
      }
    }
  }
  return fail;
}

// One inner block column [c0, c0 + w1) of the tile sweep (block ib = 32):
// backup, complete pivoting on the diagonal block, its permutation applied,
// ApplyN on the tile rows below, ApplyT on the earlier failed columns,
// restore, UpdateNN / NT / TN (ldlt_aptp.cpp:390-588 at level 1). Returns
// the accepted pivots.
static __device__ int tile_inner_block(double *T, int ld, int w, int c0, int w1, int8_t *tags, int *rows, int *lp,
                                int *loc, double inv_u, double small, TileShared &sh) {
  // 1. backup: column c0 + t, tile rows [c0 + t, w)
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll 2
  for (int t = wid; t < w1; t += nw)
#pragma unroll 4
    for (int r = c0 + t + lane; r < w; r += 32) sh.bk1[t * kNb + r] = T[ix(c0 + t, ld) + r];
  __syncthreads();
  // 2. complete pivoting on the diagonal block
  const int ne_t = cta_complete(T + ix(c0, ld) + c0, ld, w1, tags + c0, rows + c0, sh.lpc1, loc ? loc + c0 : nullptr,
                                inv_u, small, sh, sh.pk1);
  // 3. its permutation on the rest of the tile
  if (!cta_identity(sh.lpc1, w1)) {
    cta_permute_rows(T, ld, c0, c0, w1, sh.lpc1);
    for (int t = wid; t < w1; t += nw)
      for (int r = c0 + w1 + lane; r < w; r += 32) T[ix(c0 + t, ld) + r] = sh.bk1[sh.lpc1[t] * kNb + r];
    if ((int)threadIdx.x < w1) sh.itmp[threadIdx.x] = lp[c0 + sh.lpc1[threadIdx.x]];
    __syncthreads();
    if ((int)threadIdx.x < w1) lp[c0 + threadIdx.x] = sh.itmp[threadIdx.x];
    __syncthreads();
  }
  const double *Tb = T + ix(c0, ld) + c0;  // the block's diagonal tile
  const int8_t *tb = tags + c0;
  if ((int)threadIdx.x < ne_t) {
    const int j = threadIdx.x;
    if (tb[j] == 2) {
      double i00, i10, i11;
      inv2(Tb[ix(j, ld) + j], Tb[ix(j, ld) + j + 1], Tb[ix(j + 1, ld) + j + 1], i00, i10, i11);
      sh.dinv1[2 * j] = i00;
      sh.dinv1[2 * j + 1] = i10;
      sh.dinv1[2 * (j + 1)] = i11;
      sh.dinv1[2 * (j + 1) + 1] = 0.0;
    } else if (tb[j] == 1) {
      sh.dinv1[2 * j] = 1.0 / Tb[ix(j, ld) + j];
      sh.dinv1[2 * j + 1] = 0.0;
    }
  }
  for (int e = threadIdx.x; e < kIb * kIb; e += blockDim.x) {
    const int p = e / kIb, j = e % kIb;
    sh.lt[p][j] = (p < ne_t && j > p && j < w1 && !(tb[p] == 2 && j == p + 1)) ? Tb[ix(p, ld) + j] : 0.0;
  }
  if (threadIdx.x == 0) sh.nmin = ne_t;
  __syncthreads();
  // 4. ApplyN on the tile rows below the block and ApplyT (check pass) on
  // the earlier failed columns: the first failing pivot over all rows
  const int nq = sh.nq1;
  if (ne_t > 0) {
    const int nbelow = w - c0 - w1;
    int fail = ne_t;
    for (int t = threadIdx.x; t < nbelow + nq; t += blockDim.x) {
      double x[kIb];
      const bool below = t < nbelow;
      const int r = below ? c0 + w1 + t : 0;
      const double *src = below ? T + ix(c0, ld) + r : T + ix(sh.q1[t - nbelow], ld) + c0;
      const size_t stride = below ? (size_t)ld : 1;
#pragma unroll
      for (int u = 0; u < kIb; ++u) x[u] = (u < ne_t) ? src[u * stride] : 0.0;
      const int fl = row_solve_scale<kIb>(x, ne_t, sh.lt, tb, sh.dinv1, inv_u);
      if (below) {
#pragma unroll
        for (int u = 0; u < kIb; ++u)
          if (u < ne_t) T[ix(c0 + u, ld) + r] = x[u];
      }
      fail = min(fail, fl);
    }
    atomicMin(&sh.nmin, fail);
  }
  __syncthreads();
  int nelim = sh.nmin;
  if (ne_t > 0 && nelim > 0 && tb[nelim - 1] == 2) --nelim;  // a 2x2 never splits
  // 5. restore the failed columns [nelim, w1) from the backup (permuted)
  if (nelim < w1) {
    for (int s2 = nelim; s2 < w1; ++s2) {
      double *col = T + ix(c0 + s2, ld);
      const int b2 = sh.lpc1[s2];
      for (int s1 = s2 + threadIdx.x; s1 < w1; s1 += blockDim.x) {
        const int a1 = sh.lpc1[s1];
        col[c0 + s1] = (a1 >= b2) ? sh.bk1[b2 * kNb + c0 + a1] : sh.bk1[a1 * kNb + c0 + b2];
      }
      for (int r = c0 + w1 + threadIdx.x; r < w; r += blockDim.x) col[r] = sh.bk1[b2 * kNb + r];
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int s2 = nelim; s2 < w1; ++s2) tags[c0 + s2] = 0;
  }
  __syncthreads();
  if (nelim > 0) {
    // ApplyT, final: the failed columns' L rows for the accepted pivots
    for (int t = threadIdx.x; t < nq; t += blockDim.x) {
      double x[kIb];
      double *src = T + ix(sh.q1[t], ld) + c0;
#pragma unroll
      for (int u = 0; u < kIb; ++u) x[u] = (u < nelim) ? src[u] : 0.0;
      row_solve_scale<kIb>(x, nelim, sh.lt, tb, sh.dinv1, inv_u);
#pragma unroll
      for (int u = 0; u < kIb; ++u)
        if (u < nelim) src[u] = x[u];
    }
    // UpdateNN: W = (L D)^T of the columns [e0, w) into their strict upper
    // triangle rows [c0, c0 + nelim), and with the rows' L in shared memory
    // (past the backup, which is done with; row r of pivot p at [p][r])
    const int e0 = c0 + nelim;
    double(*Lp)[kNb] = reinterpret_cast<double(*)[kNb]>(sh.pk);
    double(*Wp)[kNb] = reinterpret_cast<double(*)[kNb]>(sh.pk + kIb * kNb);
    static_assert(2 * kIb * kNb <= kPackDoubles, "L and W panels");
    __syncthreads();  // (the restore has read the backup)
    for (int t = wid; t < nelim; t += nw)
      for (int col = e0 + lane; col < w; col += 32) {
        const double l0 = T[ix(c0 + t, ld) + col];
        double v;
        if (tb[t] == 2) {
          const double l1 = T[ix(c0 + t + 1, ld) + col];
          v = fma(l1, Tb[ix(t, ld) + t + 1], __dmul_rn(l0, Tb[ix(t, ld) + t]));
        } else if (tb[t] == -1) {
          const double lm1 = T[ix(c0 + t - 1, ld) + col];
          v = fma(lm1, Tb[ix(t - 1, ld) + t], __dmul_rn(l0, Tb[ix(t, ld) + t]));
        } else {
          v = __dmul_rn(l0, Tb[ix(t, ld) + t]);
        }
        T[ix(col, ld) + c0 + t] = v;
        Wp[t][col] = v;
        Lp[t][col] = l0;
      }
    __syncthreads();
    // a warp four columns at a time, lanes over the rows
    for (int j0 = e0 + 4 * wid; j0 < w; j0 += 4 * nw) {
      for (int ri = j0 + lane; ri < w; ri += 32) {
        double c[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) c[u] = (j0 + u <= ri) ? T[ix(j0 + u, ld) + ri] : 0.0;
        for (int p = 0; p < nelim; ++p) {
          const double a = -Lp[p][ri];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const double bw = Wp[p][min(j0 + u, w - 1)];
            const double y = fma(a, bw, c[u]);
            c[u] = bw != 0.0 ? y : c[u];
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (j0 + u <= ri) T[ix(j0 + u, ld) + ri] = c[u];
      }
    }
    // UpdateNT / TN: the earlier failed columns, tile rows [e0, w) and their
    // block among themselves; each entry one chain from zero, then one
    // subtraction. (L D) of the failed columns' rows first, into bk1 (the
    // panels are done with). A warp takes four columns, lanes the rows.
    double(*ldq)[kIb] = reinterpret_cast<double(*)[kIb]>(sh.bk1);
    __syncthreads();
    for (int e = threadIdx.x; e < nq * nelim; e += blockDim.x) {
      const int jq = e / nelim, p = e % nelim;
      const double *lq = T + ix(sh.q1[jq], ld) + c0;
      ldq[jq][p] = (tb[p] == -1) ? ld_of(Tb, ld, tb, p, lq[p - 1], lq[p])
                                 : ld_of(Tb, ld, tb, p, lq[p], tb[p] == 2 ? lq[p + 1] : 0.0);
    }
    __syncthreads();
    for (int j0 = 4 * wid; j0 < nq; j0 += 4 * nw) {
      const int nj = min(4, nq - j0);
      // rows [e0, w) of the tile, then the failed columns' rows from j0 on
      const int nr = w - e0;
      for (int t = lane; t < nr + nq - j0; t += 32) {
        const bool in = t < nr;
        const int r = in ? e0 + t : sh.q1[j0 + t - nr];
        const double *row = in ? T + ix(c0, ld) + r : T + ix(r, ld) + c0;
        const size_t stride = in ? (size_t)ld : 1;
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        for (int p = 0; p < nelim; ++p) {
          const double l = row[p * stride];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const double bw = u < nj ? ldq[j0 + u][p] : 0.0;
            const double y = fma(l, bw, acc[u]);
            acc[u] = bw != 0.0 ? y : acc[u];
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (u < nj && (in || t - nr >= u)) {  // (of the failed block its lower part)
            double *c = T + ix(sh.q1[j0 + u], ld) + r;
            *c = __dsub_rn(*c, acc[u]);
          }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int s = nelim; s < w1; ++s) sh.q1[sh.nq1++] = c0 + s;
  }
  __syncthreads();
  return nelim;
}

// Moves the failed columns behind the eliminated ones, eliminated order
// kept (ldlt_aptp.cpp:603-614), on an m x m view.
static __device__ void cta_compact(double *A, int ld, int m, int ne, int8_t *tags, int *rows, int *lp, int *loc) {
  int dst = 0;
  for (int src = 0; src < ne; ++src) {
    if (tags[src] == 0) continue;
    if (src != dst) cta_swap<false>(FullView{A, ld}, m, dst, src, tags, rows, lp, loc);
    ++dst;
  }
  __syncthreads();
}

// The diagonal tile (w x w at T): the inner sweep, then complete pivoting
// on what failed inside it (ldlt_aptp.cpp:335-350). lp: the tile's
// permutation record. Returns the tile's pivots.
static __device__ int tile_factor(double *T, int ld, int w, int8_t *tags, int *rows, int *lp, int *loc, double inv_u,
                           double small, TileShared &sh) {
  if (w <= kIb) return cta_complete(T, ld, w, tags, rows, lp, loc, inv_u, small, sh, sh.pk1);
  for (int t = threadIdx.x; t < w; t += blockDim.x) {
    lp[t] = t;
    tags[t] = 0;
  }
  if (threadIdx.x == 0) sh.nq1 = 0;
  __syncthreads();
  int ne1 = 0;
  for (int c0 = 0; c0 < w; c0 += kIb) ne1 += tile_inner_block(T, ld, w, c0, min(kIb, w - c0), tags, rows, lp, loc,
                                                             inv_u, small, sh);
  if (ne1 < w) cta_compact(T, ld, w, w, tags, rows, lp, loc);
  if (ne1 < w) {
    const int n2 = w - ne1;
    const int ne2 = cta_complete(T + ix(ne1, ld) + ne1, ld, n2, tags + ne1, rows + ne1, sh.cp_lp,
                                 loc ? loc + ne1 : nullptr, inv_u, small, sh, n2 <= kPackCols ? sh.pk : nullptr);
    if (!cta_identity(sh.cp_lp, n2)) {
      cta_permute_rows(T, ld, ne1, ne1, n2, sh.cp_lp);
      if ((int)threadIdx.x < n2) sh.itmp[threadIdx.x] = lp[ne1 + sh.cp_lp[threadIdx.x]];
      __syncthreads();
      if ((int)threadIdx.x < n2) lp[ne1 + threadIdx.x] = sh.itmp[threadIdx.x];
      __syncthreads();
    }
    ne1 += ne2;
  }
  return ne1;
}

}  // namespace aptp
}  // namespace smfg
