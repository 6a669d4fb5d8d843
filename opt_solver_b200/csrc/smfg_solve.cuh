// The solves' level kernels: forward and backward sweep of one tree level's
// fronts, one launch each, up to kSolveRhs right-hand sides at a time.
//
// What bounds them is latency (a front's pivots are one chain, levels follow
// one another), so a front's L is brought into shared memory (up to 64 rows)
// or requested into L2 (more) before the kernel waits for the one before it
// (programmatic dependent launch), every right-hand side's chain runs beside
// the others, and the reciprocals of an SPD diagonal are formed off the chain.
// One grid: a block per front -- of up to 64 rows with L in shared memory and
// a warp per right-hand side, of more in 32-column strips -- then blocks of
// eight tiny fronts
// (up to 32 rows), a warp each, where the sizes are known beforehand (SPD
// fronts, leaves): delays may grow the others. Before them a block per large
// front and right-hand side: it only gathers (forward) or applies D^-1
// (backward), the block kernels go on.
// Sums run in a fixed order (deterministic); solve_forward.cpp:116-293 and
// solve_backward.cpp:135-350 compute the same quantities.
// Measured on one B200 against the two kernels a level and direction before
// (a warp per small front, the right-hand sides one after another), solve
// only: a 200-stage trajectory with 8 right-hand sides 1.76 -> 0.60 ms, 256
// of them 5.0 -> 2.4, a 40^3 operator with 16 12.5 -> 7.8, a 52 x 49 x 50 one
// with 1 3.08 -> 2.58.
#pragma once
#include <type_traits>

#include "smfg_kernels.cuh"

namespace smfg {

constexpr int kSolveRhs = 8;     // right-hand sides per sweep
constexpr int kLvlNT = 256;      // threads of the level kernels
constexpr int kLvlWarps = kLvlNT / 32;
constexpr int kTinyRows = 32;    // a warp per front
constexpr int kStageRows = 64;   // a block per front, L in shared memory
// doubles a warp stages: a tiny front's L (32 x 33) and its vectors
constexpr int kTinyDoubles = kTinyRows * (kTinyRows + 1) + 4 * kTinyRows;
// Dynamic shared memory of a level kernel: eight tiny fronts, or one staged
// front with its vectors, or a larger front's vectors (bigger ones in global
// memory).
constexpr int kLvlDoubles = kLvlWarps * kTinyDoubles;
constexpr int kLvlSmem = kLvlDoubles * 8;
static_assert(kLvlDoubles >= kStageRows * (kStageRows + 1) + 3 * kSolveRhs * kStageRows, "staged front");

// The blocks of a level's launch: nl large fronts (list lg), a block for each
// right-hand side; n fronts P.lvl_sn[i0 + block], a block each (the large
// ones among them leave); nc tiny ones from ic, a warp each. Every front is
// taken, so every launch has a block that waits for the kernel before it.
struct LevelGrid {
  const int *lg;
  int nl, i0, n, ic, nc;
};
// The larger fronts' strip: its triangle and solved values, then vectors.
constexpr int kStripDoubles = 32 * 33 + 32 * kSolveRhs;

// w / d from d's rounded reciprocal r: the product corrected by its remainder
// (Markstein), so that a pivot costs a multiply and two fused multiply-adds in
// the chain in place of a division, and rounds as one. The product alone left
// backward errors 5% larger on small 5- and 7-point operators; the correction
// costs 0 to 0.6% of a solve (52 x 49 x 50: 2.35 -> 2.37 ms).
__device__ __forceinline__ double quotient(double w, double d, double r) {
  const double q = w * r, e = fma(-q, d, w), y = fma(e, r, q);
  return e == e ? y : q;
}

// Four right-hand sides' (or one's) forward chain over a front in shared
// memory (Ls: column j at j * ld, rows 0..f): rows lane (and lane + 32 when
// two) of w.
template <int R, bool TWO>
__device__ __forceinline__ void small_fwd_chain(const double *Ls, int ld, int f, int p, const double *rd, bool spd,
                                                double (&w0)[R], double (&w1)[R]) {
  const int lane = threadIdx.x & 31;
  for (int j0 = 0; j0 < p; j0 += 8) {
    double l0[8], l1[8], r[8], d[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = j0 + u;
      d[u] = (spd && j < p) ? Ls[j * ld + j] : 1.0;
      l0[u] = (j < p && lane > j && lane < f) ? Ls[j * ld + lane] : 0.0;
      l1[u] = (TWO && j < p && lane + 32 > j && lane + 32 < f) ? Ls[j * ld + lane + 32] : 0.0;
      r[u] = (spd && j < p) ? rd[j] : 1.0;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = j0 + u;
      if (j >= p) break;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        double wj = __shfl_sync(0xffffffffu, (TWO && j >= 32) ? w1[q] : w0[q], j & 31);
        if (spd) {
          wj = quotient(wj, d[u], r[u]);
          w0[q] = lane == j ? wj : w0[q];
          if (TWO) w1[q] = lane + 32 == j ? wj : w1[q];
        }
        const double a = fma(-l0[u], wj, w0[q]);
        w0[q] = l0[u] != 0.0 ? a : w0[q];
        if (TWO) {
          const double b = fma(-l1[u], wj, w1[q]);
          w1[q] = l1[u] != 0.0 ? b : w1[q];
        }
      }
    }
  }
}

// The backward chain: columns lane (and lane + 32) of v, L^T from the last
// pivot on.
template <int R, bool TWO>
__device__ __forceinline__ void small_bwd_chain(const double *Ls, int ld, int p, const double *rd, bool spd,
                                                double (&v0)[R], double (&v1)[R]) {
  const int lane = threadIdx.x & 31;
  for (int j1 = p; j1 > 0; j1 -= 8) {
    double l0[8], l1[8], r[8], d[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = j1 - 1 - u;  // row j of L11
      d[u] = (spd && j >= 0) ? Ls[j * ld + j] : 1.0;
      l0[u] = (j >= 0 && lane < j) ? Ls[lane * ld + j] : 0.0;
      l1[u] = (TWO && j >= 0 && lane + 32 < j) ? Ls[(lane + 32) * ld + j] : 0.0;
      r[u] = (spd && j >= 0) ? rd[j] : 1.0;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = j1 - 1 - u;
      if (j < 0) break;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        double xj = __shfl_sync(0xffffffffu, (TWO && j >= 32) ? v1[q] : v0[q], j & 31);
        if (spd) {
          xj = quotient(xj, d[u], r[u]);
          v0[q] = lane == j ? xj : v0[q];
          if (TWO) v1[q] = lane + 32 == j ? xj : v1[q];
        }
        const double a = fma(-l0[u], xj, v0[q]);
        v0[q] = l0[u] != 0.0 ? a : v0[q];
        if (TWO) {
          const double b = fma(-l1[u], xj, v1[q]);
          v1[q] = l1[u] != 0.0 ? b : v1[q];
        }
      }
    }
  }
}

// L of a front of f <= 64 rows (its p stored columns, each from the row
// before its diagonal on: the slot above holds a 2x2 pivot's off-diagonal)
// into shared memory by threads t of nt (whole warps), a warp per column.
__device__ __forceinline__ void stage_front(const double *L, int f, int p, double *Ls, int ld, int t, int nt) {
  const int lane = t & 31, nw = nt >> 5;
  constexpr int G = 4;
  for (int c0 = t >> 5; c0 < p; c0 += G * nw) {
    for (int i = lane; i < f; i += 32) {
      double v[G];
#pragma unroll
      for (int u = 0; u < G; ++u) {
        const int c = c0 + u * nw;
        v[u] = (c < p && i >= c - 1) ? __ldg(L + (size_t)c * f + i) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < G; ++u) {
        const int c = c0 + u * nw;
        if (c < p) Ls[c * ld + i] = v[u];
      }
    }
  }
}

// v_c for the pivot column c of a front (Lc: column c; the next column f
// further, ldn apart): the D^-1-applied value of column c and, for a 2x2
// pivot's first column, of c + 1; false when column c is a pair's second.
__device__ __forceinline__ bool pivot_value(const double *Lc, int ldn, int c, int p, bool use_d, double y0, double y1,
                                            double &z0, double &z1, bool &pair) {
  pair = false;
  z0 = y0;
  z1 = 0.0;
  if (!use_d) return true;
  if (c > 0 && Lc[c - 1] != 0.0) return false;
  const double d00 = Lc[c];
  const double d10 = c + 1 < p ? Lc[ldn + c] : 0.0;
  if (d10 != 0.0) {
    pair = true;
    dinv2_apply(d00, d10, Lc[ldn + c + 1], y0, y1, z0, z1);
  } else {
    z0 = (d00 == 0.0 || !isfinite(d00)) ? 0.0 : y0 / d00;
  }
  return true;
}

// A child's update vectors added into the parent's vectors in child order.
// sw: the parent's vectors, right-hand side r at sw + r * stride; threads t
// of nt; sync() between children.
template <int RB, typename Sync>
__device__ __forceinline__ void add_children(const DevPlan &P, const DevFactor &X, int s, const double *wk,
                                             int64_t rows_total, int r0, int r1, double *sw, int64_t stride, int t,
                                             int nt, Sync sync) {
  for (int ti = P.child_ptr[s]; ti < P.child_ptr[s + 1]; ++ti) {
    const int c = P.child_idx[ti];
    const int pc = X.sn_pstore[c], n = X.sn_f[c] - pc;
    const int64_t co = X.sn_roff[c] + pc;
    const int *cmap = X.cbmap + co;
    for (int i0 = t; i0 < n; i0 += 4 * nt) {
      int m[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) m[u] = i0 + u * nt < n ? cmap[i0 + u * nt] : 0;
      for (int r = r0; r < r1; r += RB) {  // RB right-hand sides' loads in flight
        double v[RB][4];
#pragma unroll
        for (int q = 0; q < RB; ++q)
#pragma unroll
          for (int u = 0; u < 4; ++u)
            v[q][u] = (r + q < r1 && i0 + u * nt < n) ? wk[(int64_t)(r + q) * rows_total + co + i0 + u * nt] : 0.0;
#pragma unroll
        for (int q = 0; q < RB; ++q)
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (r + q < r1 && i0 + u * nt < n) sw[(r + q) * stride + m[u]] += v[q][u];
      }
    }
    sync();
  }
}

// Requests the p stored columns of a front into L2 (a column from its
// diagonal on), 128-byte lines.
__device__ __forceinline__ void prefetch_front(const double *L, int f, int p) {
  for (int c = threadIdx.x >> 5; c < p; c += blockDim.x >> 5)
    for (int i = c + 16 * (int)(threadIdx.x & 31); i < f; i += 16 * 32)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(L + (size_t)c * f + i));
}

__global__ void __launch_bounds__(kLvlNT, 2) k_fwd_level(DevPlan P, DevFactor X, LevelGrid g, int posdef, double *x,
                                                      double *wk, int64_t rows_total, int nrhs) {
  extern __shared__ __align__(16) double lvl_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int blk = (int)blockIdx.x - g.nl * nrhs;
  if (blk < 0) {
    // --- a large front, one right-hand side: gather, children
    const int s = g.lg[blockIdx.x / nrhs], r = (int)blockIdx.x % nrhs;
    const int f = X.sn_f[s], p = X.sn_pstore[s];
    const int64_t roff = X.sn_roff[s];
    const int *rows = X.rows + roff;
    double *w = wk + (int64_t)r * rows_total + roff;
    const double *xr = x + (int64_t)r * P.n;
    pdl_wait();
    pdl_trigger();
    for (int i0 = tid; i0 < f; i0 += 8 * kLvlNT) {
      int ri[8];
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) ri[u] = i0 + u * kLvlNT < p ? rows[i0 + u * kLvlNT] : 0;
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = i0 + u * kLvlNT < p ? xr[ri[u]] : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (i0 + u * kLvlNT < f) w[i0 + u * kLvlNT] = v[u];
    }
    __syncthreads();
    add_children<1>(P, X, s, wk + (int64_t)r * rows_total, rows_total, 0, 1, w, 0, tid, kLvlNT, [] { __syncthreads(); });
    return;
  }
  if (blk >= g.n) {
    // --- tiny fronts, a warp each
    const int item = (blk - g.n) * kLvlWarps + warp;
    if (item >= g.nc) return;
    const int s = P.lvl_sn[g.ic + item];
    const int f = X.sn_f[s];
    const int p = X.sn_pstore[s], ld = f | 1;
    const int64_t roff = X.sn_roff[s];
    const int *rows = X.rows + roff;
    double *Ls = lvl_smem + warp * kTinyDoubles, *sw = Ls + kTinyRows * (kTinyRows + 1);
    stage_front(X.arena + X.sn_off[s], f, p, Ls, ld, lane, 32);
    const int my = lane < p ? rows[lane] : 0;
    __syncwarp();
    const double dv = (posdef && lane < p) ? Ls[lane * ld + lane] : 1.0, rdv = 1.0 / dv;
    pdl_wait();
    pdl_trigger();
    auto one = [&](int r0, auto tag) {
      constexpr int R = decltype(tag)::value;
      const int rn = min(R, nrhs - r0);
      for (int q = 0; q < rn; ++q)
        if (lane < f) sw[q * kTinyRows + lane] = lane < p ? x[(int64_t)(r0 + q) * P.n + my] : 0.0;
      __syncwarp();
      add_children<R>(P, X, s, wk + (int64_t)r0 * rows_total, rows_total, 0, rn, sw, kTinyRows, lane, 32,
                   [] { __syncwarp(); });
      double w0[R];
#pragma unroll
      for (int q = 0; q < R; ++q) {
        w0[q] = (q < rn && lane < f) ? sw[q * kTinyRows + lane] : 0.0;
      }
      __syncwarp();
      for (int j0 = 0; j0 < p; j0 += 8) {
        double l[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int j = j0 + u;
          l[u] = (j < p && lane > j && lane < f) ? Ls[j * ld + lane] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int j = j0 + u;
          if (j >= p) break;
#pragma unroll
          for (int q = 0; q < R; ++q) {
            if (posdef) {
              const double sc = quotient(w0[q], dv, rdv);
              w0[q] = lane == j ? sc : w0[q];
            }
            const double wj = __shfl_sync(0xffffffffu, w0[q], j);
            const double a = fma(-l[u], wj, w0[q]);
            w0[q] = l[u] != 0.0 ? a : w0[q];
          }
        }
      }
#pragma unroll
      for (int q = 0; q < R; ++q)
        if (q < rn) {
          if (lane < p) x[(int64_t)(r0 + q) * P.n + my] = w0[q];
          else if (lane < f) wk[(int64_t)(r0 + q) * rows_total + roff + lane] = w0[q];
        }
    };
    if (nrhs == 1) one(0, std::integral_constant<int, 1>{});
    else
      for (int r0 = 0; r0 < nrhs; r0 += 4) one(r0, std::integral_constant<int, 4>{});
    return;
  }
  const int s = P.lvl_sn[g.i0 + blk];
  const int f = X.sn_f[s], p = X.sn_pstore[s];
  if (P.sn_large[s]) return;
  const int64_t roff = X.sn_roff[s];
  const int *rows = X.rows + roff;
  if (f <= kStageRows) {
    // --- up to 64 rows: L in shared memory, a warp per right-hand side
    const int ld = f | 1;
    double *Ls = lvl_smem, *rd = Ls + kStageRows * (kStageRows + 1), *sw = rd + kStageRows + warp * kStageRows;
    stage_front(X.arena + X.sn_off[s], f, p, Ls, ld, tid, kLvlNT);
    const int r0 = lane < p ? rows[lane] : 0, r1 = lane + 32 < p ? rows[lane + 32] : 0;
    __syncthreads();
    if (posdef) {
      if (tid < p) rd[tid] = 1.0 / Ls[tid * ld + tid];
      __syncthreads();
    }
    pdl_wait();
    pdl_trigger();
    if (warp >= nrhs) return;
    double *xr = x + (int64_t)warp * P.n;
    double *w = wk + (int64_t)warp * rows_total;
    sw[lane] = lane < p ? xr[r0] : 0.0;
    sw[lane + 32] = lane + 32 < p ? xr[r1] : 0.0;
    __syncwarp();
    add_children<1>(P, X, s, w, rows_total, 0, 1, sw, 0, lane, 32, [] { __syncwarp(); });
    double w0[1] = {sw[lane]}, w1[1] = {sw[lane + 32]};
    small_fwd_chain<1, true>(Ls, ld, f, p, rd, posdef != 0, w0, w1);
    if (lane < p) xr[r0] = w0[0];
    else if (lane < f) w[roff + lane] = w0[0];
    if (lane + 32 < p) xr[r1] = w1[0];
    else if (lane + 32 < f) w[roff + lane + 32] = w1[0];
    return;
  }
  // --- more than 64 rows
  const double *L = X.arena + X.sn_off[s];
  const size_t sf = (size_t)f;
  prefetch_front(L, f, p);
  pdl_wait();
  pdl_trigger();
  double(*wt)[kSolveRhs] = reinterpret_cast<double(*)[kSolveRhs]>(lvl_smem);  // the strip's solved values, a row a column
  double(*Ls)[33] = reinterpret_cast<double(*)[33]>(lvl_smem + 32 * kSolveRhs);
  // the vectors in shared memory when they fit
  const bool in_smem = (int64_t)f * nrhs <= kLvlDoubles - kStripDoubles;
  double *sw = in_smem ? lvl_smem + kStripDoubles : wk + roff;
  const int64_t stride = in_smem ? f : rows_total;
  auto gather = [&](auto tag) {
    constexpr int R = decltype(tag)::value;  // right-hand sides' loads in flight
    for (int i0 = tid; i0 < f; i0 += 2 * kLvlNT) {
      const int i1 = i0 + kLvlNT, ra = i0 < p ? rows[i0] : 0, rb = i1 < p ? rows[i1] : 0;
      for (int r0 = 0; r0 < nrhs; r0 += R) {
        double va[R], vb[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
          va[q] = (i0 < p && r0 + q < nrhs) ? x[(int64_t)(r0 + q) * P.n + ra] : 0.0;
          vb[q] = (i1 < p && r0 + q < nrhs) ? x[(int64_t)(r0 + q) * P.n + rb] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < R; ++q)
          if (r0 + q < nrhs) {
            sw[(r0 + q) * stride + i0] = va[q];
            if (i1 < f) sw[(r0 + q) * stride + i1] = vb[q];
          }
      }
    }
    __syncthreads();
    add_children<R>(P, X, s, wk, rows_total, 0, nrhs, sw, stride, tid, kLvlNT, [] { __syncthreads(); });
  };
  if (nrhs == 1) gather(std::integral_constant<int, 1>{});
  else gather(std::integral_constant<int, 4>{});
  for (int jb = 0; jb < p; jb += 32) {
    const int nb = min(32, p - jb);
    // the strip's triangle and this thread's first row below it loaded
    // before the barriers and the triangle solves (in flight meanwhile)
    double tv[1024 / kLvlNT];
#pragma unroll
    for (int u = 0; u < 1024 / kLvlNT; ++u) {
      const int t = tid + kLvlNT * u, r = t & 31, c = t >> 5;
      tv[u] = (r < nb && c < nb && c <= r) ? __ldg(L + (size_t)(jb + c) * sf + jb + r) : 0.0;
    }
    const int i1 = jb + nb + tid;
    double l[32];
#pragma unroll
    for (int u = 0; u < 32; ++u) l[u] = (i1 < f && u < nb) ? __ldg(L + (size_t)(jb + u) * sf + i1) : 0.0;
    __syncthreads();  // the previous strip's readers of Ls, wt and the vectors are done
#pragma unroll
    for (int u = 0; u < 1024 / kLvlNT; ++u) {
      const int t = tid + kLvlNT * u;
      Ls[t & 31][t >> 5] = tv[u];
    }
    __syncthreads();
    for (int r = warp; r < nrhs; r += kLvlWarps) {
      tri_fwd_warp(sw + r * stride, jb, nb, posdef, Ls);
      wt[lane][r] = lane < nb ? sw[r * stride + jb + lane] : 0.0;
    }
    __syncthreads();
    for (int i = i1; i < f; i += kLvlNT) {
      if (i != i1) {
        const double *li = L + (size_t)jb * sf + i;
#pragma unroll
        for (int u = 0; u < 32; ++u) l[u] = (u < nb) ? __ldg(li + (size_t)u * sf) : 0.0;
      }
      if (nrhs == 1) {
        double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int u = 0; u < 32; ++u) a[u & 3] = fma(l[u], wt[u][0], a[u & 3]);
        sw[i] -= sum4(a);
      } else {
        for (int r = 0; r < nrhs; r += 2) {  // two right-hand sides a load
          double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0;
#pragma unroll
          for (int u = 0; u < 32; u += 2) {
            const double2 y0 = *reinterpret_cast<const double2 *>(&wt[u][r]);
            const double2 y1 = *reinterpret_cast<const double2 *>(&wt[u + 1][r]);
            a0 = fma(l[u], y0.x, a0);
            b0 = fma(l[u], y0.y, b0);
            a1 = fma(l[u + 1], y1.x, a1);
            b1 = fma(l[u + 1], y1.y, b1);
          }
          sw[r * stride + i] -= a0 + a1;
          if (r + 1 < nrhs) sw[(r + 1) * stride + i] -= b0 + b1;
        }
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < f; i += kLvlNT) {
    const int ri = i < p ? rows[i] : 0;
    for (int r = 0; r < nrhs; ++r) {
      const double v = sw[r * stride + i];
      if (i < p) x[(int64_t)r * P.n + ri] = v;
      else if (in_smem) wk[(int64_t)r * rows_total + roff + i] = v;
    }
  }
}

__global__ void __launch_bounds__(kLvlNT, 2) k_bwd_level(DevPlan P, DevFactor X, LevelGrid g, int posdef, double *x,
                                                      double *wk, int64_t rows_total, int nrhs, int apply_d,
                                                      int apply_lt) {
  extern __shared__ __align__(16) double lvl_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int blk = (int)blockIdx.x - g.nl * nrhs;
  const bool use_d = apply_d && !posdef;
  if (blk < 0) {
    // --- a large front, one right-hand side: D^-1 of its pivot blocks, minus
    // L21^T x_ext (in v[0:p))
    const int s = g.lg[blockIdx.x / nrhs], r = (int)blockIdx.x % nrhs;
    const int f = X.sn_f[s], p = X.sn_pstore[s];
    const int *rows = X.rows + X.sn_roff[s];
    const double *L = X.arena + X.sn_off[s];
    pdl_wait();
    pdl_trigger();
    double *xr = x + (int64_t)r * P.n, *v = wk + (int64_t)r * rows_total + X.sn_roff[s];
#pragma unroll 4
    for (int c = tid; c < p; c += kLvlNT) {
      const double *Lc = L + (size_t)c * f;
      const double y0 = xr[rows[c]], y1 = (use_d && c + 1 < p) ? xr[rows[c + 1]] : 0.0;
      double z0, z1;
      bool pair;
      if (!pivot_value(Lc, f, c, p, use_d, y0, y1, z0, z1, pair)) continue;
      if (apply_lt) {
        z0 -= v[c];
        if (pair) z1 -= v[c + 1];
      }
      v[c] = z0;
      if (pair) v[c + 1] = z1;
    }
    if (apply_lt) return;
    __syncthreads();
    for (int c = tid; c < p; c += kLvlNT) xr[rows[c]] = v[c];
    return;
  }
  if (blk >= g.n) {
    // --- tiny fronts, a warp each
    const int item = (blk - g.n) * kLvlWarps + warp;
    if (item >= g.nc) return;
    const int s = P.lvl_sn[g.ic + item];
    const int f = X.sn_f[s];
    const int p = X.sn_pstore[s], ld = f | 1;
    const int *rows = X.rows + X.sn_roff[s];
    double *Ls = lvl_smem + warp * kTinyDoubles, *sx = Ls + kTinyRows * (kTinyRows + 1);
    stage_front(X.arena + X.sn_off[s], f, p, Ls, ld, lane, 32);
    const int my = lane < f ? rows[lane] : 0;
    __syncwarp();
    const double *Lc = Ls + lane * ld;
    const double dv = (posdef && lane < p) ? Lc[lane] : 1.0, rdv = 1.0 / dv;
    pdl_wait();
    pdl_trigger();
    auto one = [&](int r0, auto tag) {
      constexpr int R = decltype(tag)::value;
      const int rn = min(R, nrhs - r0);
      double v[R];
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const double xv = (q < rn && lane < f) ? x[(int64_t)(r0 + q) * P.n + my] : 0.0;
        sx[q * kTinyRows + lane] = xv;
        v[q] = xv;
      }
      __syncwarp();
      if (use_d) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
          const double y1 = __shfl_down_sync(0xffffffffu, v[q], 1);
          double z0 = v[q], z1 = 0.0;
          bool pair = false;
          if (lane < p) pivot_value(Lc, ld, lane, p, true, v[q], y1, z0, z1, pair);
          const double up = __shfl_up_sync(0xffffffffu, z1, 1);
          const bool second = __shfl_up_sync(0xffffffffu, (int)pair, 1) && lane > 0;
          if (lane < p) v[q] = second ? up : z0;
        }
      }
      if (apply_lt) {
        // the rows past the pivots, then the pivots from the last
#pragma unroll
        for (int q = 0; q < R; ++q) {
          double a0 = 0.0, a1 = 0.0;
          if (lane < p) {
            int i = p;
            for (; i + 1 < f; i += 2) {
              a0 = fma(Lc[i], sx[q * kTinyRows + i], a0);
              a1 = fma(Lc[i + 1], sx[q * kTinyRows + i + 1], a1);
            }
            if (i < f) a0 = fma(Lc[i], sx[q * kTinyRows + i], a0);
          }
          v[q] -= a0 + a1;
        }
        for (int j = p - 1; j >= 0; --j) {
          const double l = lane < j ? Lc[j] : 0.0;
#pragma unroll
          for (int q = 0; q < R; ++q) {
            const double sc = quotient(v[q], dv, rdv);
            v[q] = lane == j ? sc : v[q];
            const double xj = __shfl_sync(0xffffffffu, v[q], j);
            const double a = fma(-l, xj, v[q]);
            v[q] = l != 0.0 ? a : v[q];
          }
        }
      }
#pragma unroll
      for (int q = 0; q < R; ++q)
        if (q < rn && lane < p) x[(int64_t)(r0 + q) * P.n + my] = v[q];
      __syncwarp();
    };
    if (nrhs == 1) one(0, std::integral_constant<int, 1>{});
    else
      for (int r0 = 0; r0 < nrhs; r0 += 4) one(r0, std::integral_constant<int, 4>{});
    return;
  }
  const int s = P.lvl_sn[g.i0 + blk];
  const int f = X.sn_f[s], p = X.sn_pstore[s];
  if (P.sn_large[s]) return;
  const int64_t roff = X.sn_roff[s];
  const int *rows = X.rows + roff;
  if (f <= kStageRows) {
    // --- up to 64 rows
    const int ld = f | 1;
    double *Ls = lvl_smem, *rd = Ls + kStageRows * (kStageRows + 1), *sx = rd + kStageRows + warp * kStageRows;
    stage_front(X.arena + X.sn_off[s], f, p, Ls, ld, tid, kLvlNT);
    const int r0 = lane < f ? rows[lane] : 0, r1 = lane + 32 < f ? rows[lane + 32] : 0;
    __syncthreads();
    if (posdef) {
      if (tid < p) rd[tid] = 1.0 / Ls[tid * ld + tid];
      __syncthreads();
    }
    pdl_wait();
    pdl_trigger();
    if (warp >= nrhs) return;
    double *xr = x + (int64_t)warp * P.n;
    double v0[1] = {lane < f ? xr[r0] : 0.0}, v1[1] = {lane + 32 < f ? xr[r1] : 0.0};
    sx[lane] = v0[0];
    sx[lane + 32] = v1[0];
    __syncwarp();
    if (use_d) {
      // a pair may straddle the lanes' two halves: by shared memory
      double z0a = v0[0], z1a = 0.0, z0b = v1[0], z1b = 0.0;
      bool pa = false, pb = false, fa = false, fb = false;
      if (lane < p)
        fa = pivot_value(Ls + lane * ld, ld, lane, p, true, v0[0], sx[lane + 1], z0a, z1a, pa);
      if (lane + 32 < p)
        fb = pivot_value(Ls + (lane + 32) * ld, ld, lane + 32, p, true, v1[0], lane < 31 ? sx[lane + 33] : 0.0,
                         z0b, z1b, pb);
      __syncwarp();
      if (fa) sx[lane] = z0a;
      if (pa) sx[lane + 1] = z1a;
      if (fb) sx[lane + 32] = z0b;
      if (pb) sx[lane + 33] = z1b;
      __syncwarp();
      if (lane < p) v0[0] = sx[lane];
      if (lane + 32 < p) v1[0] = sx[lane + 32];
    }
    if (apply_lt) {
      const double *La = Ls + lane * ld, *Lb = La + 32 * ld;
      double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0;
      const bool ha = lane < p, hb = lane + 32 < p;
      int i = p;
      for (; i + 1 < f; i += 2) {
        const double y0 = sx[i], y1 = sx[i + 1];
        if (ha) {
          a0 = fma(La[i], y0, a0);
          a1 = fma(La[i + 1], y1, a1);
        }
        if (hb) {
          b0 = fma(Lb[i], y0, b0);
          b1 = fma(Lb[i + 1], y1, b1);
        }
      }
      if (i < f) {
        if (ha) a0 = fma(La[i], sx[i], a0);
        if (hb) b0 = fma(Lb[i], sx[i], b0);
      }
      v0[0] -= a0 + a1;
      v1[0] -= b0 + b1;
      small_bwd_chain<1, true>(Ls, ld, p, rd, posdef != 0, v0, v1);
    }
    if (lane < p) xr[r0] = v0[0];
    if (lane + 32 < p) xr[r1] = v1[0];
    return;
  }
  // --- more than 64 rows
  const double *L = X.arena + X.sn_off[s];
  const size_t sf = (size_t)f;
  if (apply_lt) prefetch_front(L, f, p);
  pdl_wait();
  pdl_trigger();
  double(*Ls)[33] = reinterpret_cast<double(*)[33]>(lvl_smem);
  const bool in_smem = (int64_t)f * nrhs <= kLvlDoubles - kStripDoubles;
  double *sv = in_smem ? lvl_smem + kStripDoubles : wk + roff;  // the pivots' values, then the rows past them
  const int64_t stride = in_smem ? f : rows_total;
  // the rows' values (four right-hand sides' loads in flight), then D^-1 of
  // each pivot block
  for (int i = tid; i < (apply_lt ? f : p); i += kLvlNT) {
    const int ri = rows[i];
    for (int r0 = 0; r0 < nrhs; r0 += 4) {
      double v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = r0 + q < nrhs ? x[(int64_t)(r0 + q) * P.n + ri] : 0.0;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (r0 + q < nrhs) sv[(r0 + q) * stride + i] = v[q];
    }
  }
  if (use_d) {
    __syncthreads();
    for (int c = tid; c < p; c += kLvlNT) {
      const double *Lc = L + (size_t)c * sf;
      for (int r = 0; r < nrhs; ++r) {
        double *v = sv + r * stride;
        double z0, z1;
        bool pair;
        // (a pair's values are read and written by its first column's thread)
        if (c > 0 && Lc[c - 1] != 0.0) break;
        pivot_value(Lc, f, c, p, true, v[c], c + 1 < p ? v[c + 1] : 0.0, z0, z1, pair);
        v[c] = z0;
        if (pair) v[c + 1] = z1;
      }
    }
  }
  __syncthreads();
  if (apply_lt) {
    // strips of 32 columns from the last: their products with every row past
    // them (solved pivots and the rows past the pivots), a warp four columns
    // at a time, lanes over the rows; then the 32 x 32 triangle
    for (int je = p; je > 0; je = (je - 1) & ~31) {
      const int jb = (je - 1) & ~31, nb = je - jb;
      load_tri32_async<kLvlNT>(L, sf, jb, nb, Ls);
      constexpr int CW = 32 / kLvlWarps;  // columns a warp
      const int j0 = jb + warp * CW;
      if (j0 < je) {
        auto dots = [&](int r0, auto tag) {
          constexpr int R = decltype(tag)::value;
          double acc[CW][R];
#pragma unroll
          for (int c = 0; c < CW; ++c)
#pragma unroll
            for (int q = 0; q < R; ++q) acc[c][q] = 0.0;
          for (int i = je + lane; i < f; i += 32) {
            double l[CW];
#pragma unroll
            for (int c = 0; c < CW; ++c) l[c] = j0 + c < je ? __ldg(L + (size_t)(j0 + c) * sf + i) : 0.0;
#pragma unroll
            for (int q = 0; q < R; ++q) {
              const double y = r0 + q < nrhs ? sv[(r0 + q) * stride + i] : 0.0;
#pragma unroll
              for (int c = 0; c < CW; ++c) acc[c][q] = fma(l[c], y, acc[c][q]);
            }
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int c = 0; c < CW; ++c)
#pragma unroll
              for (int q = 0; q < R; ++q) acc[c][q] += __shfl_xor_sync(0xffffffffu, acc[c][q], o);
          if (lane == 0)
#pragma unroll
            for (int c = 0; c < CW; ++c)
#pragma unroll
              for (int q = 0; q < R; ++q)
                if (j0 + c < je && r0 + q < nrhs) sv[(r0 + q) * stride + j0 + c] -= acc[c][q];
        };
        if (nrhs == 1) dots(0, std::integral_constant<int, 1>{});
        else
          for (int r0 = 0; r0 < nrhs; r0 += 4) dots(r0, std::integral_constant<int, 4>{});
      }
      cp_async_wait_all();
      __syncthreads();
      for (int r = warp; r < nrhs; r += kLvlWarps) tri_bwd_warp(sv + r * stride, jb, nb, posdef, Ls);
      __syncthreads();
    }
  }
  for (int c = tid; c < p; c += kLvlNT) {
    const int rc = rows[c];
    for (int r = 0; r < nrhs; ++r) x[(int64_t)r * P.n + rc] = sv[r * stride + c];
  }
}

}  // namespace smfg
