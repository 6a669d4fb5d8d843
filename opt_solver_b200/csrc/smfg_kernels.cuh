// Device kernels of the numeric phase: value placement, per-level front
// set-up, assembly / extend-add, front factorization by size class, the
// supernodal solves and the residual.
#pragma once
#include "smfg_aptp_host.h"
#include "smfg_internal.cuh"
#include "smfg_tc.cuh"

namespace smfg {

// counters[] slots
enum : int { kCArena = 0, kCRows = 1, kCFlags = 2, kCMaxAbs = 3, kCAux = 4, kCEffSmall = 5,
             kCActive = 6, kCGemmFlops = 7, kCTcFlops = 8, kCDeferBytes = 9, kCDeferUpd = 10,
             kCDeferSmall = 11, kCAptpMiss = 12, kCNegSoFar = 13, kCWorkSoFar = 14, kCFailLevel = 15,
             kCCount = 16 };
// error flag bits (counters[kCFlags])
enum : unsigned { kFArena = 1u, kFRows = 2u, kFNonfinite = 4u, kFNotPosdef = 8u, kFNonfiniteD = 16u,
                  kFMap = 32u, kFInternal = 64u, kFTcWait = 128u, kFTcCap = 256u, kFSteps = 512u,
                  kFAptpMiss = 1024u, kFInertia = 2048u, kFWork = 4096u, kFStatic = 8192u };
// flags after which the rest of a factorization is skipped (retried with
// more room, or reported)
constexpr unsigned kFAbort = kFArena | kFRows | kFTcWait | kFTcCap | kFAptpMiss | kFInertia | kFWork | kFStatic;
// fronts recorded per factorization that grew past the APTP size outside the
// large-front path (they join it, and the factorization is redone)
constexpr int kAptpMissCap = 1024;

__device__ __forceinline__ void set_flag(unsigned long long *cnt, unsigned bit) {
  atomicOr(cnt + kCFlags, (unsigned long long)bit);
}

// Whether the factorization is given up. For one thread of a block.
__device__ __forceinline__ bool abort_flagged(const DevFactor &X) { return (X.counters[kCFlags] & kFAbort) != 0; }

// The same answer for every thread of the block: one thread reads the flags. Kernels beside this one may set one at
// any time (the size classes of a level run side by side, and blocks of one
// launch too), and threads that read it for themselves could part: those that
// go on would pass the block's barriers without the shared data of those that
// left. Blocks may differ: the next kernel of the stream sees the flag in all.
// Every thread of the block calls it, before any of them returns.
__device__ __forceinline__ bool block_aborted(const DevFactor &X) {
  return __syncthreads_or(threadIdx.x == 0 && abort_flagged(X)) != 0;
}

// A pivot of the SPD front s failed: on the static layout, which has no room
// for delayed columns, the factorization stops there and goes on from the
// front's level on the level-by-level one. (Every front that fails in a run on
// the static layout is of one level: the next level's kernels see the flag.)
__device__ __forceinline__ void flag_not_posdef(const DevPlan &P, const DevFactor &X, int s) {
  if (X.spd_static) X.counters[kCFailLevel] = (unsigned long long)P.sn_level[s];
  set_flag(X.counters, kFNotPosdef | (X.spd_static ? kFStatic : 0u));
}

// ---------------------------------------------------------------------------
// Value placement: map_values_to_permuted + S A S (workspace.cpp:129-281,
// factor_indef.cpp:513-559). Each permuted slot sums its caller entries in
// input order, then takes v * (s_row * s_col). max |S A S| and the
// finiteness of every input value are reduced on the way.
__global__ void k_values(const double *__restrict__ vin, int64_t nnz_in, const int *__restrict__ vptr,
                         const int *__restrict__ vsrc, const int *__restrict__ pcp_col,
                         const int *__restrict__ pri, const int *__restrict__ perm,
                         const double *__restrict__ scale, int64_t nnz, double *__restrict__ pv,
                         double *__restrict__ pv_raw, unsigned long long *cnt) {
  __shared__ double red[32];
  double m = 0.0;
  bool bad = false;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz_in; k += stride)
    bad = bad || !isfinite(vin[k]);
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < nnz; s += stride) {
    double v = 0.0;
    for (int k = vptr[s]; k < vptr[s + 1]; ++k) v = __dadd_rn(v, vin[vsrc[k]]);
    pv_raw[s] = v;
    if (scale) v = __dmul_rn(v, __dmul_rn(scale[perm[pri[s]]], scale[perm[pcp_col[s]]]));
    pv[s] = v;
    m = fmax(m, fabs(v));
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) set_flag(cnt, kFNonfinite);
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) atomicMax(cnt + kCMaxAbs, (unsigned long long)__double_as_longlong(m));
  }
}

// eff_small of factor_indef.cpp:631-636 from max |S A S|; on the static
// layout the arena and rows in use.
__global__ void k_eff_small(unsigned long long *cnt, double small_pivot, long long arena, long long rows) {
  cnt[kCArena] = (unsigned long long)arena;
  cnt[kCRows] = (unsigned long long)rows;
  const double m = __longlong_as_double((long long)cnt[kCMaxAbs]);
  const double e = (m > 0.0 && m < small_pivot) ? small_pivot * m : small_pivot;
  cnt[kCEffSmall] = (unsigned long long)__double_as_longlong(e);
}

// A factorization that failed on the static layout goes on level by level: its
// flags cleared, the arena and rows in use those of the levels below.
__global__ void k_resume(unsigned long long *cnt, long long arena, long long rows) {
  cnt[kCFlags] &= ~(unsigned long long)(kFStatic | kFNotPosdef);
  cnt[kCArena] = (unsigned long long)arena;
  cnt[kCRows] = (unsigned long long)rows;
}

// ---------------------------------------------------------------------------
// Per-level set-up (one block): realized front sizes (delays in), storage
// offsets by exclusive scan, delay offsets of the children in the parent's
// row list (multifrontal_serial.cpp:510-545), assembly work items.
template <int NT>
__global__ void k_level_setup(DevPlan P, DevFactor X, int lo, int hi, int lvl, int nb, int fuse, int cols) {
  static_assert(NT % 32 == 0 && NT <= 1024, "block size");
  constexpr int NW = NT / 32;
  __shared__ long long wa[NW], wr[NW], wb[NW];
  __shared__ long long base_a, base_r, run_a, run_r, run_b;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long *cnt = X.counters;
  if (threadIdx.x == 0) {
    base_a = (long long)cnt[kCArena];
    base_r = (long long)cnt[kCRows];
    run_a = run_r = run_b = 0;
  }
  __syncthreads();
  for (int c0 = lo; c0 < hi; c0 += NT) {
    const int i = c0 + threadIdx.x;
    long long fa = 0, fr = 0, fb = 0;
    int s = -1, f = 0;
    if (i < hi) {
      s = P.lvl_sn[i];
      int nd = 0;
      for (int t = P.child_ptr[s]; t < P.child_ptr[s + 1]; ++t) {
        X.child_doff[t] = nd;
        nd += X.sn_dout[P.child_idx[t]];
      }
      f = nd + P.sn_fsym[s];
      X.sn_nd[s] = nd;
      X.sn_f[s] = f;
      X.sn_ne[s] = nd + P.sn_width[s];
      fa = (long long)f * f + (long long)f * nb;
      fr = f;
      // (fronts of at most fuse rows are assembled by their front kernel)
      fb = (f <= fuse && !P.sn_large[s]) ? 0 : (f + cols - 1) / cols;
    }
    // inclusive block scan of (fa, fr, fb): warp shuffles, then the warps'
    // totals scanned by warp 0
    long long va = fa, vr = fr, vb = fb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long ya = __shfl_up_sync(0xffffffffu, va, o);
      const long long yr = __shfl_up_sync(0xffffffffu, vr, o);
      const long long yb = __shfl_up_sync(0xffffffffu, vb, o);
      if (lane >= o) {
        va += ya;
        vr += yr;
        vb += yb;
      }
    }
    if (lane == 31) {
      wa[warp] = va;
      wr[warp] = vr;
      wb[warp] = vb;
    }
    __syncthreads();
    if (warp == 0) {
      long long ta = lane < NW ? wa[lane] : 0, tr = lane < NW ? wr[lane] : 0, tb = lane < NW ? wb[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const long long ya = __shfl_up_sync(0xffffffffu, ta, o);
        const long long yr = __shfl_up_sync(0xffffffffu, tr, o);
        const long long yb = __shfl_up_sync(0xffffffffu, tb, o);
        if (lane >= o) {
          ta += ya;
          tr += yr;
          tb += yb;
        }
      }
      if (lane < NW) {
        wa[lane] = ta;
        wr[lane] = tr;
        wb[lane] = tb;
      }
    }
    __syncthreads();
    if (warp > 0) {
      va += wa[warp - 1];
      vr += wr[warp - 1];
      vb += wb[warp - 1];
    }
    if (i < hi) {
      X.sn_off[s] = base_a + run_a + va - fa;
      X.sn_roff[s] = base_r + run_r + vr - fr;
      X.lvl_blk[i + lvl] = (int)(run_b + vb - fb);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      run_a += wa[NW - 1];
      run_r += wr[NW - 1];
      run_b += wb[NW - 1];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    X.lvl_blk[hi + lvl] = (int)run_b;
    cnt[kCArena] = (unsigned long long)(base_a + run_a);
    cnt[kCRows] = (unsigned long long)(base_r + run_r);
    cnt[kCAux] = (unsigned long long)run_b;
    if (base_a + run_a > X.arena_cap) set_flag(cnt, kFArena);
    if (base_r + run_r > X.rows_cap) set_flag(cnt, kFRows);
  }
}

// Rows of each front of more than fuse rows (children's delayed rows in child
// order, then its symbolic rows) and each child's contribution-block row map
// into it. Fronts P.lvl_sn[lo + block].
// STATIC: the SPD layout made ahead of any factorization (no delays, the
// children's pivots are their widths).
template <bool STATIC>
__global__ void k_level_rows(DevPlan P, DevFactor X, int lo, int fuse) {
  if (!STATIC && block_aborted(X)) return;
  const int s = P.lvl_sn[lo + blockIdx.x];
  const int64_t roff = X.sn_roff[s];
  const int nd = X.sn_nd[s], f = X.sn_f[s], fsym = P.sn_fsym[s];
  if (f <= fuse && !P.sn_large[s]) return;
  int *rows = X.rows + roff;
  for (int t = P.child_ptr[s]; t < P.child_ptr[s + 1]; ++t) {
    const int c = P.child_idx[t];
    const int dc = STATIC ? 0 : X.sn_dout[c];
    const int pc = STATIC ? P.sn_width[c] : X.sn_p[c];
    const int fc = X.sn_f[c];
    const int q = fc - pc;
    const int doff = X.child_doff[t];
    const int *crow = X.rows + X.sn_roff[c] + pc;
    int *cmap = X.cbmap + X.sn_roff[c] + pc;
    const int *cpr = P.cpr_idx + P.cpr_off[t];
    for (int u = threadIdx.x; u < q; u += blockDim.x) {
      if (u < dc) {
        rows[doff + u] = crow[u];
        cmap[u] = doff + u;
      } else {
        cmap[u] = nd + cpr[u - dc];
      }
    }
  }
  const int *fr = P.frow_idx + P.frow_ptr[s];
  for (int u = threadIdx.x; u < fsym; u += blockDim.x) rows[nd + u] = fr[u];
  for (int u = threadIdx.x; u < f; u += blockDim.x) X.tags[roff + u] = 0;
}

// First index in [lo, hi) of the increasing a[] whose value is >= key (hi
// if none), by the 32 lanes of a warp: 32 probes a round (one load
// latency), about three rounds for a few thousand entries.
__device__ __forceinline__ int warp_lower_bound(const int *__restrict__ a, int lo, int hi, int key) {
  const int lane = threadIdx.x & 31;
  while (hi - lo > 32) {
    const int step = (hi - lo + 31) / 32;
    const int pos = min(lo + step * (lane + 1) - 1, hi - 1);
    const int nl = __popc(__ballot_sync(0xffffffffu, a[pos] < key));  // a prefix of the lanes
    const int nlo = min(lo + step * nl, hi);
    hi = nl == 32 ? hi : min(lo + step * (nl + 1), hi);
    lo = nlo;
  }
  const int pos = lo + lane;
  return lo + __popc(__ballot_sync(0xffffffffu, pos < hi && a[pos] < key));
}

// Assembly of one level's fronts past the fused sizes (process_front,
// multifrontal_serial.cpp:720-789): each work item is a block of `cols` columns
// of one front. An entry is zero, plus its original value (pivot columns), plus
// the children's Schur blocks in child order (the reference's order of
// additions, so every entry is the reference's sum); a child's block is read in
// place from its own front.
//
// Gather form (at most kAsmKids children whose inverse row maps fit in shared
// memory, kAsmMap entries): every entry is formed in a register -- zero, then the
// children in order, each read at the row its inverse map gives -- and
// written once; the few entries with an original value are formed again from
// it. It replaces a zeroing pass and a read-modify-write pass a child, whose
// dependent loads bound it (64^3 operator: 4.2 -> 3.4 ms a factorization, a
// level of 1,500-row fronts 290 -> 200 us for 310 MB). Fronts whose maps do
// not fit take the passes: the lower part of the item's columns zeroed, the
// original entries added, then each child's block.
constexpr int kAsmMap = 12288, kAsmKids = 16;

__global__ void __launch_bounds__(256) k_level_assemble(DevPlan P, DevFactor X, int lo, int hi, int lvl, int cols) {
  unsigned long long *cnt = X.counters;
  if (block_aborted(X)) return;
  const int *pref = X.lvl_blk + lo + lvl;  // m + 1 prefix entries
  const int m = hi - lo;
  const int total = pref[m];
  __shared__ int rng[2];
  __shared__ __align__(16) unsigned short inv[kAsmMap];
  __shared__ long long ch_off[kAsmKids], ch_map[kAsmKids];
  __shared__ int ch_f[kAsmKids], ch_q[kAsmKids];
  int have = -1;  // the front whose inverse maps are in inv
  for (int w = blockIdx.x; w < total; w += gridDim.x) {
    int a = 0, b = m;  // largest i with pref[i] <= w
    while (b - a > 1) {
      const int mid = (a + b) >> 1;
      if (pref[mid] <= w) a = mid;
      else b = mid;
    }
    const int s = P.lvl_sn[lo + a];
    const int f = X.sn_f[s], nd = X.sn_nd[s];
    const int j0 = (w - pref[a]) * cols;
    const int j1 = min(j0 + cols, f);
    double *F = X.arena + X.sn_off[s];
    const size_t sf = (size_t)f;
    const int t0 = P.child_ptr[s], nk = P.child_ptr[s + 1] - t0;
    if (nk <= kAsmKids && (long long)nk * f <= kAsmMap && f < 65535) {
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
      if (have != s) {
        __syncthreads();  // the item before has read its maps
        for (int k = threadIdx.x; k < nk * f; k += blockDim.x) inv[k] = 0xffff;
        if ((int)threadIdx.x < nk) {
          const int c = P.child_idx[t0 + threadIdx.x];
          const int pc = X.sn_p[c], fc = X.sn_f[c];
          ch_f[threadIdx.x] = fc;
          ch_q[threadIdx.x] = fc - pc;
          ch_map[threadIdx.x] = X.sn_roff[c] + pc;
          ch_off[threadIdx.x] = X.sn_off[c] + (long long)pc * fc + pc;
        }
        __syncthreads();
        for (int t = 0; t < nk; ++t) {
          const int *cmap = X.cbmap + ch_map[t];
          bool bad = false;
          for (int u = threadIdx.x; u < ch_q[t]; u += blockDim.x) {
            const int r = cmap[u];
            bad = bad || (u > 0 && cmap[u - 1] >= r);  // (maps increase)
            inv[t * f + r] = (unsigned short)u;
          }
          if (bad) set_flag(cnt, kFMap);
        }
        __syncthreads();
        have = s;
      }
      for (int jj = j0 + warp; jj < j1; jj += nwarp) {
        double *Fj = F + jj * sf;
        for (int i0 = jj + lane; i0 < f; i0 += 4 * 32) {
          double v[4] = {0.0, 0.0, 0.0, 0.0};
          for (int t = 0; t < nk; t += 2) {  // two children's loads in flight
            double x[2][4];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int tt = min(t + e, nk - 1);
              // (the same for the whole warp)
              const int uj = t + e < nk ? inv[tt * f + jj] : 0xffff;
              const double *Fc = X.arena + ch_off[tt] + (size_t)(uj == 0xffff ? 0 : uj) * ch_f[tt];
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const int ui = (uj != 0xffff && i0 + 32 * u < f) ? inv[tt * f + i0 + 32 * u] : 0xffff;
                x[e][u] = ui != 0xffff ? Fc[ui] : -0.0;  // (v + -0.0 is v)
              }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = (v[u] + x[0][u]) + x[1][u];
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (i0 + 32 * u < f) Fj[i0 + 32 * u] = v[u];
        }
      }
      // entries with an original value: it, then the children in order
      const int cs = P.sn_start[s], wdt = P.sn_width[s];
      const int ca = max(j0 - nd, 0), cb = min(j1 - nd, wdt);
      if (ca < cb) {
        __syncthreads();
        const int k0 = P.pcp[cs + ca], k1 = P.pcp[cs + cb];
        for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
          const int col = nd + P.pcol[k] - cs, row = nd + P.amap[k];
          double v = 0.0 + X.pv[k];
          for (int t = 0; t < nk; ++t) {
            const int uj = inv[t * f + col], ui = inv[t * f + row];
            if (uj != 0xffff && ui != 0xffff) v += X.arena[ch_off[t] + (size_t)uj * ch_f[t] + ui];
          }
          F[(size_t)col * sf + row] = v;
        }
      }
      continue;
    }
    have = -1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    __syncthreads();
    // 1. zero the lower part of columns [j0, j1): a warp per column
    for (int jj = j0 + warp; jj < j1; jj += nwarp) {
      double *Fj = F + jj * sf;
      for (int i = jj + lane; i < f; i += 32) Fj[i] = 0.0;
    }
    __syncthreads();
    // 2. original entries of the pivot columns in [j0, j1): their slots are
    // one contiguous range (consecutive columns), each slot a distinct entry
    const int cs = P.sn_start[s], wdt = P.sn_width[s];
    const int ca = max(j0 - nd, 0), cb = min(j1 - nd, wdt);
    if (ca < cb) {
      const int k0 = P.pcp[cs + ca], k1 = P.pcp[cs + cb];
      for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        int c = ca;  // the column of slot k (at most cols candidates)
        while (c + 1 < cb && P.pcp[cs + c + 1] <= k) ++c;
        F[(nd + c) * sf + nd + P.amap[k]] += X.pv[k];
      }
    }
    __syncthreads();
    // 3. children in order
    for (int t = P.child_ptr[s]; t < P.child_ptr[s + 1]; ++t) {
      const int c = P.child_idx[t];
      const int pc = X.sn_p[c], fc = X.sn_f[c];
      const int q = fc - pc;
      if (q <= 0) continue;
      const int *cmap = X.cbmap + X.sn_roff[c] + pc;
      // the child's CB rows mapped into [j0, j1): warp 0 finds the first
      // with cmap >= j0, warp 1 the first with cmap >= j1
      if (warp < 2) {
        const int r = warp_lower_bound(cmap, 0, q, warp == 0 ? j0 : j1);
        if (lane == 0) rng[warp] = r;
      }
      __syncthreads();
      const int ja = rng[0], jb = rng[1];
      const double *Fc = X.arena + X.sn_off[c];
      const size_t sfc = (size_t)fc;
      // the child's block columns [ja, jb): a warp per column, lanes over
      // its rows (contiguous in the child, increasing in the parent), four a
      // lane in flight; its targets are distinct
      for (int jj = ja + warp; jj < jb; jj += nwarp) {
        const int lj = cmap[jj];
        const double *Fcj = Fc + (size_t)(pc + jj) * sfc + pc;
        double *Fj = F + (size_t)lj * sf;
        for (int i0 = jj + lane; i0 < q; i0 += 4 * 32) {
          double sv[4], dv[4];
          int li[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int ii = i0 + 32 * u;
            li[u] = -1;
            sv[u] = dv[u] = 0.0;
            if (ii < q) {
              li[u] = cmap[ii];
              if (li[u] < lj) {
                set_flag(cnt, kFMap);
                li[u] = -1;
              } else {
                sv[u] = Fcj[ii];
                dv[u] = Fj[li[u]];
              }
            }
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (li[u] >= 0) Fj[li[u]] = dv[u] + sv[u];
        }
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------------
template <int NT, bool SMEM>
__device__ void store_front(DevPlan &P, DevFactor &X, int s, const FrontRef &v, int p,
                            const PivotParams &prm, FrontShared &sh, int *inv, double *Fg,
                            int *rows_g, int8_t *tags_g);

// Fronts of at least this many symbolic rows take the multi-block path.
constexpr int kLargeMin = 384;
// SPD fronts already from fewer: one block takes a front of 380 rows 400 us,
// the multi-block steps 130 (one SM's FP64 rate bounds the block). Measured
// with 384 / 256 / 192 / 144: 701 x 433 Laplacian 6.85 / 5.75 / 5.64 / 5.79 ms,
// 23 x 19 x 21 operator 4.39 / 4.04 / 3.93 / 3.95, 64^3 36.8 / 37.1 / 37.2 / 37.7
// (more fronts a level in the multi-block kernels).
constexpr int kLargeMinSpd = 192;

// Unit-LDL^T of the nbp x nbp lower block T (the SPD panels' diagonal
// blocks), all 256 threads or more: pivot k's value to dv[k], its reciprocal
// to linv[k], its multipliers l_kj = t_jk / d_k to lm[k][j]; every entry (i, j),
// k < j <= i, takes t_ij - t_ik l_kj (skipped for l_kj = 0) in pivot order,
// multiply and subtract rounded separately. Columns past the pivots taken
// keep their updated values in T. Stops at the first pivot that is not
// positive and finite; returns the pivots taken. Starts and ends at a
// barrier. `zero` (shared, optional) is set to 1 when a multiplier is zero.
//
// A chain of pivots, bound by latency: two pivots a barrier (each thread
// forms the second pivot's column entries it needs itself, from the two
// columns as they stood), a block of 16 in 6,700 cycles of a launch against
// 7,300. With EXT the 16 rows below the block (T rows NB..) and the second
// panel's diagonal block ride along: the rows take the same eliminations,
// their unscaled values w to Wr[row][pivot] and multipliers to Lr, and v2, the
// thread's entry of the second block, its fused chain c = fma(-l, w, c) (w = 0
// skipped) -- in place of a chain of 16 steps on 16 threads after the block
// (3,600 cycles). One pivot a barrier with the same additions: 19.6 us a
// launch on the 64^3 operator against 17.1.
template <int NB, bool EXT, int NT = 256>
__device__ __forceinline__ int spd_diag_factor(double (*T)[NB + 1], double (*lm)[NB], double *linv, double *dv, int nbp,
                                               int *zero = nullptr, int next = 0, double (*Wr)[NB] = nullptr,
                                               double (*Lr)[NB] = nullptr, double *v2 = nullptr) {
  static_assert(NB * NB <= NT, "an entry a thread");
  const int t = threadIdx.x, ti = t / NB, tj = t % NB;
  const bool mine = t < NB * NB;
  __syncthreads();
  int k = 0;
  while (k < nbp) {
    const double d = T[k][k];
    if (!(d > 0.0 && isfinite(d))) break;
    const double inv = __drcp_rn(d);  // 1.0 / d, correctly rounded
    // columns k and k + 1 at this thread's rows
    double ci = 0.0, cj = 0.0, cr = 0.0, cq = 0.0, bi = 0.0, bj = 0.0, br = 0.0, bq = 0.0;
    const bool pair = k + 1 < nbp;
    double lp = 0.0, d1 = 0.0;
    if (pair) {
      const double cp = T[k + 1][k], bp = T[k + 1][k + 1];
      lp = __dmul_rn(cp, inv);
      const double u = __dsub_rn(bp, __dmul_rn(cp, lp));
      d1 = lp != 0.0 ? u : bp;
    }
    const bool two = pair && d1 > 0.0 && isfinite(d1);
    if (mine) {
      ci = T[ti][k];
      cj = T[tj][k];
      bi = T[ti][k + 1 < NB ? k + 1 : k];
      bj = T[tj][k + 1 < NB ? k + 1 : k];
      if (EXT) {
        cr = T[NB + ti][k];
        cq = T[NB + tj][k];
        br = T[NB + ti][k + 1 < NB ? k + 1 : k];
        bq = T[NB + tj][k + 1 < NB ? k + 1 : k];
      }
    }
    // (the second failed: column k + 1, which every thread has read, is
    // written below)
    if (pair && !two) __syncthreads();
    const double inv1 = two ? __drcp_rn(d1) : 0.0;
    if (mine) {
      const double lj = __dmul_rn(cj, inv);
      // pivot k on column k + 1 (its entries as pivot k + 1 finds them)
      auto step = [&](double b, double c) {
        const double u = __dsub_rn(b, __dmul_rn(c, lp));
        return lp != 0.0 ? u : b;
      };
      bi = step(bi, ci);
      bj = step(bj, cj);
      if (EXT) {
        br = step(br, cr);
        bq = step(bq, cq);
      }
      const double lj1 = __dmul_rn(bj, inv1);
      const int last = two ? k + 1 : k;
      auto entry = [&](double v, double c, double b) {
        const double u = __dsub_rn(v, __dmul_rn(c, lj));
        v = lj != 0.0 ? u : v;
        const double w = __dsub_rn(v, __dmul_rn(b, lj1));
        return two && lj1 != 0.0 ? w : v;
      };
      // (the columns of the pivots taken are not needed any more; column
      // k + 1 alone when it failed)
      if (tj > last && tj <= ti && ti < nbp) T[ti][tj] = entry(T[ti][tj], ci, bi);
      if (EXT && tj > last && tj < nbp && ti < next) T[NB + ti][tj] = entry(T[NB + ti][tj], cr, br);
      if (ti == 0) {
        if (tj > k && tj < nbp) {
          lm[k][tj] = lj;
          if (zero && lj == 0.0) *zero = 1;
        }
        if (two && tj > k + 1 && tj < nbp) {
          lm[k + 1][tj] = lj1;
          if (zero && lj1 == 0.0) *zero = 1;
        }
        if (tj == k) {
          linv[k] = inv;
          dv[k] = d;
        }
        if (two && tj == k + 1) {
          linv[k + 1] = inv1;
          dv[k + 1] = d1;
        }
      }
      if (EXT) {
        const double a0 = __dmul_rn(cr, inv), a1 = __dmul_rn(br, inv1);
        if (tj == 0 && ti < next) {
          Wr[ti][k] = cr;
          Lr[ti][k] = a0;
          if (cr == 0.0) *zero = 1;
          if (two) {
            Wr[ti][k + 1] = br;
            Lr[ti][k + 1] = a1;
            if (br == 0.0) *zero = 1;
          }
        }
        const double y0 = fma(-a0, cq, *v2);
        if (cq != 0.0) *v2 = y0;
        const double y1 = fma(-a1, bq, *v2);
        if (two && bq != 0.0) *v2 = y1;
      }
    }
    __syncthreads();
    k += two ? 2 : 1;
    if (pair && !two) break;
  }
  return k;
}

// SPD fronts of the blocked size classes (nb = 16, at least
// blocked_min_front rows) in their one block of threads: the medium
// kernel's pivoting steps (tpp_step_blk, one pivot at a time) replaced by
// the large fronts' panel arithmetic. Panels of 16 pivots: the diagonal
// block factored by all threads (spd_diag_factor), every row of the
// panel's columns by one thread (the multiply-subtract chain of
// k_large_panel_spd2's rows, w kept in W), then the medium kernel's own
// deferred update of the eligible columns and, at the end, its Schur update
// of the contribution block. A pivot that is not positive ends the
// pivoting. Returns the pivots taken.
template <int NT>
__device__ int spd_front_panels(FrontRef &v, const PivotParams &prm, FrontShared &sh) {
  constexpr int NB = 16;
  __shared__ double T[NB][NB + 1], lm[NB][NB], linv[NB], dv[NB];
  const int f = v.f, ne = v.ne;
  const size_t sf = (size_t)v.ld;
  double *F = v.F, *W = v.W;  // W row q (f doubles): w of the panel's pivot q
  int p = 0;
  for (int ps = 0; ps < ne; ps += NB) {
    const int pe = min(ne, ps + NB), nbp = pe - ps;
    for (int t = threadIdx.x; t < NB * NB; t += NT) {
      const int r = t / NB, c = t % NB;
      T[r][c] = (r < nbp && c <= r) ? F[(size_t)(ps + c) * sf + ps + r] : 0.0;
    }
    const int np = spd_diag_factor<NB, false, NT>(T, lm, linv, dv, nbp);
    for (int i = ps + threadIdx.x; i < f; i += NT) {
      double a[NB];
#pragma unroll
      for (int c = 0; c < NB; ++c) a[c] = (c < nbp && ps + c <= i) ? F[(size_t)(ps + c) * sf + i] : 0.0;
#pragma unroll
      for (int k = 0; k < NB; ++k) {
        if (k < np && i > ps + k) {
          const double w = a[k];
          W[(size_t)k * f + i] = w;
#pragma unroll
          for (int j = k + 1; j < NB; ++j) {
            if (j < nbp && ps + j <= i) {
              const double l = lm[k][j];
              if (l != 0.0) a[j] = __dsub_rn(a[j], __dmul_rn(w, l));
            }
          }
          a[k] = __dmul_rn(w, linv[k]);
        }
      }
#pragma unroll
      for (int c = 0; c < NB; ++c)
        if (c < nbp && ps + c <= i) F[(size_t)(ps + c) * sf + i] = a[c];
    }
    if (threadIdx.x == 0) {
      for (int k = 0; k < np; ++k) {
        v.tags[ps + k] = 1;
        inertia_1x1(dv[k], prm.eff_small, sh.st);
        const double rem = (double)(f - (ps + k + 1));
        sh.st.flops += rem + rem * (rem + 1.0);
      }
    }
    p = ps + np;
    __syncthreads();
    if (np < nbp) break;
    // the eligible columns past the panel, every row below: the medium
    // kernel's deferred update
    deferred_update_blk<NT>(v, ps, pe, pe, ne);
  }
  // the contribution block: its Schur update over every pivot, as the
  // medium kernel takes it
  schur_update_blk<NT>(v, 0, p, ne, NB);
  return p;
}

// Front factorization + store (process_front's kernel call and D handling,
// multifrontal_serial.cpp:790-945): one block per front of the size class
// [FMIN, FMAX]; SMEM: the front is copied into shared memory.
template <int NT, bool SMEM>
__device__ void factor_one_front(DevPlan &P, DevFactor &X, int s, const PivotParams &prm0,
                                 double *smem) {
  __shared__ FrontShared sh;
  const int f = X.sn_f[s], ne = X.sn_ne[s], nb = prm0.nb;
  const size_t sf = (size_t)f;
  double *Fg = X.arena + X.sn_off[s];
  int *rows_g = X.rows + X.sn_roff[s];
  int8_t *tags_g = X.tags + X.sn_roff[s];
  PivotParams prm = prm0;
  prm.eff_small = __longlong_as_double((long long)X.counters[kCEffSmall]);
  FrontRef v;
  v.ld = SMEM ? smem_front_ld(f, nb) : f;
  v.f = f;
  v.ne = ne;
  int *inv;
  if (SMEM) {
    // F, then W only where the blocked path runs (the launch's shared
    // memory holds W only for buckets that can reach it), then the ints
    const bool blocked = f >= prm0.blocked_min_front && nb > 1;
    double *F = smem;
    double *W = F + sf * v.ld;
    int *rows = (int *)(W + (blocked ? sf * nb : 0));
    int *loc = rows + f;
    inv = loc + f;
    int8_t *tags = (int8_t *)(inv + f);
    // the lower part, a warp per column, four columns in flight
    constexpr int NWF = NT / 32;
    const int lane = threadIdx.x & 31;
    for (int j0 = threadIdx.x >> 5; j0 < f; j0 += 4 * NWF)
      for (int i = j0 + lane; i < f; i += 32) {
        double x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = (j0 + u * NWF <= i) ? Fg[(size_t)(j0 + u * NWF) * f + i] : 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (j0 + u * NWF <= i) F[(size_t)(j0 + u * NWF) * v.ld + i] = x[u];
      }
    for (int t = threadIdx.x; t < f; t += NT) {
      rows[t] = rows_g[t];
      loc[t] = t;
      tags[t] = 0;
    }
    v.F = F;
    v.W = W;
    v.rows = rows;
    v.tags = tags;
    v.loc = loc;
  } else {
    v.F = Fg;
    v.W = Fg + sf * sf;
    v.rows = rows_g;
    v.tags = tags_g;
    v.loc = X.ploc + X.sn_roff[s];
    inv = X.ploc + X.rows_cap + X.sn_roff[s];
    for (int t = threadIdx.x; t < f; t += NT) v.loc[t] = t;
  }
  if (threadIdx.x == 0) sh.st = FrontStats{0, 0, 0, 0, 0.0};
  __syncthreads();
  const bool spd_panels = prm.posdef && nb == 16 && f >= prm0.blocked_min_front && NT >= 128;
  const int p = spd_panels ? spd_front_panels<NT>(v, prm, sh) : ldlt_factor_front_blk<NT>(v, prm, sh);
  store_front<NT, SMEM>(P, X, s, v, p, prm, sh, inv, Fg, rows_g, tags_g);
}

// D and the stored L of a factored front, its counts, and its children's
// row maps in pivot order (multifrontal_serial.cpp:884-945).
template <int NT, bool SMEM>
__device__ void store_front(DevPlan &P, DevFactor &X, int s, const FrontRef &v, int p,
                            const PivotParams &prm, FrontShared &sh, int *inv, double *Fg,
                            int *rows_g, int8_t *tags_g) {
  const int f = v.f, ne = v.ne;
  const size_t sf = (size_t)v.ld;
  const bool is_root = P.sn_parent[s] < 0;
  int pstore = p;
  if (is_root && p < ne) {
    for (int c = p + threadIdx.x; c < ne; c += NT) v.tags[c] = 0;
    if (threadIdx.x == 0) sh.st.zero += ne - p;
    pstore = ne;
  }
  __syncthreads();
  if (prm.posdef) {
    if (p < ne && threadIdx.x == 0) flag_not_posdef(P, X, s);
    // L = L_unit sqrt(D), upper part zero
    // (a warp per column: its square root taken once)
    for (int c = threadIdx.x >> 5; c < pstore; c += NT / 32) {
      double *Lc = v.F + (size_t)c * sf;
      const double sq = sqrt(Lc[c]);
      __syncwarp();
      for (int i = threadIdx.x & 31; i < f; i += 32) Lc[i] = i < c ? 0.0 : i == c ? sq : __dmul_rn(Lc[i], sq);
    }
  } else {
    // D inline: d on the diagonal, a 2x2 block's off-diagonal in the upper
    // slot (c, c + 1); zero pivots' columns zero.
    bool bad = false;
    for (int c = threadIdx.x; c < pstore; c += NT) {
      const double *Lc = v.F + (size_t)c * sf;
      const int8_t tag = v.tags[c];
      if (tag == 1) bad = bad || !isfinite(Lc[c]);
      else if (tag == 2) bad = bad || !isfinite(Lc[c]) || !isfinite(Lc[c + 1]) || !isfinite(Lc[sf + c + 1]);
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) set_flag(X.counters, kFNonfiniteD);
    for (int c = threadIdx.x; c < pstore; c += NT) {
      if (v.tags[c] == -1) {  // move d10 from (c, c-1) to the upper slot (c-1, c)
        double *Lc = v.F + (size_t)c * sf;
        Lc[c - 1] = v.F[(size_t)(c - 1) * sf + c];
      }
    }
    __syncthreads();
    for (int c = threadIdx.x >> 5; c < pstore; c += NT / 32) {
      double *Lc = v.F + (size_t)c * sf;
      const int8_t tag = v.tags[c];
      const int end = tag == 0 ? f : tag == 2 ? c + 2 : c;  // rows past it keep their values
      for (int i = threadIdx.x & 31; i < end; i += 32)
        if (tag == 0 || (i != c && !(tag == -1 && i == c - 1))) Lc[i] = 0.0;
    }
  }
  __syncthreads();
  if (SMEM) {
    // the pivot columns whole, the contribution block's lower part
    for (int c = threadIdx.x >> 5; c < f; c += NT / 32)
      for (int i = (c < pstore ? 0 : c) + (int)(threadIdx.x & 31); i < f; i += 32) Fg[(size_t)c * f + i] = v.F[c * sf + i];
    for (int t = threadIdx.x; t < f; t += NT) {
      rows_g[t] = v.rows[t];
      tags_g[t] = v.tags[t];
    }
  }
  // The children's row maps, built in assembly order, now point at the
  // rows' final (pivot-order) positions: the solves read them that way.
  if (!prm.posdef) {  // (SPD rows keep their order)
    for (int t = threadIdx.x; t < f; t += NT) inv[v.loc[t]] = t;
    __syncthreads();
    for (int t = P.child_ptr[s]; t < P.child_ptr[s + 1]; ++t) {
      const int c = P.child_idx[t];
      const int pc = X.sn_p[c];
      int *cmap = X.cbmap + X.sn_roff[c] + pc;
      for (int u = threadIdx.x; u < X.sn_f[c] - pc; u += NT) cmap[u] = inv[cmap[u]];
    }
  }
  if (threadIdx.x == 0) {
    X.sn_p[s] = p;
    X.sn_pstore[s] = pstore;
    X.sn_dout[s] = is_root ? 0 : ne - p;
    int *st = X.sn_stat + 4 * s;
    st[0] = sh.st.pos;
    st[1] = sh.st.neg;
    st[2] = sh.st.zero;
    st[3] = sh.st.two_by_two;
    X.sn_flops[s] = sh.st.flops;
  }
}

// Fronts of fmin..fmax rows among P.lvl_sn[i0 + block].
template <int NT, bool SMEM>
__global__ void __launch_bounds__(NT) k_factor(DevPlan P, DevFactor X, int i0, PivotParams prm, int fmin, int fmax) {
  extern __shared__ __align__(16) double smem[];
  if (block_aborted(X)) return;
  const int s = P.lvl_sn[i0 + blockIdx.x];
  const int f = X.sn_f[s];
  if (f < fmin || f > fmax || P.sn_large[s]) return;
  if (!SMEM && prm.aptp_min > 0 && !prm.posdef && f >= prm.aptp_min && prm.u >= kWeakPivotRatio) {
    // delays took the front to the APTP size: it must take the large-front
    // path; recorded, and the factorization is redone
    if (threadIdx.x == 0) {
      const unsigned long long i = atomicAdd(X.counters + kCAptpMiss, 1ull);
      if (i < (unsigned long long)kAptpMissCap) X.aptp_miss[i] = s;
      set_flag(X.counters, kFAptpMiss);
    }
    return;
  }
  factor_one_front<NT, SMEM>(P, X, s, prm, smem);
}

// ---------------------------------------------------------------------------
// Large fronts: one block per front steps the blocked pivoting (tpp_step_blk)
// while all blocks of the GPU run its deferred updates and, at the end, its
// Schur update, as tiled GEMMs whose every entry takes the same fused
// multiply-adds in the same pivot order as the block kernel.

__device__ __forceinline__ FrontRef large_view(DevPlan &P, DevFactor &X, int s) {
  FrontRef v;
  const int f = X.sn_f[s];
  v.F = X.arena + X.sn_off[s];
  v.ld = f;
  v.f = f;
  v.ne = X.sn_ne[s];
  v.rows = X.rows + X.sn_roff[s];
  v.tags = X.tags + X.sn_roff[s];
  v.W = v.F + (size_t)f * f;
  v.loc = X.ploc + X.sn_roff[s];
  v.inv = X.ploc + X.rows_cap + X.sn_roff[s];
  return v;
}

// The state of each large front of a level before its first step. The kernels
// of the steps and of the Schur update take every decision from it, without a
// look at the abort flags: a team's CTAs and a launch's blocks agree, and
// nothing is asked for of a front that is closed here because the factorization
// is given up. (A flag set later, by a kernel beside them, costs the rest of
// the level's work; the test in each of them cost 0.7% of a 64^3 factorization.)
__global__ void k_large_init(DevPlan P, DevFactor X, const int *__restrict__ large, int nlarge,
                             int posdef, int nbo) {
  if (block_aborted(X)) {
    if (threadIdx.x == 0) {
      TppState S;
      tpp_init(S, 0, posdef != 0);
      S.phase = 2;
      X.tpp[blockIdx.x] = S;
    }
    return;
  }
  const int s = large[blockIdx.x];
  const int f = X.sn_f[s];
  int *loc = X.ploc + X.sn_roff[s];
  int *inv = X.ploc + X.rows_cap + X.sn_roff[s];
  for (int t = threadIdx.x; t < f && !posdef; t += blockDim.x) {
    loc[t] = t;
    inv[t] = t;
  }
  if (threadIdx.x == 0) {
    TppState S;
    const bool mixed = X.sn_mixed != nullptr && X.sn_mixed[s] != 0 && nbo > 0;
    tpp_init(S, X.sn_ne[s], posdef != 0, mixed, nbo);
    S.pad[0] = 0;  // deferred update pending
    S.f = f;
    S.ne = X.sn_ne[s];
    S.off = X.sn_off[s];
    X.tpp[blockIdx.x] = S;
  }
}

// The early stops of an indefinite factorization, after each level
// (multifrontal_serial.cpp:1619-1628, :660-671): the negative pivots and the
// front work (fully summed columns x rows^2, exact integers) of the fronts
// factored so far; past max_negative_pivots (neg_limit >= 0) or past the
// work cap (work_cap >= 0) the rest of the factorization is skipped. Both
// counts only grow, so a run that stops is exactly one whose finished count
// would have passed the limit.
__global__ void k_level_limits(DevPlan P, DevFactor X, int lo, int hi, long long neg_limit, long long work_cap) {
  __shared__ long long red[2][32];
  if (block_aborted(X)) return;
  long long neg = 0, work = 0;
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    const int s = P.lvl_sn[i];
    const long long f = X.sn_f[s];
    neg += X.sn_stat[4 * s + 1];
    work += (long long)X.sn_ne[s] * f * f;
  }
  for (int o = 16; o > 0; o >>= 1) {
    neg += __shfl_xor_sync(0xffffffffu, neg, o);
    work += __shfl_xor_sync(0xffffffffu, work, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = neg;
    red[1][threadIdx.x >> 5] = work;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    neg = work = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      neg += red[0][w];
      work += red[1][w];
    }
    const long long tn = (long long)atomicAdd(X.counters + kCNegSoFar, (unsigned long long)neg) + neg;
    const long long tw = (long long)atomicAdd(X.counters + kCWorkSoFar, (unsigned long long)work) + work;
    if (neg_limit >= 0 && tn > neg_limit) set_flag(X.counters, kFInertia);
    if (work_cap >= 0 && tw > work_cap) set_flag(X.counters, kFWork);
  }
}

// Realized rows, eligible columns, arena and row offsets of a level's large
// fronts (read by the host to set up their APTP sweep).
__global__ void k_large_sizes(DevFactor X, const int *__restrict__ large, int nlarge, int64_t *__restrict__ out) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nlarge) return;
  const int s = large[q];
  out[4 * q] = X.sn_f[s];
  out[4 * q + 1] = X.sn_ne[s];
  out[4 * q + 2] = X.sn_off[s];
  out[4 * q + 3] = X.sn_roff[s];
}

// The threshold kernel's state of the APTP fronts after their sweep: it
// continues from the APTP pivots on the columns the sweep failed (blocked,
// or unblocked when fewer than blocked_min_front rows remain:
// multifrontal_serial.cpp:810-814, ldlt_kernel.cpp:977), its Schur update
// from those pivots on; the sweep's counts carried, and the position map
// (inv, the inverse of loc, which the sweep permuted) rebuilt. One block per
// front. An aborted factorization's fronts are closed (a flag set after the
// host looked, ahead of the sweep: k_large_init may have left loc unset).
__global__ void k_aptp_to_tpp(const aptp::Front *__restrict__ fr, const aptp::State *__restrict__ st,
                              const int *__restrict__ qpos, DevFactor X, int bmf) {
  const int i = blockIdx.x;
  if (block_aborted(X)) {
    if (threadIdx.x == 0) X.tpp[qpos[i]].phase = 2;
    return;
  }
  const aptp::Front F = fr[i];
  int *inv = F.loc + X.rows_cap;
  for (int t = threadIdx.x; t < F.f; t += blockDim.x) inv[F.loc[t]] = t;
  if (threadIdx.x != 0) return;
  const aptp::State &A = st[i];
  TppState &T = X.tpp[qpos[i]];
  T.k = A.num_elim;
  T.live = F.ne;
  T.k_paired = -1;
  T.post = 0;
  T.st = A.st;
  T.pad[3] = A.num_elim;
  T.mixed = 0;
  T.se = 1 << 30;
  T.phase = (A.num_elim >= F.ne) ? 2 : (F.f - A.num_elim < bmf ? 3 : 0);
}

// One blocked-TPP step (tpp_step_blk) of each large front of a level; a
// front is taken by a team of C CTAs launched as one thread-block cluster
// (blockIdx.x / C = the front), the pivot decisions taken by every CTA of
// the team alike and the swaps and panel eliminations split over it.
template <int NT, int C>
__global__ void __launch_bounds__(NT) k_large_panel(DevPlan P, DevFactor X, const int *__restrict__ large,
                                                    PivotParams prm, int iter) {
  __shared__ TeamShared sh;
  __shared__ PairScratch s_pair;
  const int q = blockIdx.x / C;
  const bool lead = team_rank<C>() == 0 && threadIdx.x == 0;
  const int s = large[q];
  TppState S = X.tpp[q];
  if (S.phase == 2) {
    if (lead) X.tpp[q].pad[0] = 0;
    return;
  }
  prm.eff_small = __longlong_as_double((long long)X.counters[kCEffSmall]);
  FrontRef v = large_view(P, X, s);
  v.pair = &s_pair;
  if (threadIdx.x == 0) {
    sh.st = S.st;
    sh.tr_seq = 0;
  }
  __syncthreads();
  // every CTA has read the state before the leader may write it back
  if constexpr (C > 1) team_sync<C>();
  const bool more = tpp_step_blk<NT, C>(v, prm, sh, S);
  __syncthreads();
  if (lead) {
    S.st = sh.st;
    S.pad[0] = more ? 1 : 0;
    X.tpp[q] = S;
    if (more) {
      atomicMax(X.counters + kCActive, (unsigned long long)(iter + 1));
      // algorithmic flops of the deferred update asked for (2 per FMA)
      // and its bytes (each element read and written once)
      const long long m = S.g_e - S.g_c0, h = v.f - S.g_c0;
      if (m > 0 && S.g_p1 > S.g_p0) {
        const double elems = (double)(m * h - m * (m - 1) / 2);
        atomicAdd(reinterpret_cast<double *>(X.counters + kCGemmFlops), 2.0 * (double)(S.g_p1 - S.g_p0) * elems);
        atomicAdd(reinterpret_cast<double *>(X.counters + kCDeferBytes), 16.0 * elems);
        atomicAdd(X.counters + kCDeferUpd, 1ull);
        if (S.g_p1 - S.g_p0 <= 2) atomicAdd(X.counters + kCDeferSmall, 1ull);
      }
    }
  }
}

// pref[q + 1] = counts of items 0..q of a launch's fronts (pref[0] = 0), one
// front a thread: count(q) by threads q < cnt <= NT, a block scan; ends at a
// barrier. (One thread adding them up waited for each front's loads in turn:
// 100 us and more a launch on a level of a few hundred fronts.)
template <int NT, typename Count>
__device__ __forceinline__ void front_prefix(int cnt, int *pref, Count count) {
  __shared__ int wsum[NT / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __syncthreads();  // the chunk before is done with pref
  int v = tid < cnt ? count(tid) : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  if (lane == 31) wsum[warp] = v;
  __syncthreads();
  int base = 0;
  for (int w = 0; w < warp; ++w) base += wsum[w];
  if (tid < cnt) pref[tid + 1] = base + v;
  if (tid == 0) pref[0] = 0;
  __syncthreads();
}
constexpr int kFrontChunk = 256;  // fronts a chunk (a thread each)

// Work items of a level's tiled GEMMs: each large front contributes tiles of
// kGT x kGT over a lower-trapezoidal region [r0, f) x [r0, c1) with tile
// (ti, tj) needed when ti >= tj.
constexpr int kGT = 64;

__device__ __forceinline__ int trap_tiles(int rows, int cols) {  // rows >= cols
  const int rt = (rows + kGT - 1) / kGT, ct = (cols + kGT - 1) / kGT;
  return ct * rt - ct * (ct - 1) / 2;
}

__device__ __forceinline__ void trap_tile(int w, int rows, int cols, int &ti, int &tj) {
  const int rt = (rows + kGT - 1) / kGT;
  tj = 0;
  while (w >= rt - tj) {
    w -= rt - tj;
    ++tj;
  }
  ti = tj + w;
}

// (L D)(j, c) of a front in global memory (fill_ld_column).
__device__ __forceinline__ double ld_entry_g(const double *F, size_t sf, const int8_t *tags, int c, int j) {
  const double *Lc = F + (size_t)c * sf;
  const int8_t tag = tags[c];
  if (tag == 1) return __dmul_rn(Lc[j], Lc[c]);
  if (tag == 2) return __dadd_rn(__dmul_rn(Lc[j], Lc[c]), __dmul_rn(Lc[sf + j], Lc[c + 1]));
  if (tag == -1) {
    const double *L0 = Lc - sf;
    return __dadd_rn(__dmul_rn(L0[j], L0[c]), __dmul_rn(Lc[j], Lc[c]));
  }
  return 0.0;
}

// One 128 x 64 tile of C -= A B^T (lower part: i >= j, i < rmax, j < cmax)
// over K = kk pivots in order: A(i, p) = F(i, a0 + p); B(j, p) = W(j, p)
// (deferred update) or (L D)(j, a0 + p) (Schur update). 8 warps of 32 x 32
// entries each, K in chunks of 16 staged in shared memory with the next chunk
// prefetched in registers. Every entry takes one fused multiply-add per pivot
// in pivot order, a zero B(j, p) skipped, as the reference's GEMM loops do.
//
// The multiply-adds are FP64 matrix instructions (mma.m8n8k4): on this GPU
// they round as a chain of fused multiply-adds over k in ascending order
// (tests/test_front_classes.py checks it against such chains), so the result
// is the scalar loop's bit for bit; they take one operand load per 8
// multiply-adds in place of 3 (the scalar loop, bound by its shared-memory
// reads and by waiting for a chunk's loads before the one before it was used,
// ran at 12 TFLOP/s of the 33 the FP64 units give). A skipped update and a
// product with zero agree unless the sum is -0 or A is not finite: a warp that
// meets either in a chunk with a zero B entry takes that chunk in scalar steps
// (a sum that underflows to -0 inside the chunk may keep the other sign of
// zero). A is negated as it is read; the padding of a last chunk is -0 x 0,
// which leaves every sum as it is.
constexpr int kTM = 128, kTN = 64, kTK = 16;
constexpr int kTAS = kTM + 4, kTBS = kTN + 4;  // row strides: the fragments' reads hit distinct banks

struct TileSmem {
  double A[2][kTK][kTAS];
  double B[2][kTK][kTBS];
};

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// KIND 0: B = W; 1: B = (L D) with the pivots' tags; 2: B = L D, every pivot
// 1 x 1 (SPD).
template <int KIND>
__device__ __forceinline__ void tile_update(double *F, size_t sf, const double *W, int wld, const int8_t *tags,
                                            int i0, int j0, int rmax, int cmax, int a0, int kk, TileSmem &sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;  // fragment coordinates
  const int wr = 32 * (warp & 3), wc = 32 * (warp >> 2);
  // fragment (mi, ni): rows wr + 8 mi + g, columns wc + 8 ni + 2 t4 + e
  double c[4][4][2];
#pragma unroll
  for (int mi = 0; mi < 4; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = i0 + wr + 8 * mi + g, j = j0 + wc + 8 * ni + 2 * t4 + e;
        c[mi][ni][e] = (i < rmax && j < cmax && i >= j) ? F[(size_t)j * sf + i] : 0.0;
      }
  // (a warp wholly above the diagonal or past the edge has nothing to do)
  const bool idle = i0 + wr + 31 < j0 + wc || i0 + wr >= rmax || j0 + wc >= cmax;
  double pb[4], pd[4];
  // chunk k0: A copied asynchronously (zero past its edges), B's factors into
  // registers; nothing here waits for a load
  auto fetch = [&](int k0, int buf) {
    const int kc = min(kTK, kk - k0);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int p = (threadIdx.x >> 7) + 2 * u, r = threadIdx.x & 127;
      const bool in = p < kc && i0 + r < rmax;
      const double *src = in ? F + (size_t)(a0 + k0 + p) * sf + i0 + r : F;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(&sm.A[buf][p][r]);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(in ? 8 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int p = (threadIdx.x >> 6) + 4 * u, j = j0 + (int)(threadIdx.x & 63), c = a0 + k0 + p;
      const bool in = p < kc && j < cmax;
      if (KIND == 0) pb[u] = in ? W[(size_t)(k0 + p) * wld + j] : 0.0;
      else if (KIND == 1) pb[u] = in ? ld_entry_g(F, sf, tags, c, j) : 0.0;
      else {
        pb[u] = in ? F[(size_t)c * sf + j] : 0.0;
        pd[u] = in ? F[(size_t)c * sf + c] : 0.0;
      }
    }
  };
  // B of the fetched chunk into buffer buf; whether a real one is zero (the
  // padding's zeros only reach entries that are not stored)
  auto stash = [&](int k0, int buf) {
    const int kc = min(kTK, kk - k0);
    int zb = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int p = (threadIdx.x >> 6) + 4 * u, r = threadIdx.x & 63;
      const double b = KIND == 2 ? __dmul_rn(pb[u], pd[u]) : pb[u];
      sm.B[buf][p][r] = b;
      zb |= (b == 0.0 && p < kc && j0 + r < cmax) ? 1 : 0;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    return zb;
  };
  int buf = 0;
  fetch(0, 0);
  int anyz = __syncthreads_or(stash(0, 0));
  for (int k0 = 0; k0 < kk; k0 += kTK) {
    const int kc = min(kTK, kk - k0);
    if (k0 + kTK < kk) fetch(k0 + kTK, buf ^ 1);
    bool scalar = false;
    if (anyz && !idle) {
      // a skipped update matters where the sum is -0 or A is not finite
#pragma unroll
      for (int mi = 0; mi < 4; ++mi) {
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            scalar = scalar || __double_as_longlong(c[mi][ni][e]) == (long long)0x8000000000000000ull;
#pragma unroll
        for (int p4 = 0; p4 < kTK; p4 += 4) scalar = scalar || !isfinite(sm.A[buf][p4 + t4][wr + 8 * mi + g]);
      }
      scalar = __any_sync(0xffffffffu, scalar);
    }
    if (idle) {
    } else if (!scalar) {
#pragma unroll
      for (int p4 = 0; p4 < kTK; p4 += 4) {
        double av[4], bv[4];
#pragma unroll
        for (int mi = 0; mi < 4; ++mi) av[mi] = -sm.A[buf][p4 + t4][wr + 8 * mi + g];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) bv[ni] = sm.B[buf][p4 + t4][wc + 8 * ni + g];
#pragma unroll
        for (int mi = 0; mi < 4; ++mi)
#pragma unroll
          for (int ni = 0; ni < 4; ++ni) dmma884(c[mi][ni], av[mi], bv[ni]);
      }
    } else {
      for (int p = 0; p < kc; ++p) {
        double av[4];
#pragma unroll
        for (int mi = 0; mi < 4; ++mi) av[mi] = -sm.A[buf][p][wr + 8 * mi + g];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const double bv = sm.B[buf][p][wc + 8 * ni + 2 * t4 + e];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi) {
              const double x = fma(av[mi], bv, c[mi][ni][e]);
              c[mi][ni][e] = bv != 0.0 ? x : c[mi][ni][e];
            }
          }
      }
    }
    if (k0 + kTK < kk) {
      anyz = __syncthreads_or(stash(k0 + kTK, buf ^ 1));
      buf ^= 1;
    }
  }
#pragma unroll
  for (int mi = 0; mi < 4; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int i = i0 + wr + 8 * mi + g, j = j0 + wc + 8 * ni + 2 * t4 + e;
        if (i < rmax && j < cmax && i >= j) F[(size_t)j * sf + i] = c[mi][ni][e];
      }
  __syncthreads();
}

// Tiles of a lower-trapezoidal region rows [r0, f) x cols [r0, c1): tile
// (ti, tj) of kTM x kTN is needed when its last row reaches its first column.
__device__ __forceinline__ int trap_tiles2(int rows, int cols) {
  const int ct = (cols + kTN - 1) / kTN;
  int n = 0;
  for (int tj = 0; tj < ct; ++tj) {
    const int first_ti = (tj * kTN) / kTM;  // tile rows from where column tile tj starts
    n += (rows + kTM - 1) / kTM - first_ti;
  }
  return n;
}

__device__ __forceinline__ void trap_tile2(int w, int rows, int cols, int &ti, int &tj) {
  const int rt = (rows + kTM - 1) / kTM, ct = (cols + kTN - 1) / kTN;
  for (tj = 0;; ++tj) {
    const int first = (tj * kTN) / kTM;
    const int cnt = rt - first;
    if (w < cnt || tj + 1 >= ct) {
      ti = first + w;
      return;
    }
    w -= cnt;
  }
}

// Deferred updates of all large fronts with one pending (ldlt_kernel.cpp:705-761).
__global__ void __launch_bounds__(256) k_large_gemm(DevPlan P, DevFactor X, const int *__restrict__ large,
                                                    int nlarge, const TppState *__restrict__ tpp) {
  extern __shared__ __align__(16) double dsm_g[];
  TileSmem &sm = *reinterpret_cast<TileSmem *>(dsm_g);
  __shared__ int pref[kFrontChunk + 1];
  for (int chunk = 0; chunk < nlarge; chunk += kFrontChunk) {
    const int cnt = min(kFrontChunk, nlarge - chunk);
    front_prefix<256>(cnt, pref, [&](int q) {
      const TppState &S = tpp[chunk + q];
      return S.pad[0] && S.g_p1 > S.g_p0 && S.g_e > S.g_c0
                 ? trap_tiles2(X.sn_f[large[chunk + q]] - S.g_c0, S.g_e - S.g_c0) : 0;
    });
    const int total = pref[cnt];
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
      int a = 0, b = cnt;
      while (b - a > 1) {
        const int mid = (a + b) >> 1;
        if (pref[mid] <= w) a = mid;
        else b = mid;
      }
      const int q = chunk + a;
      const int s = large[q];
      const TppState S = tpp[q];
      const int f = X.sn_f[s];
      const size_t sf = (size_t)f;
      double *F = X.arena + X.sn_off[s];
      int ti, tj;
      trap_tile2(w - pref[a], f - S.g_c0, S.g_e - S.g_c0, ti, tj);
      tile_update<0>(F, sf, F + sf * sf, f, nullptr, S.g_c0 + ti * kTM, S.g_c0 + tj * kTN, f, S.g_e,
                         S.g_p0, S.g_p1 - S.g_p0, sm);
    }
  }
}

// ---------------------------------------------------------------------------
// Deferred updates, streamed (up to kDK pivots): the same update as k_large_gemm,
// F[c0:f, c0:e] -= L[c0:f, p0:p1] W[:, c0:e] on the lower trapezoid, each
// element by the same chain c = fma(-l_p, w_p, c) over p in order (w_p = 0
// skipped), so the results are bitwise those of k_large_gemm. With K = 16 or
// 32 pivots an element costs 2 K flops for 16 bytes of traffic: the update
// is bound by HBM, and the kernel is shaped for that: 64 x 64 tiles (every
// front of the launch in one list), 16 elements a thread, at most 64
// registers so that four blocks share an SM and their load, update and
// store phases overlap; the L and W slices of a tile are read once into
// shared memory. Measured on one 16,000-row front (K = 16): 4.6 TB/s,
// against 3.0 TB/s for the general tiled kernel.
constexpr int kDT = 64, kDK = 32, kDFronts = 256, kDBlocksPerSM = 4;

// Tiles of a lower trapezoid rows x cols (rows >= cols) in kDT squares:
// column tile tj holds the row tiles [tj, rt).
__device__ __forceinline__ int defer_tiles(int rows, int cols) {
  const int rt = (rows + kDT - 1) / kDT, ct = (cols + kDT - 1) / kDT;
  return ct * rt - ct * (ct - 1) / 2;
}

// Tile w of that order: the largest tj with S(tj) = tj rt - tj (tj - 1) / 2
// <= w (a root of the quadratic, then corrected by exact integer steps).
__device__ __forceinline__ void defer_tile(int w, int rows, int cols, int &ti, int &tj) {
  const long long rt = (rows + kDT - 1) / kDT, ct = (cols + kDT - 1) / kDT;
  auto S = [&](long long x) { return x * rt - x * (x - 1) / 2; };
  const double b = 2.0 * (double)rt + 1.0;
  long long t = (long long)((b - sqrt(fmax(b * b - 8.0 * (double)w, 0.0))) * 0.5);
  if (t < 0) t = 0;
  while (t > 0 && S(t) > w) --t;
  while (t + 1 < ct && S(t + 1) <= w) ++t;
  tj = (int)t;
  ti = (int)(t + (w - S(t)));
}

// mode: 0 the whole update, 1 only the next step's kDK columns [c0, c0 +
// kDK), 2 only the columns past them (look-ahead). At most kDK pivots; W
// buffer pad[1] (kDK rows each).
__global__ void __launch_bounds__(256, kDBlocksPerSM) k_large_defer(DevPlan P, DevFactor X,
                                                                    const int *__restrict__ large, int nlarge,
                                                                    const TppState *__restrict__ tpp, int mode) {
  __shared__ double Ls[kDK][kDT];  // [pivot][row of the tile]
  __shared__ double Ws[kDK][kDT];  // [pivot][column of the tile]
  __shared__ int pref[kDFronts + 1];
  __shared__ int m_f[kDFronts], m_c0[kDFronts], m_e[kDFronts], m_p0[kDFronts], m_kk[kDFronts];
  __shared__ long long m_off[kDFronts];
  __shared__ int m_wo[kDFronts];
  __shared__ int wsum[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = tid & 15, ty = tid >> 4;
  for (int chunk = 0; chunk < nlarge; chunk += kDFronts) {
    const int cnt = min(kDFronts, nlarge - chunk);
    __syncthreads();
    int nt = 0;
    if (tid < cnt) {
      const TppState &S = tpp[chunk + tid];
      const int f = S.f;
      // the columns of this launch's share of the update
      const int split = min(S.g_e, S.g_c0 + kDK);  // the next step's 32 columns
      const int cs = mode == 2 ? split : S.g_c0, ce = mode == 1 ? split : S.g_e;
      if (S.pad[0] && S.g_p1 > S.g_p0 && ce > cs) nt = defer_tiles(f - cs, ce - cs);
      m_f[tid] = f;
      m_c0[tid] = cs;
      m_e[tid] = ce;
      m_p0[tid] = S.g_p0;
      m_kk[tid] = S.g_p1 - S.g_p0;
      // (W of the panel: the second buffer for odd look-ahead panels)
      m_off[tid] = S.off;
      m_wo[tid] = S.pad[1];
    }
    // inclusive block scan of the tile counts
    int v = nt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += y;
    }
    if (lane == 31) wsum[warp] = v;
    __syncthreads();
    int base = 0;
    for (int w = 0; w < warp; ++w) base += wsum[w];
    if (tid < cnt) pref[tid + 1] = base + v;
    if (tid == 0) pref[0] = 0;
    __syncthreads();
    const int total = pref[cnt];
    // diagonal rows a two-panel SPD step staged in W: into F (block q of the
    // grid takes front q; the tiles below never touch these rows)
    if (mode != 2) {
      for (int q = blockIdx.x; q < cnt; q += gridDim.x) {
        const TppState &S = tpp[chunk + q];
        const int nd = S.pad[2];
        if (!S.pad[0] || nd <= 0) continue;
        const int s = large[chunk + q];
        const int f = X.sn_f[s];
        const size_t sf = (size_t)f;
        double *F = X.arena + X.sn_off[s];
        const double *Wd = F + sf * sf + (size_t)S.pad[1] * kDK * sf;
        for (int t = tid; t < nd * nd; t += 256) {
          const int c = t / nd, r = t % nd;
          if (r >= c) F[(size_t)(S.g_p0 + c) * sf + S.g_p0 + r] = Wd[(size_t)c * f + S.g_p0 + r];
        }
      }
    }
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
      int lo = 0, hi = cnt;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pref[mid] <= w) lo = mid;
        else hi = mid;
      }
      const int a = lo;
      int ti, tj;
      defer_tile(w - pref[a], m_f[a] - m_c0[a], m_e[a] - m_c0[a], ti, tj);
      const int f = m_f[a], e = m_e[a], kk = m_kk[a], p0 = m_p0[a];
      const size_t sf = (size_t)f;
      double *F = X.arena + m_off[a];
      const double *Wp = F + sf * sf + (size_t)m_wo[a] * kDK * sf;  // second W buffer: kDK rows on
      const int i0 = m_c0[a] + ti * kDT, j0 = m_c0[a] + tj * kDT;
      double c[4][4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int i = i0 + tx + 16 * r, j = j0 + ty + 16 * q;
          c[r][q] = (i < f && j < e && i >= j) ? F[(size_t)j * sf + i] : 0.0;
        }
      int zw = 0;  // a zero among the tile's w (a skipped update)
#pragma unroll
      for (int u = 0; u < kDK * kDT / 256; ++u) {
        const int t = tid + 256 * u, p = t >> 6, r = t & 63;
        Ls[p][r] = (p < kk && i0 + r < f) ? F[(size_t)(p0 + p) * sf + i0 + r] : 0.0;
        const bool real = p < kk && j0 + r < e;
        const double wv = real ? Wp[(size_t)p * sf + j0 + r] : 0.0;
        Ws[p][r] = wv;
        zw |= (real && wv == 0.0) ? 1 : 0;
      }
      if (!__syncthreads_or(zw)) {
        // no zero w: every update applies (the padding's zeros only reach
        // entries that are not stored)
        for (int p = 0; p < kk; ++p) {
          double av[4], bv[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) av[r] = Ls[p][tx + 16 * r];
#pragma unroll
          for (int q = 0; q < 4; ++q) bv[q] = Ws[p][ty + 16 * q];
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int r = 0; r < 4; ++r) c[r][q] = fma(-av[r], bv[q], c[r][q]);
        }
      } else {
        for (int p = 0; p < kk; ++p) {
          double av[4], bv[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) av[r] = Ls[p][tx + 16 * r];
#pragma unroll
          for (int q = 0; q < 4; ++q) bv[q] = Ws[p][ty + 16 * q];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (bv[q] != 0.0) {
#pragma unroll
              for (int r = 0; r < 4; ++r) c[r][q] = fma(-av[r], bv[q], c[r][q]);
            }
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int i = i0 + tx + 16 * r, j = j0 + ty + 16 * q;
          if (i < f && j < e && i >= j) F[(size_t)j * sf + i] = c[r][q];
        }
      __syncthreads();  // Ls / Ws are refilled by the next tile
    }
  }
}

// Schur updates of all large fronts of a level (schur_update,
// ldlt_kernel.cpp:820-933): F[e:f, e:f] -= L LD^T over pivots [0, k).
template <bool POSDEF>
__global__ void __launch_bounds__(256, 2) k_large_schur(DevPlan P, DevFactor X, const int *__restrict__ large,
                                                     int nlarge, const TppState *__restrict__ tpp) {
  extern __shared__ __align__(16) double dsm_g[];
  TileSmem &sm = *reinterpret_cast<TileSmem *>(dsm_g);
  __shared__ int pref[kFrontChunk + 1];
  for (int chunk = 0; chunk < nlarge; chunk += kFrontChunk) {
    const int cnt = min(kFrontChunk, nlarge - chunk);
    front_prefix<256>(cnt, pref, [&](int q) {
      const int s = large[chunk + q];
      // pivots [pad[3], k): an APTP front's trailing update covered its own
      const int e = X.sn_ne[s], f = X.sn_f[s], k = tpp[chunk + q].k, k0 = tpp[chunk + q].pad[3];
      // mixed fronts: the tensor-core updates covered the contribution block
      const bool fp64 = !tpp[chunk + q].mixed;
      return (f > e && k > k0 && fp64) ? trap_tiles2(f - e, f - e) : 0;
    });
    const int total = pref[cnt];
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
      int a = 0, b = cnt;
      while (b - a > 1) {
        const int mid = (a + b) >> 1;
        if (pref[mid] <= w) a = mid;
        else b = mid;
      }
      const int q = chunk + a;
      const int s = large[q];
      const int f = X.sn_f[s], e = X.sn_ne[s], k0 = tpp[q].pad[3], kk = tpp[q].k - k0;
      const size_t sf = (size_t)f;
      double *F = X.arena + X.sn_off[s];
      int ti, tj;
      trap_tile2(w - pref[a], f - e, f - e, ti, tj);
      tile_update<POSDEF ? 2 : 1>(F, sf, nullptr, 0, X.tags + X.sn_roff[s], e + ti * kTM, e + tj * kTN, f, f, k0, kk,
                                  sm);
    }
  }
}

// Bookkeeping of a factored large front (one block): zero pivots at a root,
// status flags, 2x2 off-diagonals moved to their upper slots, counts, and
// the children's row maps in pivot order. The column-parallel part of the
// store (the SPD sqrt(D) fold, zeroing) is k_large_store.
template <int NT>
__global__ void __launch_bounds__(NT) k_large_finish(DevPlan P, DevFactor X, const int *__restrict__ large,
                                                     const TppState *__restrict__ tpp, PivotParams prm) {
  if (block_aborted(X)) return;
  const int s = large[blockIdx.x];
  const TppState S = tpp[blockIdx.x];
  const FrontRef v = large_view(P, X, s);
  const int f = v.f, ne = v.ne, p = S.k;
  const size_t sf = (size_t)f;
  if (threadIdx.x == 0 && !S.mixed) {
    const double q = (double)(f - ne);
    if (q > 0 && p > S.pad[3])
      atomicAdd(reinterpret_cast<double *>(X.counters + kCGemmFlops), 2.0 * (p - S.pad[3]) * (q * (q + 1) / 2));
  }
  const bool is_root = P.sn_parent[s] < 0;
  int pstore = p;
  if (is_root && p < ne) {
    for (int c = p + threadIdx.x; c < ne; c += NT) v.tags[c] = 0;
    pstore = ne;
  }
  __syncthreads();
  if (prm.posdef) {
    if (p < ne && threadIdx.x == 0) flag_not_posdef(P, X, s);
  } else {
    bool bad = false;
    for (int c = threadIdx.x; c < pstore; c += NT) {
      double *Lc = v.F + (size_t)c * sf;
      const int8_t tag = v.tags[c];
      if (tag == 1) bad = bad || !isfinite(Lc[c]);
      else if (tag == 2) bad = bad || !isfinite(Lc[c]) || !isfinite(Lc[c + 1]) || !isfinite(Lc[sf + c + 1]);
      else if (tag == -1) Lc[c - 1] = v.F[(size_t)(c - 1) * sf + c];
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) set_flag(X.counters, kFNonfiniteD);
  }
  if (!prm.posdef) {  // (SPD rows keep their order)
    int *inv = X.ploc + X.rows_cap + X.sn_roff[s];
    for (int t = threadIdx.x; t < f; t += NT) inv[v.loc[t]] = t;
    __syncthreads();
    for (int t = P.child_ptr[s]; t < P.child_ptr[s + 1]; ++t) {
      const int c = P.child_idx[t];
      const int pc = X.sn_p[c];
      int *cmap = X.cbmap + X.sn_roff[c] + pc;
      for (int u = threadIdx.x; u < X.sn_f[c] - pc; u += NT) cmap[u] = inv[cmap[u]];
    }
  }
  if (threadIdx.x == 0) {
    X.sn_p[s] = p;
    X.sn_pstore[s] = pstore;
    X.sn_dout[s] = is_root ? 0 : ne - p;
    int *st = X.sn_stat + 4 * s;
    st[0] = S.st.pos;
    st[1] = S.st.neg;
    st[2] = S.st.zero + (is_root ? ne - p : 0);
    st[3] = S.st.two_by_two;
    X.sn_flops[s] = S.st.flops;
  }
}

// Column-parallel store of the large fronts' pivot columns
// (multifrontal_serial.cpp:903-945): SPD L = L_unit sqrt(D) with the upper
// part zero; indefinite D inline (zero pivots' columns zero, the 2x2
// blocks' lower off-diagonal slot zero, the upper part zero but for the
// slot k_large_finish filled). Work items: 32 columns of one front.
__global__ void __launch_bounds__(256) k_large_store(DevPlan P, DevFactor X, const int *__restrict__ large,
                                                     int nlarge, int posdef) {
  __shared__ int pref[kFrontChunk + 1];
  __shared__ double sdv[32];
  if (block_aborted(X)) return;
  for (int chunk = 0; chunk < nlarge; chunk += kFrontChunk) {
    const int cnt = min(kFrontChunk, nlarge - chunk);
    front_prefix<256>(cnt, pref, [&](int q) { return (X.sn_pstore[large[chunk + q]] + 31) / 32; });
    const int total = pref[cnt];
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
      int a = 0, b = cnt;
      while (b - a > 1) {
        const int mid = (a + b) >> 1;
        if (pref[mid] <= w) a = mid;
        else b = mid;
      }
      const int s = large[chunk + a];
      const int f = X.sn_f[s], pstore = X.sn_pstore[s];
      const size_t sf = (size_t)f;
      double *F = X.arena + X.sn_off[s];
      const int8_t *tags = X.tags + X.sn_roff[s];
      const int c0 = (w - pref[a]) * 32, c1 = min(c0 + 32, pstore);
      if (posdef) {
        if (threadIdx.x < c1 - c0) sdv[threadIdx.x] = sqrt(F[(size_t)(c0 + threadIdx.x) * sf + c0 + threadIdx.x]);
        __syncthreads();
        // a warp per column, eight rows a lane in flight
        const int lane = threadIdx.x & 31;
        for (int c = c0 + (threadIdx.x >> 5); c < c1; c += 8) {
          double *Lc = F + (size_t)c * sf;
          const double sq = sdv[c - c0];
          for (int i = lane; i < c; i += 32) Lc[i] = 0.0;
          for (int i0 = c + 1 + lane; i0 < f; i0 += 8 * 32) {
            double y[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) y[u] = i0 + 32 * u < f ? Lc[i0 + 32 * u] : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u)
              if (i0 + 32 * u < f) Lc[i0 + 32 * u] = __dmul_rn(y[u], sq);
          }
        }
        __syncthreads();
        if (threadIdx.x < c1 - c0) F[(size_t)(c0 + threadIdx.x) * sf + c0 + threadIdx.x] = sdv[threadIdx.x];
      } else {
        for (int c = c0; c < c1; ++c) {
          double *Lc = F + (size_t)c * sf;
          const int8_t tag = tags[c];
          for (int i = threadIdx.x; i < f; i += 256) {
            if (tag == 0) Lc[i] = 0.0;
            else if (i < c) {
              if (!(tag == -1 && i == c - 1)) Lc[i] = 0.0;
            } else if (tag == 2 && i == c + 1) {
              Lc[i] = 0.0;
            }
          }
        }
      }
      __syncthreads();
    }
    __syncthreads();
  }
}

// Two SPD panels per launch (32 pivots, then one rank-32 deferred update:
// half the launches and half the deferred traffic of one panel at a time).
// Per entry the operations and their order are the one-panel path's: the
// second panel's columns take the first panel's update as the deferred
// update would (c = fma(-l_p, w_p, c) over its pivots in order, w_p = 0
// skipped) before the second panel's eliminations, and the columns past
// both take one chain over the 32 pivots in order. Every block factors both
// diagonal blocks itself: the first with the second panel's 16 rows (their
// unscaled values w and multipliers l to shared memory) and diagonal block
// beside it, then the second. A failing pivot in the first panel ends the
// front there (as the one-panel path ends it). rpb rows a block: 128 when the
// launch has few blocks (the rows' chains are bound by one SM's FP64 rate:
// 8,000 cycles for 256 rows, 4,700 for 128). The front's sizes come with its
// state, two dependent loads fewer ahead of everything else.
template <int NB>
__global__ void __launch_bounds__(256) k_large_panel_spd2(DevPlan P, DevFactor X, const int *__restrict__ large,
                                                          const TppState *__restrict__ cur,
                                                          TppState *__restrict__ nxt, int iter, int w2, int rpb) {
  __shared__ double T[2 * NB][NB + 1], T2[NB][NB + 1];
  // (rows of multipliers and of w read two at a time)
  __shared__ __align__(16) double lm[NB][NB], lm2[NB][NB];
  __shared__ double linv[NB], linv2[NB], dv[NB], dv2[NB];
  __shared__ __align__(16) double Wr[NB][NB];  // [row of panel 2][pivot of panel 1]
  __shared__ double Lr[NB][NB];
  __shared__ int zero_sh;
  const int q = blockIdx.y;
  const TppState S = cur[q];
  const bool lead = blockIdx.x == 0;
  if (S.phase == 2) {
    if (lead && threadIdx.x == 0) {
      TppState o = S;
      o.pad[0] = 0;
      nxt[q] = o;
    }
    return;
  }
  const int f = S.f, ne = S.ne;
  const int ps = S.k, pl = min(ne, ps + NB), nbp = pl - ps;
  const int ps2 = pl, pl2 = min(ne, ps2 + NB), nbp2 = pl2 - ps2;
  const int r0 = ps + blockIdx.x * rpb;  // rows [r0, r0 + rpb), a thread each
  if (r0 >= f) return;
  const size_t sf = (size_t)f;
  double *F = X.arena + S.off;
  // W: rows [0, 16) panel 1, [16, 32) panel 2; w2 (look-ahead): two such
  // buffers alternating by step
  const int wpar = w2 ? (iter & 1) : 0;
  double *W = F + sf * sf + (size_t)wpar * 2 * NB * sf;
  const double eff_small = __longlong_as_double((long long)X.counters[kCEffSmall]);
  // Every load of F this thread needs is issued here, so that their
  // latency overlaps the two diagonal factors: none of these entries is
  // written in this launch before it is read (the panels' diagonal rows are
  // staged in W, and each row below belongs to one thread, which writes
  // panel 1's columns only after reading panel 2's).
  const int i = (int)threadIdx.x < rpb ? r0 + (int)threadIdx.x : f;
  static_assert(NB * NB == 256, "one entry of T and T2 per thread");
  const int tr = threadIdx.x / NB, tc = threadIdx.x % NB;
  const double t1v = (tr < nbp && tc <= tr) ? F[(size_t)(ps + tc) * sf + ps + tr] : 0.0;
  const double t2v = (tr < nbp2 && tc <= tr) ? F[(size_t)(ps2 + tc) * sf + ps2 + tr] : 0.0;
  const double txv = (tr < nbp2 && tc < nbp) ? F[(size_t)(ps + tc) * sf + ps2 + tr] : 0.0;
  double ra[NB], rb[NB];
#pragma unroll
  for (int c = 0; c < NB; ++c) {
    ra[c] = (i < f && c < nbp && ps + c <= i) ? F[(size_t)(ps + c) * sf + i] : 0.0;
    rb[c] = (i < f && c < nbp2 && ps2 + c <= i) ? F[(size_t)(ps2 + c) * sf + i] : 0.0;
  }
  // panel 1's diagonal block, with panel 2's rows and diagonal block
  T[tr][tc] = t1v;
  T[NB + tr][tc] = txv;
  if (threadIdx.x == 0) zero_sh = 0;
  double v2 = t2v;
  const int np1 = spd_diag_factor<NB, true>(T, lm, linv, dv, nbp, &zero_sh, nbp2, Wr, Lr, &v2);
  const bool two = np1 == NB && nbp == NB && nbp2 > 0;
  int np2 = 0;
  if (two) {
    T2[tr][tc] = (tr < nbp2 && tc <= tr) ? v2 : 0.0;
    np2 = spd_diag_factor<NB, false>(T2, lm2, linv2, dv2, nbp2, &zero_sh);
  }
  // warps whose rows all lie past the panels' diagonal blocks, with every
  // pivot taken and no zero multiplier or w: each entry takes every update
  // (no tests), the same operations in the same order
  const bool fast = zero_sh == 0 && nbp == NB && np1 == NB && (!two || (nbp2 == NB && np2 == NB)) &&
                    r0 + (int)(threadIdx.x & ~31u) >= (two ? pl2 : pl);
  if (fast && i < f) {
    double a[NB];
#pragma unroll
    for (int c = 0; c < NB; ++c) a[c] = ra[c];
#pragma unroll
    for (int k = 0; k < NB; ++k) {
      const double w = a[k];
      W[(size_t)k * f + i] = w;
#pragma unroll
      for (int j = (k + 1) / 2 * 2; j < NB; j += 2) {  // (two multipliers a load)
        const double2 l = *reinterpret_cast<const double2 *>(&lm[k][j]);
        if (j > k) a[j] = __dsub_rn(a[j], __dmul_rn(w, l.x));
        a[j + 1] = __dsub_rn(a[j + 1], __dmul_rn(w, l.y));
      }
      a[k] = __dmul_rn(w, linv[k]);
    }
#pragma unroll
    for (int c = 0; c < NB; ++c) F[(size_t)(ps + c) * sf + i] = a[c];
    if (two) {
      double b[NB];
#pragma unroll
      for (int c = 0; c < NB; ++c) {
        double v = rb[c];
#pragma unroll
        for (int p = 0; p < NB; p += 2) {
          const double2 w = *reinterpret_cast<const double2 *>(&Wr[c][p]);
          v = fma(-a[p], w.x, v);
          v = fma(-a[p + 1], w.y, v);
        }
        b[c] = v;
      }
#pragma unroll
      for (int k = 0; k < NB; ++k) {
        const double w = b[k];
        W[(size_t)(NB + k) * f + i] = w;
#pragma unroll
        for (int j = (k + 1) / 2 * 2; j < NB; j += 2) {
          const double2 l = *reinterpret_cast<const double2 *>(&lm2[k][j]);
          if (j > k) b[j] = __dsub_rn(b[j], __dmul_rn(w, l.x));
          b[j + 1] = __dsub_rn(b[j + 1], __dmul_rn(w, l.y));
        }
        b[k] = __dmul_rn(w, linv2[k]);
      }
#pragma unroll
      for (int c = 0; c < NB; ++c) F[(size_t)(ps2 + c) * sf + i] = b[c];
    }
  } else if (r0 == ps && i < (two ? pl2 : pl)) {
    // the panels' diagonal rows (block 0's first rows): the diagonal
    // factors computed their final values by the same operations -- the
    // multipliers (lm, Lr, lm2) for the pivots taken, the rest of T and T2
    // (unscaled, their pivots' updates applied) -- so they are staged from
    // shared memory
    const int r = i - ps;
    if (r < NB) {
#pragma unroll
      for (int c = 0; c < NB; ++c)
        if (c < nbp && c <= r) W[(size_t)c * f + i] = c >= np1 ? T[r][c] : c < r ? lm[c][r] : dv[c];
    } else {
      const int r2 = r - NB;
#pragma unroll
      for (int c = 0; c < NB; ++c) W[(size_t)c * f + i] = Lr[r2][c];
#pragma unroll
      for (int c = 0; c < NB; ++c)
        if (c < nbp2 && c <= r2) W[(size_t)(NB + c) * f + i] = c >= np2 ? T2[r2][c] : c < r2 ? lm2[c][r2] : dv2[c];
    }
  } else if (i < f) {
    double a[NB];
#pragma unroll
    for (int c = 0; c < NB; ++c) a[c] = ra[c];
#pragma unroll
    for (int k = 0; k < NB; ++k) {
      // (selects, not branches: the multipliers' loads issue ahead of the
      // chain; an entry skipped keeps its value exactly)
      const bool take = k < np1 && i > ps + k;
      const double w = a[k];
      if (take) W[(size_t)k * f + i] = w;
#pragma unroll
      for (int j = k + 1; j < NB; ++j) {
        const double l = lm[k][j];
        const double u = __dsub_rn(a[j], __dmul_rn(w, l));
        a[j] = (take && j < nbp && ps + j <= i && l != 0.0) ? u : a[j];
      }
      const double sk = __dmul_rn(w, linv[k]);
      a[k] = take ? sk : a[k];
    }
    // rows of the panels' diagonal blocks go to W (columns [ps, pend) at
    // W rows c): other blocks read their original values in this launch;
    // the deferred-update launch copies them into F
    const bool stage = i < (two ? pl2 : pl);
#pragma unroll
    for (int c = 0; c < NB; ++c)
      if (c < nbp && ps + c <= i) {
        if (stage) W[(size_t)c * f + i] = a[c];
        else F[(size_t)(ps + c) * sf + i] = a[c];
      }
    if (two && i >= ps2) {
      // the second panel's columns of this row: panel 1's update, then
      // panel 2's pivots
      double b[NB];
#pragma unroll
      for (int c = 0; c < NB; ++c) {
        b[c] = 0.0;
        if (c < nbp2 && ps2 + c <= i) {
          double v = rb[c];
#pragma unroll
          for (int p = 0; p < NB; ++p) {
            const double bw = Wr[c][p];
            const double u = fma(-a[p], bw, v);
            v = bw != 0.0 ? u : v;
          }
          b[c] = v;
        }
      }
#pragma unroll
      for (int k = 0; k < NB; ++k) {
        const bool take = k < np2 && i > ps2 + k;
        const double w = b[k];
        if (take) W[(size_t)(NB + k) * f + i] = w;
#pragma unroll
        for (int j = k + 1; j < NB; ++j) {
          const double l = lm2[k][j];
          const double u = __dsub_rn(b[j], __dmul_rn(w, l));
          b[j] = (take && j < nbp2 && ps2 + j <= i && l != 0.0) ? u : b[j];
        }
        const double sk = __dmul_rn(w, linv2[k]);
        b[k] = take ? sk : b[k];
      }
#pragma unroll
      for (int c = 0; c < NB; ++c)
        if (c < nbp2 && ps2 + c <= i) {
          if (stage) W[(size_t)(NB + c) * f + i] = b[c];
          else F[(size_t)(ps2 + c) * sf + i] = b[c];
        }
    }
  }
  if (lead && threadIdx.x < 32) {
    // the pivots' tags, inertia and flops, a lane each (lanes 0..15 panel
    // 1, 16..31 panel 2): the counts by ballot, the flop terms (integers,
    // exact in a double, as is every partial sum of a front's) summed by
    // shuffles -- the same totals as a pivot-by-pivot loop
    const int lane = threadIdx.x;
    const bool p1 = lane < np1, p2 = lane >= NB && lane - NB < np2;
    double dpv = 0.0, term = 0.0;
    if (p1 || p2) {
      const int col = p1 ? ps + lane : ps2 + lane - NB;
      X.tags[X.sn_roff[large[q]] + col] = 1;
      dpv = p1 ? dv[lane] : dv2[lane - NB];
      const double rem = (double)(f - (col + 1));
      term = rem + rem * (rem + 1.0);
    }
    const bool zr = (p1 || p2) && (!isfinite(dpv) || fabs(dpv) < eff_small);
    const bool po = (p1 || p2) && !zr && dpv > 0.0;
    const bool ng = (p1 || p2) && !zr && !(dpv > 0.0);
    const int nzr = __popc(__ballot_sync(0xffffffffu, zr)), npo = __popc(__ballot_sync(0xffffffffu, po)),
              nng = __popc(__ballot_sync(0xffffffffu, ng));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) term += __shfl_xor_sync(0xffffffffu, term, o);
    if (lane != 0) return;
    TppState o = S;
    o.st.zero += nzr;
    o.st.pos += npo;
    o.st.neg += nng;
    o.st.flops += term;
    const int np = np1 + np2;
    const int pend = two ? pl2 : pl;  // the deferred update starts past the panels done
    o.k = ps + np;
    o.g_p0 = ps;
    o.g_p1 = ps + np;
    o.g_c0 = pend;
    o.g_e = tpp_upd_end(S, ne);
    o.pad[0] = np > 0 ? 1 : 0;
    o.pad[1] = wpar;       // the W buffer of this step's update
    o.pad[2] = pend - ps;  // diagonal rows [ps, pend) staged in W (copied by k_large_defer)
    if (np1 < nbp || (two && np2 < nbp2) || o.k >= ne) o.phase = 2;
    nxt[q] = o;
    if (np > 0) {
      atomicMax(X.counters + kCActive, (unsigned long long)(iter + 1));
      const long long m = tpp_upd_end(S, ne) - pend, h = f - pend;
      if (m > 0) {
        const double elems = (double)(m * h - m * (m - 1) / 2);
        atomicAdd(reinterpret_cast<double *>(X.counters + kCGemmFlops), 2.0 * (double)np * elems);
        atomicAdd(reinterpret_cast<double *>(X.counters + kCDeferBytes), 16.0 * elems);
        atomicAdd(X.counters + kCDeferUpd, 1ull);
        if (np <= 2) atomicAdd(X.counters + kCDeferSmall, 1ull);
      }
    }
  }
}

// Tensor-core updates due on a level's mixed large fronts (one thread): a
// front whose outer block is used up (k reached min(se, ne)), that asked
// for a flush, or that finished with pivots pending gets a job applying
// the pivots [tc_done, k) to its columns from min(se, ne) on (the rows and
// columns no deferred update of the block touched); its next outer block
// then starts at k. Jobs, work-item and tile prefixes go to X.tc_*.
__global__ void k_tc_jobs(DevPlan P, DevFactor X, const int *__restrict__ large, int nlarge,
                          TppState *__restrict__ tpp, int nbo, int posdef, int ke) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  tc::Job *jobs = reinterpret_cast<tc::Job *>(X.tc_jobs);
  int nj = 0, tiles = 0;
  int64_t off = 0, items = 0;
  double flops = 0.0;
  X.tc_ipref[0] = 0;
  X.tc_tpref[0] = 0;
  const bool dead = abort_flagged(X);
  for (int q = 0; q < nlarge && !dead; ++q) {
    TppState &S = tpp[q];
    if (!S.mixed) continue;
    const int s = large[q];
    const int f = X.sn_f[s], ne = X.sn_ne[s], k = S.k;
    const int sep = min(S.se, ne);
    const bool cb_only = S.se >= ne;  // the contribution block only (indefinite fronts)
    const bool due = cb_only ? (k - S.tc_done >= nbo) : (k >= sep);
    if (S.tc_done < k && (S.flush || due || S.phase == 2)) {
      const int n = f - sep, kc = k - S.tc_done;
      if (n > 0) {
        double *F = X.arena + X.sn_off[s];
        tc::Job J;
        J.C = F;
        J.Ls = F + (int64_t)S.tc_done * f;
        J.Ws = nullptr;
        J.tags = posdef ? nullptr : X.tags + X.sn_roff[s];
        J.ld = J.ldl = J.ldw = f;
        J.r0 = J.lr0 = J.wr0 = sep;
        J.n = n;
        J.k0 = S.tc_done;
        J.kc = kc;
        J.ntr = (n + tc::kBM - 1) / tc::kBM;
        J.nkb = (kc + ke - 1) / ke;
        J.tiles = J.ntr * (J.ntr + 1) / 2;
        J.img = off;
        off += tc::image_bytes(J.ntr, J.nkb);
        items += (int64_t)J.ntr * tc::kBM * 8 * J.nkb;
        tiles += J.tiles;
        jobs[nj++] = J;
        X.tc_ipref[nj] = items;
        X.tc_tpref[nj] = tiles;
        flops += 2.0 * kc * ((double)n * (n + 1) / 2);
      }
      S.tc_done = k;
      if (!cb_only) S.se = k + nbo;
    }
    S.flush = 0;
  }
  if (off > X.tc_img_cap) {
    set_flag(X.counters, kFTcCap);
    nj = 0;
  }
  *X.tc_njobs = nj;
  if (flops > 0.0) atomicAdd(reinterpret_cast<double *>(X.counters + kCTcFlops), flops);
}

// Graph replays run a fixed number of pivoting steps per level: a front
// still asking for an update at the last one did not finish (the host then
// factors without the graph).
__global__ void k_steps_check(unsigned long long *cnt, int steps) {
  if (threadIdx.x == 0 && cnt[kCActive] >= (unsigned long long)steps) set_flag(cnt, kFSteps);
}

// Totals over all fronts, in supernode order (deterministic). On the static
// layout every front has its symbolic rows; a front that has not was laid out
// by something else meanwhile, and its class's kernel may have passed it by.
struct FactorTotals {
  long long pos, neg, zero, two_by_two, delayed, entries;
  int max_front, pad;
  double flops;
};

__global__ void k_finish(DevPlan P, DevFactor X, FactorTotals *out) {
  __shared__ long long acc[6][32];
  __shared__ int mf[32];
  __shared__ double fl[32];
  long long a[6] = {0, 0, 0, 0, 0, 0};
  int mx = 0;
  double fsum = 0.0;
  for (int s = threadIdx.x; s < P.nsn; s += blockDim.x) {
    const int *st = X.sn_stat + 4 * s;
    a[0] += st[0];
    a[1] += st[1];
    a[2] += st[2];
    a[3] += st[3];
    a[4] += X.sn_dout[s];
    a[5] += (long long)X.sn_f[s] * X.sn_pstore[s];
    mx = max(mx, X.sn_f[s]);
    if (X.spd_static && X.sn_f[s] != P.sn_fsym[s]) set_flag(X.counters, kFInternal);
    fsum += X.sn_flops[s];  // integer-valued: exact in any order
  }
  for (int o = 16; o > 0; o >>= 1) {
    for (int q = 0; q < 6; ++q) a[q] += __shfl_xor_sync(0xffffffffu, a[q], o);
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    fsum += __shfl_xor_sync(0xffffffffu, fsum, o);
  }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    for (int q = 0; q < 6; ++q) acc[q][w] = a[q];
    mf[w] = mx;
    fl[w] = fsum;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    FactorTotals t{};
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
      t.pos += acc[0][i];
      t.neg += acc[1][i];
      t.zero += acc[2][i];
      t.two_by_two += acc[3][i];
      t.delayed += acc[4][i];
      t.entries += acc[5][i];
      t.max_front = max(t.max_front, mf[i]);
      t.flops += fl[i];
    }
    *out = t;
  }
}

// ---------------------------------------------------------------------------
// Solves. x (new numbering, n x nrhs) and per-front work vectors w at the
// fronts' row offsets (rows_total x nrhs).
//
// The solve kernels are launched with programmatic stream serialization: a
// kernel may start while the one before it on the stream still runs. Before
// pdl_wait() it reads only what no solve kernel writes (the factor, its row
// maps and sizes), so that its loads of L overlap the kernel before it;
// pdl_wait() returns once that kernel has completed and its writes are
// visible (at once when the launch had no such dependency), and
// pdl_trigger() lets the next kernel start its own prologue.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__global__ void k_solve_gather(const double *__restrict__ b, int ldb, int nrhs, int n,
                               const int *__restrict__ perm, const double *__restrict__ scale,
                               double *__restrict__ x) {
  pdl_wait();
  pdl_trigger();
  const int64_t tot = (int64_t)n * nrhs;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < tot;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(t / n), i = (int)(t % n);
    const int o = perm[i];
    double v = b[(int64_t)r * ldb + o];
    if (scale) v = __dmul_rn(v, scale[o]);
    x[t] = v;
  }
}

__global__ void k_solve_scatter(double *__restrict__ b, int ldb, int nrhs, int n,
                                const int *__restrict__ perm, const double *__restrict__ scale,
                                const double *__restrict__ x) {
  pdl_wait();
  pdl_trigger();
  const int64_t tot = (int64_t)n * nrhs;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < tot;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(t / n), i = (int)(t % n);
    const int o = perm[i];
    double v = x[t];
    if (scale) v = __dmul_rn(v, scale[o]);
    b[(int64_t)r * ldb + o] = v;
  }
}

// Solves by level. Each front's work vector w (length f, at the front's row
// offset) holds its pivot rows' values and, in the forward sweep, its update
// vector for the parent (rows p..f); x (new numbering) holds the pivot
// results. Large fronts (symbolic rows >= kLargeMin, SPD kLargeMinSpd) take the
// multi-block kernels below; the others' sweeps are in smfg_solve.cuh.

// The 32 x 32 lower block L[jb:jb+nb, jb:jb+nb) copied to shared memory
// asynchronously (8-byte cp.async, zero fill
// outside the lower triangle); the caller waits with cp_async_wait_all()
// and a barrier before reading Ls.
template <int NT>
__device__ __forceinline__ void load_tri32_async(const double *L, size_t sf, int jb, int nb, double (*Ls)[33]) {
  for (int t = threadIdx.x; t < 1024; t += NT) {
    const int r = t & 31, c = t >> 5;
    const bool in = r < nb && c < nb && c <= r;
    const double *src = in ? L + (size_t)(jb + c) * sf + jb + r : L;
    const unsigned dst = (unsigned)__cvta_generic_to_shared(&Ls[r][c]);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(in ? 8 : 0) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// w[jb:jb+nb) <- L11^-1 w (unit, or non-unit for SPD): lane = row.
// (the lane's row of the triangle in registers and the SPD diagonal's
// reciprocal taken ahead: a step of the chain is a shuffle and an fma)
__device__ __forceinline__ void tri_fwd_warp(double *w, int jb, int nb, int posdef, const double (*Ls)[33]) {
  const int lane = threadIdx.x & 31;
  double lrow[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) lrow[j] = (j < lane && lane < nb) ? Ls[lane][j] : 0.0;
  const double rdiag = (posdef && lane < nb) ? 1.0 / Ls[lane][lane] : 1.0;
  double wi = (lane < nb) ? w[jb + lane] : 0.0;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    if (j < nb) {
      // (selects: no divergent branch in the chain; the values as the
      // branches would leave them)
      const double sc = wi * rdiag;
      wi = lane == j ? sc : wi;
      const double wj = __shfl_sync(0xffffffffu, wi, j);
      const double u = fma(-lrow[j], wj, wi);
      wi = lrow[j] != 0.0 ? u : wi;
    }
  }
  if (lane < nb) w[jb + lane] = wi;
}

// v[jb:jb+nb) <- L11^-T v: lane = row.
__device__ __forceinline__ void tri_bwd_warp(double *v, int jb, int nb, int posdef, const double (*Ls)[33]) {
  const int lane = threadIdx.x & 31;
  double lcol[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) lcol[j] = (j > lane && j < nb) ? Ls[j][lane] : 0.0;
  const double rdiag = (posdef && lane < nb) ? 1.0 / Ls[lane][lane] : 1.0;
  double vi = (lane < nb) ? v[jb + lane] : 0.0;
#pragma unroll
  for (int j = 31; j >= 0; --j) {
    if (j < nb) {
      const double sc = vi * rdiag;
      vi = lane == j ? sc : vi;
      const double xj = __shfl_sync(0xffffffffu, vi, j);
      const double u = fma(-lcol[j], xj, vi);
      vi = lcol[j] != 0.0 ? u : vi;
    }
  }
  if (lane < nb) v[jb + lane] = vi;
}

// D^-1 of the 2x2 pivot [d00 d10; d10 d11] applied to (r0, r1) by the scaled
// Cramer rule (solve_diag.cpp:49-123); zero for a singular block.
__device__ __forceinline__ void dinv2_apply(double d00, double d10, double d11, double r0, double r1, double &z0,
                                            double &z1) {
  const double s2 = max3_ref(fabs(d00), fabs(d10), fabs(d11));
  z0 = 0.0;
  z1 = 0.0;
  if (isfinite(s2) && s2 != 0.0) {
    const double a = d00 / s2, bb = d10 / s2, cc = d11 / s2;
    const double det = __dsub_rn(__dmul_rn(a, cc), __dmul_rn(bb, bb));
    if (isfinite(det) && det != 0.0) {
      if (!isfinite(r0) || !isfinite(r1)) {
        z0 = r0;
        z1 = r1;
      } else {
        const double rs = fmax(fabs(r0), fabs(r1));
        if (rs != 0.0) {
          const double q0 = r0 / rs, q1 = r1 / rs;
          const double u0 = __dsub_rn(__dmul_rn(cc, q0), __dmul_rn(bb, q1)) / det;
          const double u1 = __dadd_rn(__dmul_rn(-bb, q0), __dmul_rn(a, q1)) / det;
          const double ratio = rs / s2;
          z0 = __dmul_rn(u0, ratio);
          z1 = __dmul_rn(u1, ratio);
        }
      }
    }
  }
}

// t[0:p) = L21^T x_ext of the level's large fronts, stored at the front's
// work vector positions [0, p): a work item is kL21Cols columns of one front
// for every right-hand side (up to R), L read once for all of them. x_ext is
// gathered into shared memory a tile of rows at a time, once for all the
// item's columns; a warp takes kL21Cols / 8 columns, lane = row. Each
// column's sum runs over its rows as a warp per column would take them (lane
// l: rows p + l + 32m in turn), then a shuffle tree.
constexpr int kL21Cols = 16;
template <int R>
__global__ void __launch_bounds__(256) k_bwd_l21(DevPlan P, DevFactor X, const int *__restrict__ large,
                                                 int nlarge, const double *x, double *wk,
                                                 int64_t rows_total, int nrhs) {
  constexpr int CW = kL21Cols / 8;  // columns a warp
  constexpr int TILE = R == 1 ? 1024 : 512;
  __shared__ int pref[kFrontChunk + 1];
  __shared__ double xs[R][TILE];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  pdl_wait();
  pdl_trigger();
  for (int chunk = 0; chunk < nlarge; chunk += kFrontChunk) {
    const int cnt = min(kFrontChunk, nlarge - chunk);
    front_prefix<256>(cnt, pref, [&](int q) { return (X.sn_pstore[large[chunk + q]] + kL21Cols - 1) / kL21Cols; });
    const int total = pref[cnt];
    for (int wi = blockIdx.x; wi < total; wi += gridDim.x) {
      int a = 0, b = cnt;
      while (b - a > 1) {
        const int mid = (a + b) >> 1;
        if (pref[mid] <= wi) a = mid;
        else b = mid;
      }
      const int s = large[chunk + a];
      const int f = X.sn_f[s], p = X.sn_pstore[s];
      const int jw = (wi - pref[a]) * kL21Cols + warp * CW;
      const int *rows = X.rows + X.sn_roff[s] + p;
      const double *L = X.arena + X.sn_off[s] + p;
      double acc[CW][R];
#pragma unroll
      for (int c = 0; c < CW; ++c)
#pragma unroll
        for (int r = 0; r < R; ++r) acc[c][r] = 0.0;
      for (int t0 = 0; t0 < f - p; t0 += TILE) {
        const int tn = min(TILE, f - p - t0);
        __syncthreads();  // the tile before read
        for (int i = threadIdx.x; i < tn; i += 256) {
          const int ri = rows[t0 + i];
#pragma unroll
          for (int r = 0; r < R; ++r) xs[r][i] = r < nrhs ? x[(int64_t)r * P.n + ri] : 0.0;
        }
        __syncthreads();
#pragma unroll(R == 1 ? 8 : 2)
        for (int i = lane; i < tn; i += 32) {
          double l[CW];
#pragma unroll
          for (int c = 0; c < CW; ++c) l[c] = (jw + c < p) ? L[(size_t)(jw + c) * f + t0 + i] : 0.0;
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const double xv = xs[r][i];
#pragma unroll
            for (int c = 0; c < CW; ++c) acc[c][r] = fma(l[c], xv, acc[c][r]);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < CW; ++c)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          double v = acc[c][r];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          if (lane == 0 && r < nrhs && jw + c < p) wk[(int64_t)r * rows_total + X.sn_roff[s] + jw + c] = v;
        }
    }
  }
}

// Large fronts' L11 solves in blocks of kSB columns: one block of threads
// per front solves the block's triangle (32-column steps), then all blocks
// of the GPU update the rows below it (forward) or the dot products of the
// next block's columns with the solved rows (backward). The loops are
// latency-bound (each front's block waits for the one before it), so every
// thread keeps its loads of L in flight together: a warp takes 32 rows of
// one 32-column strip (32 loads a lane), and partial sums over strips or
// row ranges meet in shared memory in a fixed order (deterministic).
constexpr int kSB = 256;
constexpr int kTriNT = 256;  // threads of the triangle kernels

// The 256-column blocks' strips of L staged in shared memory: strip k (32
// columns, the block's rows from the strip's first on) at
// buf[k % kRing][column][row - j0], copied with cp.async ahead of its use.
// Rows are padded to kSBP doubles, so that lanes reading one row across a
// strip's 32 columns hit distinct banks.
constexpr int kSBP = kSB + 1;
constexpr int kRing = 3;
// Right-hand sides of one block of threads in the block solves: their warps run
// the triangle chains, the others the rest of the block a strip behind. More
// right-hand sides take more blocks.
constexpr int kPipeRhs = 4;
struct TriSmem {
  double buf[kRing][32][kSBP];
  double w[kPipeRhs][kSB];  // the block's values, per right-hand side
};

// Inverses of the SPD large fronts' 32 x 32 diagonal blocks of L (after
// the store: L = L_unit sqrt(D)), for the triangle solves: a warp per
// block, lane c forms column c of the inverse by forward substitution
// (x_c = 1 / l_cc, x_i = -(sum_{c <= k < i} l_ik x_k) / l_ii, the sum in k
// order), the result written column-major through shared memory.
constexpr int kInvWarps = 8;
constexpr int kInvSmem = kInvWarps * 32 * 33 * (int)sizeof(double);
__global__ void __launch_bounds__(32 * kInvWarps) k_tri_invert(DevFactor X) {
  extern __shared__ __align__(16) unsigned char inv_smem[];
  double(*S)[33] = reinterpret_cast<double(*)[33]>(inv_smem) + (threadIdx.x >> 5) * 32;
  if (block_aborted(X)) return;
  const int lane = threadIdx.x & 31;
  const int item = blockIdx.x * kInvWarps + (threadIdx.x >> 5);
  if (item >= X.inv_nitems) return;
  const int s = X.inv_items[2 * item], blk = X.inv_items[2 * item + 1];
  const int f = X.sn_f[s], p = X.sn_pstore[s];
  const int jb = 32 * blk, nb = min(32, p - jb);
  double *out = X.tri_inv + X.sn_ioff[s] + (int64_t)blk * 1024;
  const double *L = X.arena + X.sn_off[s];
  // S[i][k] = l_ik (rows of the block, lower part)
  for (int k = 0; k < 32; ++k) S[lane][k] = (k < nb && lane < nb && lane >= k) ? L[(size_t)(jb + k) * f + jb + lane] : 0.0;
  __syncwarp();
  double x[32];
  const int c = lane;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < i; ++k) acc = fma(S[i][k], x[k], acc);
    const double rd = (i < nb) ? 1.0 / S[i][i] : 0.0;
    x[i] = (i < nb && c < nb && i >= c) ? ((i == c) ? rd : -acc * rd) : 0.0;
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 32; ++i) S[c][i] = x[i];  // S[c][i] = (L^-1)_ic
  __syncwarp();
  for (int k = 0; k < 32; ++k) out[k * 32 + lane] = S[k][lane];
}

// Strip [jb, jb + nb) of the block [j0, j1) (its rows [jb, j1)) into dst by
// threads [t0, t0 + nt): a warp per column (coalesced rows), one cp.async
// group.
__device__ __forceinline__ void tri_strip_async(const double *L, size_t sf, int j0, int j1, int jb, int nb,
                                                double (*dst)[kSBP], int t0 = 0, int nt = kTriNT,
                                                const double *inv = nullptr) {
  const int rows = j1 - jb;
  const int lane = threadIdx.x & 31;
  for (int u = ((int)threadIdx.x - t0) >> 5; u < nb; u += nt / 32) {
    const double *src = L + (size_t)(jb + u) * sf + jb;
    const unsigned d = (unsigned)__cvta_generic_to_shared(&dst[u][jb - j0]);
    for (int rr = lane; rr < rows; rr += 32) {
      // the diagonal block's rows from its inverse (inv: the front's
      // blocks; jb is a multiple of 32), when there is one
      const double *sp = (inv && rr < 32) ? inv + (size_t)(jb >> 5) * 1024 + (size_t)u * 32 + rr : src + rr;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d + 8u * (unsigned)rr), "l"(sp) : "memory");
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// Columns [c0, c1) of the block ending at j1 (each from its strip's first
// row: the strips start at multiples of 32) into L2, 128-byte lines, with
// their strips' inverse blocks when there are any: the strips past the
// first kRing are copied to shared memory later, from L2 then.
__device__ __forceinline__ void tri_prefetch_l2(const double *L, size_t sf, int j1, int c0, int c1,
                                                const double *inv) {
  constexpr int kLines = 17;  // 128-byte lines a column of at most 256 rows can touch
  for (int e = threadIdx.x; e < (c1 - c0) * kLines; e += blockDim.x) {
    const int c = c0 + e / kLines, q = e % kLines, jb = c & ~31;
    if (jb + 16 * q < j1) asm volatile("prefetch.global.L2 [%0];" ::"l"(L + (size_t)c * sf + jb + 16 * q));
  }
  if (inv) {
    const int b0 = c0 >> 5, b1 = (c1 + 31) >> 5;
    for (int e = threadIdx.x; e < (b1 - b0) * 64; e += blockDim.x)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(inv + (size_t)(b0 + e / 64) * 1024 + 16 * (e % 64)));
  }
}

// wait until at most `pending` (0..2) of this thread's cp.async groups are in flight
__device__ __forceinline__ void cp_async_wait_pending(int pending) {
  if (pending >= 2) asm volatile("cp.async.wait_group 2;" ::: "memory");
  else if (pending == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
  else asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// All threads of a subset of whole warps (n of them, from warp-aligned
// threads) meet at barrier `id` (1..15; 0 is __syncthreads).
__device__ __forceinline__ void warps_sync(int id, int n) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// Strips of a forward block: strip k covers [j0 + 32k, ...).
__device__ __forceinline__ void fwd_strip(int j0, int j1, int k, int &jb, int &nb) {
  jb = j0 + 32 * k;
  nb = min(32, j1 - jb);
}
// Strips of a backward block, numbered from the last.
__device__ __forceinline__ void bwd_strip(int j0, int j1, int k, int &jb, int &nb) {
  const int nstrip = (j1 - j0 + 31) / 32;
  jb = j0 + 32 * (nstrip - 1 - k);
  nb = min(32, j1 - jb);
}

// Block [j0, j1) of a large front: its first kRing strips of L issued to
// shared memory (all threads; one cp.async group each).
__device__ __forceinline__ void fwd_block_issue(const double *L, size_t sf, int j0, int j1, TriSmem &sm,
                                                const double *inv) {
  const int nstrip = (j1 - j0 + 31) / 32;
  for (int k = 0; k < min(kRing, nstrip); ++k) {
    int jb, nb;
    fwd_strip(j0, j1, k, jb, nb);
    tri_strip_async(L, sf, j0, j1, jb, nb, sm.buf[k], 0, kTriNT, inv);
  }
}
__device__ __forceinline__ void bwd_block_issue(const double *L, size_t sf, int j0, int j1, TriSmem &sm,
                                                const double *inv) {
  const int nstrip = (j1 - j0 + 31) / 32;
  for (int k = 0; k < min(kRing, nstrip); ++k) {
    int jb, nb;
    bwd_strip(j0, j1, k, jb, nb);
    tri_strip_async(L, sf, j0, j1, jb, nb, sm.buf[k], 0, kTriNT, inv);
  }
}

// The forward 32 x 32 triangle of strip [jb, jb + nb) for one right-hand
// side (a warp; lane = row jb + lane), `pre` (the product of the strip
// before, from the look-ahead) subtracted first: w[jb + lane] <- its solved
// value, also returned. The row of the triangle is in registers and the SPD
// diagonal's reciprocal taken ahead, so a step of the chain is one shuffle
// and one fused multiply-add.
__device__ __forceinline__ double fwd_chain32(const double (*Lb)[kSBP], int j0, int jb, int nb, int posdef,
                                              double *w, double pre, bool use_inv) {
  const int lane = threadIdx.x & 31;
  if (use_inv) {
    // the strip's diagonal block holds its inverse: x = L_bb^-1 (w - pre),
    // lane i's row of the inverse against the lanes' values (four partial
    // sums, no dependent chain across the lanes)
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    const double r = (lane < nb) ? w[jb - j0 + lane] - pre : 0.0;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const double g = (j <= lane && lane < nb) ? Lb[j][jb - j0 + lane] : 0.0;
      a[j & 3] = fma(g, __shfl_sync(0xffffffffu, r, j), a[j & 3]);
    }
    const double xi = (a[0] + a[1]) + (a[2] + a[3]);
    if (lane < nb) w[jb - j0 + lane] = xi;
    return xi;
  }
  double lrow[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) lrow[j] = (j < lane && lane < nb) ? Lb[j][jb - j0 + lane] : 0.0;
  const double rdiag = (posdef && lane < nb) ? 1.0 / Lb[lane][jb - j0 + lane] : 1.0;
  double wi = (lane < nb) ? w[jb - j0 + lane] - pre : 0.0;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    if (j < nb) {
      // (selects: no divergent branch in the chain; the values as the
      // branches would leave them)
      const double sc = wi * rdiag;
      wi = lane == j ? sc : wi;
      const double wj = __shfl_sync(0xffffffffu, wi, j);
      const double u = fma(-lrow[j], wj, wi);
      wi = lrow[j] != 0.0 ? u : wi;
    }
  }
  if (lane < nb) w[jb - j0 + lane] = wi;
  return wi;
}

// The backward (transposed) 32 x 32 triangle of strip [jb, jb + nb) for one
// right-hand side (lane = column jb + lane), `pre` subtracted first.
__device__ __forceinline__ double bwd_chain32(const double (*Lb)[kSBP], int j0, int jb, int nb, int posdef,
                                              double *w, double pre, bool use_inv) {
  const int lane = threadIdx.x & 31;
  if (use_inv) {
    // x = L_bb^-T (w - pre): lane i's column of the inverse
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    const double r = (lane < nb) ? w[jb - j0 + lane] - pre : 0.0;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const double g = (j >= lane && j < nb) ? Lb[lane][jb - j0 + j] : 0.0;
      a[j & 3] = fma(g, __shfl_sync(0xffffffffu, r, j), a[j & 3]);
    }
    const double xi = (a[0] + a[1]) + (a[2] + a[3]);
    if (lane < nb) w[jb - j0 + lane] = xi;
    return xi;
  }
  double lcol[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) lcol[j] = (j > lane && j < nb) ? Lb[lane][jb - j0 + j] : 0.0;
  const double rdiag = (posdef && lane < nb) ? 1.0 / Lb[lane][jb - j0 + lane] : 1.0;
  double vi = (lane < nb) ? w[jb - j0 + lane] - pre : 0.0;
#pragma unroll
  for (int j = 31; j >= 0; --j) {
    if (j < nb) {
      const double sc = vi * rdiag;
      vi = lane == j ? sc : vi;
      const double xj = __shfl_sync(0xffffffffu, vi, j);
      const double u = fma(-lcol[j], xj, vi);
      vi = lcol[j] != 0.0 ? u : vi;
    }
  }
  if (lane < nb) w[jb - j0 + lane] = vi;
  return vi;
}

// A strip's product with one row (forward) or column (backward) is summed
// in four interleaved fused multiply-add chains (term u into chain u mod 4),
// then (c0 + c1) + (c2 + c3): the same sum wherever it is formed (the
// look-ahead, the rows or columns update, either block-solve form).
__device__ __forceinline__ double sum4(const double (&a)[4]) { return (a[0] + a[1]) + (a[2] + a[3]); }

// Look-ahead products of a solved strip (values x in the lanes of the
// warp) with the next strip. Forward: rows jn + lane of the next strip over
// the columns of this one (Lb: this strip's buffer). Backward: columns jn +
// lane of the next strip over the rows jb.. of this one (Ln: the next
// strip's buffer).
__device__ __forceinline__ double fwd_ahead32(const double (*Lb)[kSBP], int j0, int j1, int jb, double x) {
  const int i = jb + 32 + (int)(threadIdx.x & 31);
  double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int u = 0; u < 32; ++u) {
    const double xu = __shfl_sync(0xffffffffu, x, u);
    if (i < j1) a[u & 3] = fma(Lb[u][i - j0], xu, a[u & 3]);
  }
  return sum4(a);
}
__device__ __forceinline__ double bwd_ahead32(const double (*Ln)[kSBP], int j0, int jb, int nb, double x) {
  const int lane = threadIdx.x & 31;
  double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int t = 0; t < 32; ++t) {
    const double xt = __shfl_sync(0xffffffffu, x, t);
    if (t < nb) a[t & 3] = fma(Ln[lane][jb + t - j0], xt, a[t & 3]);
  }
  return sum4(a);
}

// The block's rows [r0, j1) minus a strip's products, for rhs
// 0..nrhs-1; threads [t0, t0 + nt) take rows in turn.
__device__ __forceinline__ void fwd_rows_update(const double (*Lb)[kSBP], int j0, int j1, int jb, int nb, int r0,
                                                int nrhs, TriSmem &sm, int t, int nt) {
  for (int i = r0 + t; i < j1; i += nt) {
    for (int r = 0; r < nrhs; ++r) {
      double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int u = 0; u < 32; ++u)
        if (u < nb) a[u & 3] = fma(Lb[u][i - j0], sm.w[r][jb - j0 + u], a[u & 3]);
      sm.w[r][i - j0] -= sum4(a);
    }
  }
}

// Columns of a backward strip (buffer L2, columns [j2, j2 + n2)) minus their
// products with the solved rows [r0, j1): a warp per column (warps w0.. of
// nw), lanes over the rows, a shuffle tree.
__device__ __forceinline__ void bwd_cols_update(const double (*L2)[kSBP], int j0, int j1, int j2, int n2, int r0,
                                                int nrhs, TriSmem &sm, int w0, int nw) {
  const int lane = threadIdx.x & 31;
  // four of the warp's columns at a time: their chains and shuffle trees
  // interleaved (each column's sum as one column alone would form it)
  for (int u0 = w0; u0 < n2; u0 += 4 * nw) {
    for (int r = 0; r < nrhs; ++r) {
      double acc[4] = {0.0, 0.0, 0.0, 0.0};
      for (int i = r0 + lane; i < j1; i += 32) {
        const double wv = sm.w[r][i - j0];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int u = u0 + q * nw;
          if (u < n2) acc[q] = fma(L2[u][i - j0], wv, acc[q]);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
      if (lane == 0)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (u0 + q * nw < n2) sm.w[r][j2 - j0 + u0 + q * nw] -= acc[q];
    }
  }
}

// sm.w[r][0, j1 - j0) <- L_bb^-1 sm.w[r] for each right-hand side, the
// block's first kRing strips issued by fwd_block_issue. Row i of the block
// takes each strip's product in strip order: the strips up to two before
// its own from the rows update, the one just before from the chain warp's
// look-ahead. Ends at a barrier.
__device__ void fwd_block_solve(const double *L, size_t sf, int j0, int j1, int posdef, int nrhs, TriSmem &sm,
                                const double *inv) {
  const int warp = threadIdx.x >> 5;
  const int nstrip = (j1 - j0 + 31) / 32;
  // Step k: the chain warps solve strip k and form its look-ahead product
  // with strip k + 1's rows; the other warps apply strip k - 1 to the rows
  // past strip k and then stream strip k + 2 into strip k - 1's buffer.
  const int C = nrhs, nf = kTriNT - 32 * C, ft = (int)threadIdx.x - 32 * C;
  cp_async_wait_pending(min(kRing - 1, nstrip - 1));  // strip 0 landed
  __syncthreads();
  double la = 0.0;
  for (int k = 0; k <= nstrip; ++k) {
    if (warp < C) {
      if (k < nstrip) {
        int jb, nb;
        fwd_strip(j0, j1, k, jb, nb);
        const double(*Lb)[kSBP] = sm.buf[k % kRing];
        const double x = fwd_chain32(Lb, j0, jb, nb, posdef, sm.w[warp], la, inv != nullptr);
        la = (k + 1 < nstrip) ? fwd_ahead32(Lb, j0, j1, jb, x) : 0.0;
      }
    } else {
      bool issued = false;
      if (k >= 1) {
        int jm, nm;
        fwd_strip(j0, j1, k - 1, jm, nm);
        fwd_rows_update(sm.buf[(k - 1) % kRing], j0, j1, jm, nm, jm + 64, C, sm, ft, nf);
        if (k - 1 + kRing < nstrip) {
          warps_sync(1, nf);  // every reader of strip k - 1's buffer done
          int jb3, nb3;
          fwd_strip(j0, j1, k - 1 + kRing, jb3, nb3);
          tri_strip_async(L, sf, j0, j1, jb3, nb3, sm.buf[(k - 1) % kRing], 32 * C, nf, inv);
          issued = true;
        }
      }
      // strip k + 1 (issued a step ago) landed before the chains take it
      if (k + 1 < nstrip && k + 1 >= kRing) cp_async_wait_pending(issued ? 1 : 0);
    }
    // strips 1 and 2, issued by every thread at the start
    if (k == 0 && nstrip > 1) cp_async_wait_pending(nstrip > 2 ? 1 : 0);
    if (k == 1 && nstrip > 2) cp_async_wait_pending(warp >= C && k - 1 + kRing < nstrip ? 1 : 0);
    __syncthreads();
  }
}

// Forward block b of each large front (a block of threads per front and group
// of right-hand sides): w[j0:j1) <- L_bb^-1 w[j0:j1).
__global__ void __launch_bounds__(kTriNT) k_fwd_tri(DevPlan P, DevFactor X, const int *__restrict__ large,
                                                    int b, int posdef, double *x, double *wk,
                                                    int64_t rows_total, int nrhs_all, int group) {
  extern __shared__ __align__(16) unsigned char tri_smem[];
  TriSmem &sm = *reinterpret_cast<TriSmem *>(tri_smem);
  // (front, group of right-hand sides)
  const int ng = (nrhs_all + group - 1) / group, rg = (int)blockIdx.x % ng * group;
  const int nrhs = min(group, nrhs_all - rg);
  x += (int64_t)rg * P.n;
  wk += (int64_t)rg * rows_total;
  const int s = large[blockIdx.x / ng];
  const int f = X.sn_f[s], p = X.sn_pstore[s];
  const int j0 = b * kSB;
  if (j0 >= p) return;
  const int j1 = min(p, j0 + kSB);
  const int64_t roff = X.sn_roff[s];
  const int *rows = X.rows + roff;
  const double *L = X.arena + X.sn_off[s];
  const size_t sf = (size_t)f;
  // SPD: the diagonal blocks' inverses, when the factorization formed them
  const double *inv = (posdef && X.tri_inv && X.sn_ioff[s] >= 0) ? X.tri_inv + X.sn_ioff[s] : nullptr;
  fwd_block_issue(L, sf, j0, j1, sm, inv);
  tri_prefetch_l2(L, sf, j1, min(j1, j0 + 32 * kRing), j1, inv);
  pdl_wait();  // the strips of L in flight meanwhile
  pdl_trigger();
  for (int r = 0; r < nrhs; ++r)
    for (int t = threadIdx.x; t < j1 - j0; t += kTriNT) sm.w[r][t] = wk[(int64_t)r * rows_total + roff + j0 + t];
  fwd_block_solve(L, sf, j0, j1, posdef, nrhs, sm, inv);
  for (int r = 0; r < nrhs; ++r) {
    double *w = wk + (int64_t)r * rows_total + roff;
    double *xr = x + (int64_t)r * P.n;
    for (int t = threadIdx.x; t < j1 - j0; t += kTriNT) {
      w[j0 + t] = sm.w[r][t];
      xr[rows[j0 + t]] = sm.w[r][t];
    }
  }
}

// w[j1:f) -= L[j1:f, j0:j1) w[j0:j1) of each large front: a work item is 32
// rows for every right-hand side (up to R), L read once for all of them; its
// 8 warps take 32-column strips of the block, lane = row, and the strips'
// partial sums are added in strip order.
template <int R>
__global__ void __launch_bounds__(256) k_fwd_gemv(DevPlan P, DevFactor X, const int *__restrict__ large,
                                                  int nlarge, int b, double *wk, int64_t rows_total,
                                                  int nrhs) {
  __shared__ __align__(16) double ws[R][kSB];
  __shared__ double part[8][R][33];
  __shared__ int pref[kFrontChunk + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  bool waited = false;
  for (int chunk = 0; chunk < nlarge; chunk += kFrontChunk) {
    const int cnt = min(kFrontChunk, nlarge - chunk);
    front_prefix<256>(cnt, pref, [&](int q) {
      const int s = large[chunk + q];
      const int f = X.sn_f[s], p = X.sn_pstore[s], j1 = min(p, (b + 1) * kSB);
      return (b * kSB < p && f > j1) ? (f - j1 + 31) / 32 : 0;
    });
    const int total = pref[cnt];
    for (int wi = blockIdx.x; wi < total; wi += gridDim.x) {
      int a = 0, bb = cnt;
      while (bb - a > 1) {
        const int mid = (a + bb) >> 1;
        if (pref[mid] <= wi) a = mid;
        else bb = mid;
      }
      const int s = large[chunk + a];
      const int f = X.sn_f[s], p = X.sn_pstore[s];
      const int j0 = b * kSB, j1 = min(p, j0 + kSB);
      double *w = wk + X.sn_roff[s];
      const double *L = X.arena + X.sn_off[s];
      const size_t sf = (size_t)f;
      const int i = j1 + (wi - pref[a]) * 32 + lane;
      const int jb = j0 + warp * 32;
      const int nbw = (i < f && jb < j1) ? min(32, j1 - jb) : 0;
      // this lane's 32 entries of L in flight before the wait (the first
      // item: while the triangle kernel before this one still runs)
      double l[32];
      const double *li = L + (size_t)jb * sf + i;
#pragma unroll
      for (int u = 0; u < 32; ++u) l[u] = (u < nbw) ? __ldg(li + (size_t)u * sf) : 0.0;
      if (!waited) {
        pdl_wait();
        pdl_trigger();
        waited = true;
      }
      __syncthreads();
      for (int r = 0; r < R && r < nrhs; ++r)
        ws[r][threadIdx.x] = j0 + (int)threadIdx.x < j1 ? w[(int64_t)r * rows_total + j0 + threadIdx.x] : 0.0;
      __syncthreads();
      for (int r = 0; r < R && r < nrhs; ++r) {
        // (two chains: even and odd columns)
        double a0 = 0.0, a1 = 0.0;
#pragma unroll
        for (int u = 0; u < 32; u += 2) {
          const double2 y = *reinterpret_cast<const double2 *>(&ws[r][warp * 32 + u]);
          a0 = fma(l[u], y.x, a0);
          a1 = fma(l[u + 1], y.y, a1);
        }
        part[warp][r][lane] = a0 + a1;
      }
      __syncthreads();
      for (int r = warp; r < R && r < nrhs; r += 8)
        if (i < f) {
          double sum = 0.0;
#pragma unroll
          for (int g = 0; g < 8; ++g) sum += part[g][r][lane];
          w[(int64_t)r * rows_total + i] -= sum;
        }
    }
  }
  if (!waited) pdl_wait();  // (every grid waits: the next one's wait covers all before)
}

// v[j] -= sum_{i in [j1, p)} L(i, j) v[i] for the columns j of block b of
// each large front: a work item is CW columns for every right-hand side (up
// to R), their rows split over the block's threads (a thread's loads in
// flight), partial sums added in thread order.
template <int R>
__global__ void __launch_bounds__(256) k_bwd_dots(DevPlan P, DevFactor X, const int *__restrict__ large,
                                                  int nlarge, int b, double *wk, int64_t rows_total,
                                                  int nrhs) {
  constexpr int CW = R == 1 ? 1 : 2, AHEAD = R == 1 ? 8 : 2;
  __shared__ int pref[kFrontChunk + 1];
  __shared__ double red[8][CW * R];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  pdl_wait();
  pdl_trigger();
  for (int chunk = 0; chunk < nlarge; chunk += kFrontChunk) {
    const int cnt = min(kFrontChunk, nlarge - chunk);
    front_prefix<256>(cnt, pref, [&](int q) {
      const int p = X.sn_pstore[large[chunk + q]], j0 = b * kSB, j1 = min(p, j0 + kSB);
      return (j0 < p && j1 < p) ? (j1 - j0 + CW - 1) / CW : 0;
    });
    const int total = pref[cnt];
    for (int wi = blockIdx.x; wi < total; wi += gridDim.x) {
      int a = 0, bb = cnt;
      while (bb - a > 1) {
        const int mid = (a + bb) >> 1;
        if (pref[mid] <= wi) a = mid;
        else bb = mid;
      }
      const int s = large[chunk + a];
      const int f = X.sn_f[s], p = X.sn_pstore[s];
      const int j0 = b * kSB, j1 = min(p, j0 + kSB);
      const int j = j0 + (wi - pref[a]) * CW, nj = min(CW, j1 - j);
      double *v = wk + X.sn_roff[s];
      const double *Lj = X.arena + X.sn_off[s] + (size_t)j * f;
      double acc[CW][R];
#pragma unroll
      for (int c = 0; c < CW; ++c)
#pragma unroll
        for (int r = 0; r < R; ++r) acc[c][r] = 0.0;
      for (int i0 = j1 + (int)threadIdx.x; i0 < p; i0 += AHEAD * 256) {
        double l[CW][AHEAD], y[R][AHEAD];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          const int i = i0 + u * 256;
#pragma unroll
          for (int c = 0; c < CW; ++c) l[c][u] = (i < p && c < nj) ? __ldg(Lj + (size_t)c * f + i) : 0.0;
#pragma unroll
          for (int r = 0; r < R; ++r) y[r][u] = (i < p && r < nrhs) ? v[(int64_t)r * rows_total + i] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
#pragma unroll
          for (int r = 0; r < R; ++r)
#pragma unroll
            for (int c = 0; c < CW; ++c) acc[c][r] = fma(l[c][u], y[r][u], acc[c][r]);
      }
      __syncthreads();
#pragma unroll
      for (int c = 0; c < CW; ++c)
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) acc[c][r] += __shfl_xor_sync(0xffffffffu, acc[c][r], o);
          if (lane == 0) red[warp][c * R + r] = acc[c][r];
        }
      __syncthreads();
      const int c = (int)threadIdx.x / R, r = (int)threadIdx.x % R;
      if (c < nj && r < nrhs) {
        double sum = 0.0;
        for (int g = 0; g < 8; ++g) sum += red[g][c * R + r];
        v[(int64_t)r * rows_total + j + c] -= sum;
      }
    }
  }
}

// sm.w[r][0, j1 - j0) <- L_bb^-T sm.w[r] (the rows past the block already
// taken), the block's first kRing strips issued by bwd_block_issue: strips
// from the last. A column of strip m takes, before its triangle, the
// product with the solved rows of the strips up to m - 2 (one shuffle-tree
// sum) and then that with strip m - 1's rows (the chain warp's look-ahead).
// Ends at a barrier.
__device__ void bwd_block_solve(const double *L, size_t sf, int j0, int j1, int posdef, int nrhs, TriSmem &sm,
                                const double *inv) {
  const int warp = threadIdx.x >> 5;
  const int nstrip = (j1 - j0 + 31) / 32;
  // Step k: the chain warps solve strip k and form its look-ahead product
  // with strip k + 1's columns; the other warps stream strip k + 2 into
  // strip k - 1's buffer and apply the rows solved up to strip k - 1 to
  // strip k + 1's columns.
  const int C = nrhs, nf = kTriNT - 32 * C, fw = warp - C, nfw = nf / 32;
  cp_async_wait_pending(nstrip > 2 ? 1 : 0);  // strips 0 and 1 landed
  __syncthreads();
  double la = 0.0;
  for (int k = 0; k < nstrip; ++k) {
    if (warp < C) {
      int jb, nb;
      bwd_strip(j0, j1, k, jb, nb);
      const double x = bwd_chain32(sm.buf[k % kRing], j0, jb, nb, posdef, sm.w[warp], la, inv != nullptr);
      la = 0.0;
      if (k + 1 < nstrip) la = bwd_ahead32(sm.buf[(k + 1) % kRing], j0, jb, nb, x);
    } else {
      if (k >= 1 && k - 1 + kRing < nstrip) {
        // strip k - 1's buffer: its last readers (chain k - 1, look-ahead
        // k - 2, the columns update one step before) are done
        int jb3, nb3;
        bwd_strip(j0, j1, k - 1 + kRing, jb3, nb3);
        tri_strip_async(L, sf, j0, j1, jb3, nb3, sm.buf[(k - 1) % kRing], 32 * C, nf, inv);
      }
      if (k >= 1 && k + 1 < nstrip) {
        int jm, nm, j2, n2;
        bwd_strip(j0, j1, k - 1, jm, nm);
        bwd_strip(j0, j1, k + 1, j2, n2);
        bwd_cols_update(sm.buf[(k + 1) % kRing], j0, j1, j2, n2, jm, C, sm, fw, nfw);
      }
      // strip k + 2 landed before the next step's readers take it
      if (k + 2 < nstrip && k + 2 >= kRing) cp_async_wait_pending(0);
    }
    if (k == 0 && nstrip > 2) cp_async_wait_pending(0);  // strip 2, issued by every thread at the start
    __syncthreads();
  }
}

// Backward block b of each large front (a block of threads per front and group
// of right-hand sides; its rows past the block already taken by k_bwd_dots).
__global__ void __launch_bounds__(kTriNT) k_bwd_tri(DevPlan P, DevFactor X, const int *__restrict__ large,
                                                    int b, int posdef, double *x, double *wk,
                                                    int64_t rows_total, int nrhs_all, int group) {
  extern __shared__ __align__(16) unsigned char tri_smem[];
  TriSmem &sm = *reinterpret_cast<TriSmem *>(tri_smem);
  // (front, group of right-hand sides)
  const int ng = (nrhs_all + group - 1) / group, rg = (int)blockIdx.x % ng * group;
  const int nrhs = min(group, nrhs_all - rg);
  x += (int64_t)rg * P.n;
  wk += (int64_t)rg * rows_total;
  const int s = large[blockIdx.x / ng];
  const int f = X.sn_f[s], p = X.sn_pstore[s];
  const int j0 = b * kSB;
  if (j0 >= p) return;
  const int j1 = min(p, j0 + kSB);
  const int64_t roff = X.sn_roff[s];
  const int *rows = X.rows + roff;
  const double *L = X.arena + X.sn_off[s];
  const size_t sf = (size_t)f;
  const double *inv = (posdef && X.tri_inv && X.sn_ioff[s] >= 0) ? X.tri_inv + X.sn_ioff[s] : nullptr;
  bwd_block_issue(L, sf, j0, j1, sm, inv);
  {
    int jl, nl;  // the backward strips past the first kRing: columns [j0, jl)
    bwd_strip(j0, j1, min(kRing, (j1 - j0 + 31) / 32) - 1, jl, nl);
    tri_prefetch_l2(L, sf, j1, j0, jl, inv);
  }
  pdl_wait();  // the strips of L in flight meanwhile
  pdl_trigger();
  for (int r = 0; r < nrhs; ++r)
    for (int t = threadIdx.x; t < j1 - j0; t += kTriNT) sm.w[r][t] = wk[(int64_t)r * rows_total + roff + j0 + t];
  bwd_block_solve(L, sf, j0, j1, posdef, nrhs, sm, inv);
  for (int r = 0; r < nrhs; ++r) {
    double *w = wk + (int64_t)r * rows_total + roff;
    double *xr = x + (int64_t)r * P.n;
    for (int t = threadIdx.x; t < j1 - j0; t += kTriNT) {
      w[j0 + t] = sm.w[r][t];
      xr[rows[j0 + t]] = sm.w[r][t];
    }
  }
}

// ---------------------------------------------------------------------------
// Residual r = b - A x and backward errors (refinement.cpp:39-130), on the
// full symmetric pattern, eight lanes per row, compensated dot products
// (Ogita, Rump & Oishi, "Accurate sum and dot product", SIAM J. Sci.
// Comput. 26(6), 2005: TwoProduct via fma, TwoSum) in the new numbering.
__device__ __forceinline__ void two_sum(double a, double b, double &s, double &e) {
  s = a + b;
  const double bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// kResLanes lanes per row (rows hold a few entries of the symmetric
// pattern: a warp takes 32 / kResLanes rows at a time).
constexpr int kResLanes = 8;

__global__ void k_residual(DevPlan P, const double *__restrict__ vals, const double *__restrict__ x,
                           const double *__restrict__ b, double *__restrict__ r, int n,
                           unsigned long long *mx /* [0] |r|max [1] row |A| sum max [2] |x| max [3] |b| max [4] omega */) {
  constexpr int RPW = 32 / kResLanes;
  const int lane = threadIdx.x & 31, sub = lane % kResLanes, grp = lane / kResLanes;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  double m_r = 0.0, m_a = 0.0, m_x = 0.0, m_b = 0.0, m_o = 0.0;
  for (int i0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * RPW; i0 < n; i0 += warps * RPW) {
    const int i = i0 + grp;
    double s = 0.0, c = 0.0, as = 0.0, ra = 0.0;
    if (i < n) {
      for (int k = P.sptr[i] + sub; k < P.sptr[i + 1]; k += kResLanes) {
        const double a = vals[P.sidx[k]];
        const double xj = x[P.srow[k]];
        const double pr = a * xj;
        const double pe = fma(a, xj, -pr);
        double t, e;
        two_sum(s, pr, t, e);
        s = t;
        c += e + pe;
        as = fma(fabs(a), fabs(xj), as);
        ra += fabs(a);
      }
    }
    for (int o = kResLanes / 2; o > 0; o >>= 1) {  // within the row's lanes
      const double s2 = __shfl_xor_sync(0xffffffffu, s, o);
      const double c2 = __shfl_xor_sync(0xffffffffu, c, o);
      double t, e;
      two_sum(s, s2, t, e);
      s = t;
      c += c2 + e;
      as += __shfl_xor_sync(0xffffffffu, as, o);
      ra += __shfl_xor_sync(0xffffffffu, ra, o);
    }
    if (sub == 0 && i < n) {
      const double bi = b[i];
      double t, e;
      two_sum(bi, -s, t, e);
      const double res = t + (e - c);
      r[i] = res;
      m_r = fmax(m_r, fabs(res));
      m_a = fmax(m_a, ra);
      m_x = fmax(m_x, fabs(x[i]));
      m_b = fmax(m_b, fabs(bi));
      const double den = as + fabs(bi);
      const double om = den > 0.0 ? fabs(res) / den : (res == 0.0 ? 0.0 : INFINITY);
      m_o = fmax(m_o, om);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    m_r = fmax(m_r, __shfl_xor_sync(0xffffffffu, m_r, o));
    m_a = fmax(m_a, __shfl_xor_sync(0xffffffffu, m_a, o));
    m_x = fmax(m_x, __shfl_xor_sync(0xffffffffu, m_x, o));
    m_b = fmax(m_b, __shfl_xor_sync(0xffffffffu, m_b, o));
    m_o = fmax(m_o, __shfl_xor_sync(0xffffffffu, m_o, o));
  }
  if (lane == 0) {
    atomicMax(mx + 0, (unsigned long long)__double_as_longlong(m_r));
    atomicMax(mx + 1, (unsigned long long)__double_as_longlong(m_a));
    atomicMax(mx + 2, (unsigned long long)__double_as_longlong(m_x));
    atomicMax(mx + 3, (unsigned long long)__double_as_longlong(m_b));
    atomicMax(mx + 4, (unsigned long long)__double_as_longlong(m_o));
  }
}

// Up to kResLanes right-hand sides at once: the pattern and the values read
// once for all of them, x interleaved in the new numbering (xi[i * nr + q]),
// b read and r written in the original numbering (column q at q * n). Each
// column's sums take the same operations in the same order as k_residual;
// after the row's reduction, lane sub keeps the maxima of column sub.
// Latency: a lane's next kResAhead entries have their indices, then their
// values, loaded together, the next entry's x while the current one is
// summed, and the row's b and x ahead of the entries.
constexpr int kResAhead = 4;

__global__ void __launch_bounds__(256, 2)
    k_residual_rhs(DevPlan P, const double *__restrict__ vals, const double *__restrict__ xi, int nr,
                   const double *__restrict__ b, double *__restrict__ r, int n,
                   unsigned long long *mx /* 8 per column, as k_residual */) {
  constexpr int RPW = 32 / kResLanes;
  const int lane = threadIdx.x & 31, sub = lane % kResLanes, grp = lane / kResLanes;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  double m_r = 0.0, m_a = 0.0, m_x = 0.0, m_b = 0.0, m_o = 0.0;
  for (int i0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * RPW; i0 < n; i0 += warps * RPW) {
    const int i = i0 + grp;
    double s[kResLanes], c[kResLanes], as[kResLanes], ra = 0.0;
#pragma unroll
    for (int q = 0; q < kResLanes; ++q) s[q] = c[q] = as[q] = 0.0;
    int64_t ob = 0;
    double bi = 0.0, xs = 0.0;
    if (sub < nr && i < n) {
      ob = (int64_t)sub * n + P.perm[i];
      bi = b[ob];
      xs = xi[(int64_t)i * nr + sub];
    }
    if (i < n) {
      const int ke = P.sptr[i + 1];
      for (int k0 = P.sptr[i] + sub; k0 < ke; k0 += kResLanes * kResAhead) {
        // entries past the row's end read index 0 and are not summed
        int jx[kResAhead], ix[kResAhead];
#pragma unroll
        for (int u = 0; u < kResAhead; ++u) {
          const int k = k0 + u * kResLanes;
          jx[u] = k < ke ? P.srow[k] : 0;
          ix[u] = k < ke ? P.sidx[k] : 0;
        }
        double av[kResAhead], xc[kResLanes];
#pragma unroll
        for (int u = 0; u < kResAhead; ++u) av[u] = vals[ix[u]];
#pragma unroll
        for (int q = 0; q < kResLanes; ++q) xc[q] = q < nr ? xi[(int64_t)jx[0] * nr + q] : 0.0;
#pragma unroll
        for (int u = 0; u < kResAhead; ++u) {
          double xn[kResLanes];
#pragma unroll
          for (int q = 0; q < kResLanes; ++q)
            xn[q] = (u + 1 < kResAhead && q < nr) ? xi[(int64_t)jx[u + 1 < kResAhead ? u + 1 : u] * nr + q] : 0.0;
          if (k0 + u * kResLanes < ke) {
            const double a = av[u];
#pragma unroll
            for (int q = 0; q < kResLanes; ++q) {
              if (q < nr) {
                const double xv = xc[q];
                const double pr = a * xv;
                const double pe = fma(a, xv, -pr);
                double t, e;
                two_sum(s[q], pr, t, e);
                s[q] = t;
                c[q] += e + pe;
                as[q] = fma(fabs(a), fabs(xv), as[q]);
              }
            }
            ra += fabs(a);
          }
#pragma unroll
          for (int q = 0; q < kResLanes; ++q) xc[q] = xn[q];
        }
      }
    }
    for (int o = kResLanes / 2; o > 0; o >>= 1) {  // within the row's lanes
#pragma unroll
      for (int q = 0; q < kResLanes; ++q) {
        if (q < nr) {
          const double s2 = __shfl_xor_sync(0xffffffffu, s[q], o);
          const double c2 = __shfl_xor_sync(0xffffffffu, c[q], o);
          double t, e;
          two_sum(s[q], s2, t, e);
          s[q] = t;
          c[q] += c2 + e;
          as[q] += __shfl_xor_sync(0xffffffffu, as[q], o);
        }
      }
      ra += __shfl_xor_sync(0xffffffffu, ra, o);
    }
    // the butterfly leaves the compensation term rounded differently on
    // the row's lanes: every column takes the row's first lane's values,
    // the ones k_residual uses
    double S = 0.0, C = 0.0, AS = 0.0;
    const int lead = grp * kResLanes;
#pragma unroll
    for (int q = 0; q < kResLanes; ++q) {
      if (q < nr) {
        const double s0 = __shfl_sync(0xffffffffu, s[q], lead);
        const double c0 = __shfl_sync(0xffffffffu, c[q], lead);
        const double a0 = __shfl_sync(0xffffffffu, as[q], lead);
        if (q == sub) {
          S = s0;
          C = c0;
          AS = a0;
        }
      }
    }
    if (sub < nr && i < n) {
      double t, e;
      two_sum(bi, -S, t, e);
      const double res = t + (e - C);
      r[ob] = res;
      m_r = fmax(m_r, fabs(res));
      m_a = fmax(m_a, ra);
      m_x = fmax(m_x, fabs(xs));
      m_b = fmax(m_b, fabs(bi));
      const double den = AS + fabs(bi);
      const double om = den > 0.0 ? fabs(res) / den : (res == 0.0 ? 0.0 : INFINITY);
      m_o = fmax(m_o, om);
    }
  }
  for (int o = 16; o >= kResLanes; o >>= 1) {  // across the rows, per column
    m_r = fmax(m_r, __shfl_xor_sync(0xffffffffu, m_r, o));
    m_a = fmax(m_a, __shfl_xor_sync(0xffffffffu, m_a, o));
    m_x = fmax(m_x, __shfl_xor_sync(0xffffffffu, m_x, o));
    m_b = fmax(m_b, __shfl_xor_sync(0xffffffffu, m_b, o));
    m_o = fmax(m_o, __shfl_xor_sync(0xffffffffu, m_o, o));
  }
  if (grp == 0 && sub < nr) {
    unsigned long long *m = mx + 8 * sub;
    atomicMax(m + 0, (unsigned long long)__double_as_longlong(m_r));
    atomicMax(m + 1, (unsigned long long)__double_as_longlong(m_a));
    atomicMax(m + 2, (unsigned long long)__double_as_longlong(m_x));
    atomicMax(m + 3, (unsigned long long)__double_as_longlong(m_b));
    atomicMax(m + 4, (unsigned long long)__double_as_longlong(m_o));
  }
}

// xi[i * nr + q] = x[q * n + perm[i]]: nr columns interleaved in the new
// numbering, for k_residual_rhs.
__global__ void k_gather_interleave(const double *__restrict__ x, int n, int nr, const int *__restrict__ perm,
                                    double *__restrict__ xi) {
  const int64_t tot = (int64_t)n * nr;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < tot;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(t / nr), q = (int)(t % nr);
    xi[t] = x[(int64_t)q * n + perm[i]];
  }
}

__global__ void k_axpy(double *__restrict__ x, const double *__restrict__ dx, int64_t len) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < len;
       t += (int64_t)gridDim.x * blockDim.x)
    x[t] += dx[t];
}

// ---------------------------------------------------------------------------
// Krylov helpers of the FGMRES refinement (refinement.cpp:451-643): dot
// products in a fixed order (per-block partials, then one block), vector
// updates whose coefficient stays in device memory, the product with A.

constexpr int kDotBlocks = 296;

__global__ void __launch_bounds__(256) k_dot_part(const double *__restrict__ a, const double *__restrict__ b,
                                                  int64_t n, double *__restrict__ part) {
  __shared__ double red[8];
  double s = 0.0;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    s = fma(a[t], b[t], s);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    part[blockIdx.x] = t;
  }
}

__global__ void k_dot_fin(const double *__restrict__ part, int nparts, double *__restrict__ out) {
  __shared__ double red[32];
  double s = 0.0;
  for (int t = threadIdx.x; t < nparts; t += blockDim.x) s += part[t];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    *out = t;
  }
}

// y -= coef[0] * x
__global__ void k_axpy_coef(double *__restrict__ y, const double *__restrict__ x, const double *__restrict__ coef,
                            int64_t n) {
  const double c = *coef;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    y[t] = fma(-c, x[t], y[t]);
}

// y = x * alpha; y may be x (in place), so neither pointer is restrict
__global__ void k_scale(double *y, const double *x, double alpha, int64_t n) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    y[t] = x[t] * alpha;
}

// xc = x0 + sum_l y[l] Z[l]
__global__ void k_lincomb(double *__restrict__ xc, const double *__restrict__ x0, const double *__restrict__ Z,
                          const double *__restrict__ y, int k, int64_t n) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    double v = x0[t];
    for (int l = 0; l < k; ++l) v = fma(y[l], Z[(int64_t)l * n + t], v);
    xc[t] = v;
  }
}

// y = A x in the new numbering (the unscaled values), a warp per row
__global__ void k_spmv(DevPlan P, const double *__restrict__ vals, const double *__restrict__ x,
                       double *__restrict__ y, int n) {
  constexpr int RPW = 32 / kResLanes;  // rows per warp, as k_residual
  const int lane = threadIdx.x & 31, sub = lane % kResLanes, grp = lane / kResLanes;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int i0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * RPW; i0 < n; i0 += warps * RPW) {
    const int i = i0 + grp;
    double s = 0.0;
    if (i < n)
      for (int k = P.sptr[i] + sub; k < P.sptr[i + 1]; k += kResLanes) s = fma(vals[P.sidx[k]], x[P.srow[k]], s);
    for (int o = kResLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (sub == 0 && i < n) y[i] = s;
  }
}

}  // namespace smfg
