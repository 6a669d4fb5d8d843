// Small fronts (at most kFuseMax rows, below the blocked size): assembled,
// factored and stored by one block of threads, the front in shared memory
// from its zeroing to its store.
//
// Per entry the operations and their order are those of the front kernels in
// smfg_front.cuh (the reference's): the unblocked pivoting loop, whose every
// pivot updates the whole trailing triangle, multiply and subtract rounded
// separately. What is arranged for latency, which bounds these fronts (a
// chain of up to 95 pivots, each a search, a reciprocal and an update):
//   - the leading dimension is odd, so that a row of the lower triangle is
//     read without bank conflicts;
//   - a warp tests one candidate column; its maxima are integer reductions
//     over the warp (two redux a maximum; non-negative doubles order as
//     their bits), the candidates of a round are published with one barrier;
//   - the columns of L are scaled by their pivots once at the end, while they
//     are written out, not pivot by pivot; counts come from the tags there;
//   - SPD: every thread forms the next pivot and its reciprocal itself,
//     beside the current update, so a pivot costs one barrier;
//   - up to four (update) and eight (children) columns a warp are in flight.
// Measured on one B200 against the kernels before (a warp per front of up to
// 64 rows, the size classes one after another, assembled and stored through
// global memory), factor + solve: one trajectory KKT of 10 stages 1.55 -> 0.58
// ms, of 200 stages 6.8 -> 3.9; 256 of them 23.5 -> 13.2; the 150 x 150
// Laplacian 6.7 -> 2.5, a 701 x 433 one 15.2 -> 8.0.
#pragma once
#include "smfg_kernels.cuh"

namespace smfg {

// Shared memory of a front of at most fmax rows: F (odd leading dimension),
// two arrays of pivot data, rows / loc / inv / child map, tags.
__host__ __device__ inline int small_smem_bytes(int fmax) {
  return (fmax * (fmax | 1) + 2 * fmax) * 8 + 4 * fmax * 4 + ((fmax + 7) / 8) * 8;
}

template <int NT>
__device__ __forceinline__ void small_sync() {
  if constexpr (NT == 32) __syncwarp();
  else __syncthreads();
}

// A barrier that tells every thread whether any gave true.
template <int NT>
__device__ __forceinline__ bool small_sync_or(bool b) {
  if constexpr (NT == 32) {
    const bool r = __any_sync(0xffffffffu, b) != 0;
    __syncwarp();
    return r;
  } else {
    return __syncthreads_or(b) != 0;
  }
}

// Rows and columns p < q of the front exchanged (sym_swap_blk's pairs), then
// a barrier.
template <int NT>
__device__ __forceinline__ void small_swap(double *F, int ld, int f, int *rows, int *loc, int p, int q) {
  if (p > q) {
    const int t = p;
    p = q;
    q = t;
  }
  for (int m = threadIdx.x; m < f; m += NT) {
    double *a, *b;
    if (m < p) {
      a = F + m * ld + p;
      b = F + m * ld + q;
    } else if (m == p) {
      a = F + p * ld + p;
      b = F + q * ld + q;
    } else if (m < q) {
      a = F + p * ld + m;
      b = F + m * ld + q;
    } else if (m > q) {
      a = F + p * ld + m;
      b = F + q * ld + m;
    } else {  // m == q: the entry (q, p) stays; the row ids
      const int r = rows[p], l = loc[p];
      rows[p] = rows[q];
      rows[q] = r;
      loc[p] = loc[q];
      loc[q] = l;
      continue;
    }
    const double x = *a;
    *a = *b;
    *b = x;
  }
  small_sync<NT>();
}

// One front of rows fmin..FMAX of the level list P.lvl_sn[i0 + blockIdx.x]
// (others return at once): k_level_rows, k_level_assemble, the front kernel
// and store_front in one.
template <int NT, int FMAX>
__global__ void __launch_bounds__(NT) k_small_front(DevPlan P, DevFactor X, int i0, PivotParams prm, int fmin,
                                                    int fmax) {
  constexpr int NW = NT / 32, NS = (FMAX + 31) / 32;
  constexpr int KC = 16;  // children described at a time
  extern __shared__ __align__(16) double small_smem[];
  __shared__ int sel[2][NW];
  __shared__ int ch_p[KC], ch_f[KC], ch_d[KC], ch_doff[KC], ch_cpr[KC];
  __shared__ long long ch_roff[KC], ch_off[KC];
  __shared__ int cnt_pos, cnt_neg, cnt_zero, cnt_two, bad_d;
  __shared__ unsigned long long flops_sh;
  // (one thread reads the flags, the first barrier tells the others: nothing is
  // written to global memory before it)
  const bool dead = threadIdx.x == 0 && abort_flagged(X);
  const int s = P.lvl_sn[i0 + blockIdx.x];
  const int f = X.sn_f[s];
  if (f < fmin || f > fmax || P.sn_large[s]) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ne = X.sn_ne[s], nd = X.sn_nd[s], fsym = P.sn_fsym[s];
  const int ld = f | 1;
  double *F = small_smem;
  double *q0 = F + f * ld, *q1 = q0 + f;  // pivot inverses (SPD: q1 the pivots)
  int *rows = reinterpret_cast<int *>(q1 + f);
  int *loc = rows + f, *inv = loc + f, *cm = inv + f;
  int8_t *tags = reinterpret_cast<int8_t *>(cm + f);
  prm.eff_small = __longlong_as_double((long long)X.counters[kCEffSmall]);
  const int64_t roff = X.sn_roff[s];
  double *Fg = X.arena + X.sn_off[s];

  // --- assembly (the order of additions of k_level_assemble)
  const int t0 = P.child_ptr[s], t1 = P.child_ptr[s + 1];
  auto describe = [&](int tb) {  // children [tb, tb + KC) into shared memory
    if (tid < KC && tb + tid < t1) {
      const int c = P.child_idx[tb + tid];
      ch_p[tid] = X.sn_p[c];
      ch_f[tid] = X.sn_f[c];
      ch_d[tid] = X.sn_dout[c];
      ch_doff[tid] = X.child_doff[tb + tid];
      ch_cpr[tid] = P.cpr_off[tb + tid];
      ch_roff[tid] = X.sn_roff[c];
      ch_off[tid] = X.sn_off[c];
    }
  };
  describe(t0);
  for (int t = tid; t < f * ld; t += NT) F[t] = 0.0;
  for (int u = tid; u < f; u += NT) {
    if (u < fsym) rows[nd + u] = P.frow_idx[P.frow_ptr[s] + u];
    loc[u] = u;
    tags[u] = 0;
  }
  if (tid == 0) {
    cnt_pos = cnt_neg = cnt_zero = cnt_two = bad_d = 0;
    flops_sh = 0;
  }
  if (small_sync_or<NT>(dead)) return;
  {
    const int cs = P.sn_start[s], wdt = P.sn_width[s];
    const int k0 = P.pcp[cs], k1 = P.pcp[cs + wdt];
    for (int k = k0 + tid; k < k1; k += NT) F[(nd + P.pcol[k] - cs) * ld + nd + P.amap[k]] += X.pv[k];
  }
  small_sync<NT>();
  for (int tb = t0; tb < t1; tb += KC) {
    if (tb > t0) {
      small_sync<NT>();
      describe(tb);
      small_sync<NT>();
    }
    const int nc = min(KC, t1 - tb);
    for (int c = 0; c < nc; ++c) {
      const int pc = ch_p[c], fc = ch_f[c], dc = ch_d[c], doff = ch_doff[c], q = fc - pc;
      if (q <= 0) continue;
      const int *cpr = P.cpr_idx + ch_cpr[c];
      const int *crow = X.rows + ch_roff[c] + pc;
      for (int u = tid; u < q; u += NT) {
        if (u < dc) rows[doff + u] = crow[u];
        cm[u] = u < dc ? doff + u : nd + cpr[u - dc];
      }
      const double *Fc = X.arena + ch_off[c] + (size_t)pc * fc + pc;
      small_sync<NT>();
      constexpr int G = 8;
      for (int j0 = warp; j0 < q; j0 += G * NW) {
        for (int i = j0 + lane; i < q; i += 32) {
          double x[G];
#pragma unroll
          for (int u = 0; u < G; ++u) {
            const int j = j0 + u * NW;
            x[u] = (j <= i) ? Fc[(size_t)j * fc + i] : 0.0;
          }
          const int li = cm[i];
#pragma unroll
          for (int u = 0; u < G; ++u) {
            const int j = j0 + u * NW;
            if (j <= i) {
              const int lj = cm[j];
              if (li < lj) set_flag(X.counters, kFMap);
              else F[lj * ld + li] += x[u];
            }
          }
        }
      }
      small_sync<NT>();
    }
  }

  // --- pivoting
  int p = 0;
  if (prm.posdef) {
    double d = F[0], iv = 1.0 / d;
    for (; p < ne; ++p) {
      if (!(d > 0.0 && isfinite(d))) break;
      const double *ck = F + p * ld;
      if (tid == 0) {
        q0[p] = iv;
        q1[p] = d;
        tags[p] = 1;
      }
      // the next pivot: its entry is read here and written by nobody
      double dn = 0.0, ivn = 0.0;
      if (p + 1 < ne) {
        const double w = ck[p + 1], l = __dmul_rn(w, iv);
        dn = F[(p + 1) * ld + p + 1];
        const double v = __dsub_rn(dn, __dmul_rn(w, l));
        dn = l != 0.0 ? v : dn;
        ivn = 1.0 / dn;
      }
      small_update1<NT>(F, ld, f, p, f, iv, p + 1 < ne ? p + 1 : -1);
      small_sync<NT>();
      d = dn;
      iv = ivn;
    }
    // a pivot that failed keeps its value in q1 for the store
    if (p < ne && tid == 0) q1[p] = d;
    small_sync<NT>();
    if (p < ne) {
      if (p > 0 && tid == 0) F[p * ld + p] = q1[p];
      small_sync<NT>();
    }
  } else {
    int rnd = 0;
    while (p < ne) {
      // the candidates' tests, NW at a time; the first that gives a pivot wins
      const double iv_k = 1.0 / F[p * ld + p];  // (used when column p itself is taken)
      int pick = 0;
      for (int c0 = p; c0 < ne; c0 += NW) {
        const int cand = c0 + warp;
        const int got = cand < ne ? small_cand<NS>(F, ld, f, ne, p, ne, cand, prm) : 0;
        if constexpr (NW == 1) {
          pick = got;
        } else {
          int *se = sel[rnd & 1];
          ++rnd;
          if (lane == 0) se[warp] = got;
          small_sync<NT>();
#pragma unroll
          for (int w = NW - 1; w >= 0; --w) {
            const int g = se[w];
            pick = g ? g : pick;
          }
        }
        if (pick) break;
      }
      if (!pick) break;
      const int kind = pick & 3, pa = (pick >> 2) & 255;
      if (NW == 1) small_sync<NT>();
      if (kind == 1) {
        if (pa != p) small_swap<NT>(F, ld, f, rows, loc, p, pa);
        const double iv = pa == p ? iv_k : 1.0 / F[p * ld + p];
        if (tid == 0) {
          q0[p] = iv;
          tags[p] = 1;
        }
        small_update1<NT>(F, ld, f, p, f, iv, -1);
        p += 1;
      } else {
        int partner = pick >> 10;
        if (pa != p) {
          small_swap<NT>(F, ld, f, rows, loc, p, pa);
          if (partner == p) partner = pa;
        }
        if (partner != p + 1) small_swap<NT>(F, ld, f, rows, loc, p + 1, partner);
        double i00, i10, i11;
        inverse_2x2(F[p * ld + p], F[p * ld + p + 1], F[(p + 1) * ld + p + 1], i00, i10, i11);
        if (tid == 0) {
          q0[p] = i00;
          q1[p] = i10;
          q0[p + 1] = i11;
          tags[p] = 2;
          tags[p + 1] = -1;
        }
        small_update2<NT>(F, ld, f, p, f, i00, i10, i11);
        p += 2;
      }
      small_sync<NT>();
    }
  }

  // --- store: L and D (store_front's forms), counts, row maps
  const bool is_root = P.sn_parent[s] < 0;
  const int pstore = (is_root && p < ne) ? ne : p;
  if (prm.posdef && p < ne && tid == 0) flag_not_posdef(P, X, s);
  small_sync<NT>();
  {
    int pos = 0, neg = 0, zero = 0, two = 0;
    unsigned long long fl = 0;
    bool bad = false;
    for (int c = tid; c < p; c += NT) {
      FrontStats st{0, 0, 0, 0, 0.0};
      const int tag = tags[c];
      if (tag == 1) {
        const double d = prm.posdef ? q1[c] : F[c * ld + c];
        inertia_1x1(d, prm.eff_small, st);
        const unsigned long long rem = (unsigned long long)(f - (c + 1));
        fl += rem + rem * (rem + 1);
        bad = bad || (!prm.posdef && !isfinite(d));
      } else if (tag == 2) {
        const double d00 = F[c * ld + c], d10 = F[c * ld + c + 1], d11 = F[(c + 1) * ld + c + 1];
        inertia_2x2(d00, d10, d11, prm.small_pivot, st);
        const unsigned long long rem = (unsigned long long)(f - (c + 2));
        fl += 6 * rem + 2 * rem * (rem + 1);
        ++two;
        bad = bad || !isfinite(d00) || !isfinite(d10) || !isfinite(d11);
      }
      pos += st.pos;
      neg += st.neg;
      zero += st.zero;
    }
    if (p > 0 && tid < p) {
      if (pos) atomicAdd(&cnt_pos, pos);
      if (neg) atomicAdd(&cnt_neg, neg);
      if (zero) atomicAdd(&cnt_zero, zero);
      if (two) atomicAdd(&cnt_two, two);
      if (bad) bad_d = 1;
      if (fl) atomicAdd(&flops_sh, fl);
    }
  }
  for (int c = warp; c < f; c += NW) {
    const double *Fc = F + c * ld;
    double *out = Fg + (size_t)c * f;
    if (c >= pstore) {  // contribution block
      for (int i = c + lane; i < f; i += 32) out[i] = Fc[i];
    } else if (prm.posdef) {
      const double sq = sqrt(c < p ? q1[c] : Fc[c]);
      const double iv = c < p ? q0[c] : 0.0;
      for (int i = lane; i < f; i += 32) {
        double v = 0.0;
        if (i == c) v = sq;
        else if (i > c) v = __dmul_rn(c < p ? __dmul_rn(Fc[i], iv) : Fc[i], sq);
        out[i] = v;
      }
    } else {
      const int tag = tags[c];  // 0: a zero pivot of the root, its column zero
      const double *Fa = tag == -1 ? Fc - ld : Fc, *Fb = tag == 2 ? Fc + ld : Fc;
      const double a = tag == 2 ? q0[c] : tag == -1 ? q1[c - 1] : tag == 1 ? q0[c] : 0.0;
      const double b = tag == 2 ? q1[c] : tag == -1 ? q0[c] : 0.0;
      for (int i = lane; i < f; i += 32) {
        double v = 0.0;
        if (tag == 1) {
          v = i == c ? Fc[i] : i > c ? __dmul_rn(Fc[i], a) : 0.0;
        } else if (tag == 2) {
          if (i == c) v = Fc[i];
          else if (i > c + 1) v = __dadd_rn(__dmul_rn(a, Fa[i]), __dmul_rn(b, Fb[i]));
        } else if (tag == -1) {
          if (i == c - 1) v = Fa[c];
          else if (i == c) v = Fc[i];
          else if (i > c) v = __dadd_rn(__dmul_rn(a, Fa[i]), __dmul_rn(b, Fb[i]));
        }
        out[i] = v;
      }
    }
  }
  for (int t = tid; t < f; t += NT) {
    X.rows[roff + t] = rows[t];
    X.tags[roff + t] = tags[t];
    inv[loc[t]] = t;
  }
  small_sync<NT>();
  // the children's row maps, in pivot order (the solves read them)
  for (int tb = t0; tb < t1; tb += KC) {
    if (t1 - t0 > KC) {
      small_sync<NT>();
      describe(tb);
      small_sync<NT>();
    }
    const int nc = min(KC, t1 - tb);
    for (int c = 0; c < nc; ++c) {
      const int pc = ch_p[c], dc = ch_d[c], doff = ch_doff[c], q = ch_f[c] - pc;
      const int *cpr = P.cpr_idx + ch_cpr[c];
      int *cmap = X.cbmap + ch_roff[c] + pc;
      for (int u = tid; u < q; u += NT) cmap[u] = inv[u < dc ? doff + u : nd + cpr[u - dc]];
    }
  }
  if (tid == 0) {
    if (bad_d) set_flag(X.counters, kFNonfiniteD);
    X.sn_p[s] = p;
    X.sn_pstore[s] = pstore;
    X.sn_dout[s] = is_root ? 0 : ne - p;
    int *st = X.sn_stat + 4 * s;
    st[0] = cnt_pos;
    st[1] = cnt_neg;
    st[2] = cnt_zero + (pstore - p);
    st[3] = cnt_two;
    X.sn_flops[s] = (double)flops_sh;
  }
}

}  // namespace smfg
