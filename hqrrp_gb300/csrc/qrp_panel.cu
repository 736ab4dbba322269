// qrp_panel.cu -- pivoted Householder QR of a tall panel, one cooperative
// kernel, plus the T factor of the resulting block reflector.
//
// Reference: lapack_compatible_sources/NoFLA_HQRRP_WY_blk_var4.c:520-524 runs
// NoFLA_QRPmod_WY_unb_var4 (:774-886) on the (m-j) x b panel with
// num_stages = -1 and build_T = 1: per column, idamax of the partial norms,
// swap (columns, labels, copied norms: :990-1036), dlarfg, dlarf on the
// trailing panel columns, Drmac's norm downdate with recompute on
// cancellation (:912-986); then dlarft Forward/Columnwise (:875-878).  The
// same kernel, run over all columns, serves the small-matrix path of dgeqp4
// (:189-199): LAPACK's dgeqpf and dgeqp3 pick pivots by the same rule and
// downdate norms with the same LAWN 176 test.
//
// GB300 layout: the panel's rows are split into contiguous slabs, one per CTA
// (one CTA per SM), kept in shared memory when they fit (108 rows x 128
// columns = 110 KB at m = 16384) and otherwise worked on in place in L2.
// Column swaps are then local to every CTA.  Each stage needs one grid
// exchange: every CTA adds, for its slab, the dot products of the pivot
// column with all not-yet-factored columns (the first of which is the pivot
// column's squared norm); the owner of the pivot row also publishes that row.
// The partials are summed as fixed-point integers: each CTA adds its partial
// of column k, exactly, as three 48-bit limbs of a 144-bit integer in units
// of 2^ue_k (ue_k from the two columns' norms, which bound every partial and
// their sum by Cauchy-Schwarz) to three 64-bit words with L2 atomics.
// Integer addition is associative, so the order of the atomics does not
// matter: the sums are the same in every run, and exact up to the truncation
// below 2^ue_k (2^-133 of the bound, far below FP64 rounding of the
// partials).  Every CTA reads the words of all columns, converts them to FP64
// and builds the reflector itself (identical inputs, identical results) --
// FP64 adds of 152 partials per column in every CTA would cost microseconds
// on this GPU's FP64 pipe, integer atomics do not.
//
// What bounds a stage is latency, so the exchange has no barrier and no fence:
// every add also counts one in the word's upper byte, and a reader polls each
// word until it has grown by the number of CTAs (the row travels in words
// tagged with the stage).  Words are never cleared: readers keep the value
// they last saw, so a word's growth since then is the stage's sum and count.
// Two buffers alternate -- a CTA adds to a buffer again two stages later,
// after it has seen every CTA's adds of the stage between, which each made
// after reading this one.  A column's adds are spread over R words (lines) by
// CTA, because adds and polls of 125 CTAs to one line queue up.
//
// Between two exchanges a stage works in the order the next exchange needs:
// reflector, the new row and norms of all columns and with them the next
// pivot, that pivot's column, and then one pass that updates every other
// column and takes its dot product with it.  Norms are kept squared (d^2 <-
// d^2 - r^2, recomputed when d^2 - r^2 <= tol3z e^2, LAWN 176's test without
// its divisions and square root).  The rare norm recomputation costs a barrier
// in the stages that need it (FP64 partials, summed in a fixed order in every
// CTA) and takes update and dot products one after the other.
//
// Measured on GB300 against a counter barrier, separate passes for dot products
// and update, LAPACK's norm formula and divisions (15.6k clocks a stage of
// 2000 x 64 on 125 CTAs: swap 0.5, dots 2.2, barrier 3.3, sums and reflector
// 4.4, update 1.5, norms 3.6): 2000 x 64 panels 7.5 -> 4.5 us a stage, a 641 x
// 481 factorization 5.8 -> 3.6 ms.
#include "hq_common.cuh"
#include "hq_fixedpoint.h"

namespace {

constexpr int MAX_G = 160;          // CTAs (one per SM); partial loads per lane <= 5
constexpr int CB = (MAX_G + 31) / 32;
constexpr int QB = 8;               // columns reduced per warp per batch of loads
constexpr int APART_COST = 16;      // FP64 instructions' time, 64 clocks each
constexpr int APART_ROWS = 192;

struct PnArgs {
  int mp, nc, ns, pivoting;
  double* P;
  int ldp;
  double* tau;
  double* U;
  int ldu;
  int* perm;
  double* part;             // [2][pstride][grid] partials (column q's contiguous)
  unsigned long long* acc;  // [2][R][pstride][FX_CS] fixed-point stage sums
  unsigned long long* rows; // [2][pstride][2] the pivot row, tagged
  int pstride;
  unsigned* bar;
  int* err;
  unsigned spin_limit;
  int smem_mode, rloc_max, ldxs;
  int ut;      // UT-transform convention: a zero tail gives H = I - 2 e e^T (tau 2, beta -alpha)
  const int* gram_stat;  // non-null: skip when *gram_stat == 0 (the Gram panel succeeded)
};

// Fixed-point stage sums (hq_fixedpoint.h): words 0..2 of a column are the
// limbs' signed accumulators in their lower 56 bits -- a limb's sum over one
// word's CTAs (at most 127) stays below 2^55 -- with the count of adds above.
// A non-finite partial adds FX_NONFINITE to limb 2, which finite partials
// cannot reach.
constexpr int FX_CS = HQ_PANEL_FX_CS;  // words between consecutive columns
constexpr unsigned long long FX_ONE = 1ull << 56;
constexpr unsigned long long FX_NONFINITE = 1ull << 46;

// Adds t / 2^ue, truncated to an integer, to the words w.
__device__ __forceinline__ void fx_add(unsigned long long* w, double t, int ue) {
  unsigned long long p[3] = {0ull, 0ull, 0ull};
  int L = 0;
  const int rc = hq_fx_split(t, ue, p, &L);
  unsigned long long v0 = FX_ONE, v1 = FX_ONE, v2 = FX_ONE;
  if (rc == 1) {
    v0 += L == 0 ? p[0] : 0ull;
    v1 += L == 0 ? p[1] : (L == 1 ? p[0] : 0ull);
    v2 += L == 0 ? p[2] : (L == 1 ? p[1] : p[0]);
  } else if (rc == 2) {
    v2 += FX_NONFINITE;
  }
  hq_red_word(w, v0);
  hq_red_word(w + 1, v1);
  hq_red_word(w + 2, v2);
}

// Candidate order for the pivot: larger norm, then lower column (idamax's
// first maximum); NaN never wins.
__device__ __forceinline__ void pick(long long key, int k, long long& bkey, int& bk) {
  if (key > bkey || (key == bkey && k < bk)) { bkey = key; bk = k; }
}

// The warp's pick in every lane (keys are >= -2).
__device__ __forceinline__ void warp_pick(long long& bkey, int& bk) {
  const unsigned long long u = (unsigned long long)(bkey + 4);
  const unsigned hi = (unsigned)(u >> 32);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = hi == mh ? (unsigned)u : 0u;
  const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
  bk = __reduce_min_sync(0xffffffffu, hi == mh && (unsigned)u == ml ? bk : 0x7fffffff);
  bkey = (long long)(((unsigned long long)mh << 32) | ml) - 4;
}

template <int NT, int EPT, int R>
__global__ void __launch_bounds__(NT, 1) panel_qrp_kernel(PnArgs a) {
  HQ_PDL_WAIT();
  constexpr int NWARP = NT / 32;
  extern __shared__ __align__(16) double smem[];
  // Every CTA reads the same word, written before the launch.
  if (a.gram_stat != nullptr && *a.gram_stat == 0) return;
  const int G = gridDim.x, cta = blockIdx.x, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int nc = a.nc;
  const int r_lo = (int)((long long)cta * a.mp / G);
  const int r_hi = (int)((long long)(cta + 1) * a.mp / G);
  const int nloc = r_hi - r_lo;

  double* sX = smem;
  double* sd = sX + (a.smem_mode ? (size_t)a.ldxs * nc : 0);
  double* se = sd + nc;
  double* sw = se + nc;      // reduced dots of the stage, then tau v^T X
  double* srow = sw + nc;    // pivot row of the stage, then its new values
  // The columns' labels; in shared memory also where column k lives in X.
  int* sperm = reinterpret_cast<int*>(srow + nc);
  int* sflag = sperm + nc;
  __shared__ int s_flag;
  __shared__ long long s_bd[NWARP];
  __shared__ int s_bk[NWARP];
  __shared__ double s_tau, s_scale, s_beta;

  double* X;
  int ldx;
  if (a.smem_mode) {
    X = sX;
    ldx = a.ldxs;
    for (int k = warp; k < nc; k += NWARP)
      for (int i = lane; i < nloc; i += 32) X[i + (size_t)k * ldx] = a.P[r_lo + i + (size_t)k * a.ldp];
  } else {
    X = a.P + r_lo;
    ldx = a.ldp;
  }
  for (int k = tid; k < nc; k += NT) {
    sperm[k] = k;
    sflag[k] = 0;
  }
  // A valid permutation is in place before any wait: if a wait gives up and
  // the kernel returns early, the gathers that follow still read indices
  // within range.  The stage words start at zero, ordered before the first
  // add by the barrier of the initial norms.
  if (cta == 0)
    for (int k = tid; k < nc; k += NT) a.perm[k] = k;
  for (size_t i = (size_t)cta * NT + tid; i < (size_t)2 * R * a.pstride; i += (size_t)G * NT) {
    unsigned long long* w = a.acc + i * FX_CS;
    w[0] = w[1] = w[2] = 0ull;
    if (i < (size_t)2 * a.pstride) a.rows[2 * i + 1] = 0ull;
  }
  __syncthreads();

  unsigned epoch = 0;
  auto part_w = [&](unsigned e) { return a.part + (size_t)(e & 1) * a.pstride * G + cta; };
  auto part_r = [&](unsigned e) { return a.part + (size_t)(e & 1) * a.pstride * G; };
  auto colp = [&](int k) { return X + (size_t)(a.smem_mode ? sperm[k] : k) * ldx; };
  // The words of stage s, column k, that CTAs of index rep modulo R add to.
  auto words = [&](int s, int rep, int k) {
    return a.acc + ((size_t)((s & 1) * R + rep) * a.pstride + k) * FX_CS;
  };
  const int myrep = cta & (R - 1);
  auto put_row = [&](int s, int k, double x) {
    hq_st_word(a.rows + ((size_t)(s & 1) * a.pstride + k) * 2,
               (unsigned long long)__double_as_longlong(x), (unsigned long long)s + 1ull);
  };
  // Lanes per column for na columns: a power of two, adjacent lanes.
  auto lanes_for = [&](int na) {
    int g = 1;
    while (g < 32 && 2 * g * na <= NT) g *= 2;
    return g;
  };

  // Slab-local sums over rows with global index > lo_row of x_i * X[i, k]
  // (x = column xs, or column k itself when xs < 0) for k in [k0, nc),
  // skipping columns without sflag when use_mask; column k's sum goes to
  // out[(k - k0) * G], or, without out, to stage xs's fixed-point words.
  auto slab_dots = [&](int xs, int k0, int lo_row, bool use_mask, double* out) {
    const int na = nc - k0;
    const int i0 = max(0, lo_row + 1 - r_lo);
    const int groups = lanes_for(na);
    const int g = tid & (groups - 1), stride = NT / groups;
    // The trip count is the same for every thread, so whole warps take part
    // in the shuffles; columns past the end contribute zero.
    for (int q0 = 0; q0 < na; q0 += stride) {
      const int q = q0 + tid / groups;
      const int k = k0 + q;
      double t = 0.0;
      if (q < na && (!use_mask || sflag[k])) {
        const double* xk = colp(k);
        const double* xx = xs >= 0 ? colp(xs) : xk;
        double t1 = 0.0;
        int i = i0 + g;
        for (; i + groups < nloc; i += 2 * groups) {
          t = fma(xx[i], xk[i], t);
          t1 = fma(xx[i + groups], xk[i + groups], t1);
        }
        if (i < nloc) t = fma(xx[i], xk[i], t);
        t += t1;
      }
      for (int o = groups >> 1; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (g == 0 && q < na) {
        if (out) out[(size_t)q * G] = t;
        else fx_add(words(xs, myrep, k), t, hq_fx_unit(se[xs], se[k], 1));
      }
    }
  };

  // sw[q] = sum over CTAs of the published column q (q < na), in a fixed
  // order, formed in every CTA (used for the one-off initial norms and the
  // rare norm recomputations).  Warp w takes columns w*QB.. in batches of QB,
  // lane l the CTAs l, l+32, ...; every load of a batch is issued before any
  // is used.
  auto reduce_parts = [&](unsigned e, int na) {
    const double* base = part_r(e);
    for (int q0 = warp * QB; q0 < na; q0 += NWARP * QB) {
      double v[QB][CB];
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        const int q = q0 + u;
#pragma unroll
        for (int j = 0; j < CB; ++j) {
          const int c = lane + 32 * j;
          v[u][j] = (q < na && c < G) ? hq_ldcg(base + (size_t)q * G + c) : 0.0;
        }
      }
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        double t = v[u][0];
#pragma unroll
        for (int j = 1; j < CB; ++j) t += v[u][j];
        t = hq_warp_sum(t);
        if (lane == u && q0 + u < na) sw[q0 + u] = t;
      }
    }
    __syncthreads();
  };

  // This thread polls the R words of columns k = tid + NT j, j < EPT.  h0, h1:
  // what each word held after its last stage, by the stage's parity.
  unsigned long long h0[EPT][R][3], h1[EPT][R][3];
#pragma unroll
  for (int j = 0; j < EPT; ++j)
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int i = 0; i < 3; ++i) h0[j][r][i] = h1[j][r][i] = 0ull;

  // Stage s's exchange: the sums and the pivot row of columns k >= s, as they
  // become complete, and the reflector (built by one thread of every CTA from
  // the same inputs).  Returns false in every thread if a wait gave up.
  auto gather_sums = [&](int s) {
    const bool odd = s & 1;
    const unsigned long long tag = (unsigned long long)s + 1ull;
    unsigned long long w[EPT][R][3], xr[EPT], xt[EPT];
    auto load = [&](int j, int k) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const unsigned long long* p = words(s, r, k);
        hq_ld_word(p, w[j][r][0], w[j][r][1]);
        hq_ld_word(p + 2, w[j][r][2]);
      }
      hq_ld_word(a.rows + ((size_t)odd * a.pstride + k) * 2, xr[j], xt[j]);
    };
    auto complete = [&](int j) {
      bool ok = xt[j] == tag;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const long long n_adds = (G - r + R - 1) / R;  // CTAs of this word
#pragma unroll
        for (int i = 0; i < 3; ++i)
          ok = ok && ((long long)(w[j][r][i] - (odd ? h1[j][r][i] : h0[j][r][i])) + (1LL << 55)) >> 56 == n_adds;
      }
      return ok;
    };
#pragma unroll
    for (int j = 0; j < EPT; ++j) {
      const int k = tid + NT * j;
      if (k >= s && k < nc) load(j, k);
    }
    // sw and srow, written below, are read until here by the pass before, in
    // which one thread rewrites the labels: se[s] is read from here on.
    __syncthreads();
    const double sep = se[s];
    int bad = 0;
    unsigned it = 0;
#pragma unroll
    for (int j = 0; j < EPT; ++j) {
      const int k = tid + NT * j;
      if (k < s || k >= nc) continue;
      while (!complete(j) && !bad) {
        if (++it >= a.spin_limit) {
          atomicCAS(a.err, 0, HQ_ERR_BARRIER_TIMEOUT);
          bad = 1;
        } else if ((it & 15u) == 0u && hq_ld_volatile(a.err) != 0) {
          bad = 1;
        }
        load(j, k);
      }
      long long d[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        d[i] = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          d[i] += (long long)(w[j][r][i] - (odd ? h1[j][r][i] : h0[j][r][i]));
          if (odd) h1[j][r][i] = w[j][r][i];
          else h0[j][r][i] = w[j][r][i];
        }
        d[i] -= (long long)G << 56;
      }
      const double t = d[2] > (long long)(FX_NONFINITE >> 1)
                           ? __longlong_as_double(0x7FF8000000000000LL)
                           : hq_fx_combine(d[0], d[1], d[2], hq_fx_unit(sep, se[k], 1));
      const double r = __longlong_as_double((long long)xr[j]);
      sw[k - s] = t;
      srow[k - s] = r;
      if (k == s) {
        const double tail = (a.mp - s > 1) ? t : 0.0;
        HqReflector hr;
        if (a.ut && tail == 0.0) {  // libflame's Househ2_UT: chi_1 := -chi_1, tau_UT = 1/2
          hr.tau = 2.0;
          hr.beta = -r;
          hr.scale = 1.0;
        } else {
          hr = hq_make_reflector_sq(r, tail);
        }
        s_tau = hr.tau;
        s_scale = hr.scale;
        s_beta = hr.beta;
      }
    }
    return __syncthreads_or(bad) == 0;
  };

  // Block argmax of (sd[k], k) over k in [k0, nc); every thread returns the
  // same index (k0 when no column qualifies, e.g. all norms NaN).
  auto block_argmax = [&](int k0) {
    long long bd = -2;
    int bk = 0x7fffffff;
    for (int k = k0 + tid; k < nc; k += NT) pick(hq_norm_key(sd[k]), k, bd, bk);
    warp_pick(bd, bk);
    if (lane == 0) { s_bd[warp] = bd; s_bk[warp] = bk; }
    __syncthreads();
    bd = s_bd[0];
    bk = s_bk[0];
    for (int w = 1; w < NWARP; ++w) pick(s_bd[w], s_bk[w], bd, bk);
    __syncthreads();  // s_bd is reused by the next call
    return (bk == 0x7fffffff || bd < 0) ? k0 : bk;
  };

  // The pivot among the warps' picks in s_bd, s_bk, or k0.
  auto next_pivot = [&](int k0) {
    if (!a.pivoting) return k0;
    long long bd = s_bd[0];
    int bk = s_bk[0];
    for (int w = 1; w < NWARP; ++w) pick(s_bd[w], s_bk[w], bd, bk);
    return bk != 0x7fffffff && bd >= 0 ? bk : k0;
  };
  // Whether update and dot products of na columns are made one after the other.
  // Both are bound by the FP64 pipe when a slab is long, and the pass that does
  // both deals columns out by a power of two of lanes, so some warps may have
  // none (40 columns of 4 lanes: five warps of eight); the update alone takes any
  // number of lanes.  Compared: the FP64 instructions that the busiest quarter of
  // the SM issues, and APART_COST for the barrier and the second reading.  (One
  // pass always -> this, us: 50000 x 80 1498 -> 1204, 100000 x 40 753 -> 610,
  // 200000 x 20 403 -> 331.  In shorter slabs the comparison costs a stage up to
  // 5 % and changes little; out of shared memory the second reading costs more.)
  const bool long_slab = a.smem_mode && a.rloc_max > APART_ROWS;
  auto apart = [&](int na) {
    const int g = lanes_for(na);
    const int warps = ((na * g > NT ? NT : na * g) + 127) >> 7;  // of a quarter
    const int both = (a.rloc_max * warps + g - 1) / g;
    const int groups = na < NT ? NT / na : 1;
    const int update = (a.rloc_max * (NT >> 7) + groups - 1) / groups;
    return both > update + APART_COST;
  };

  // One thread: columns s and kp change places (labels, copied norms; se[s]
  // takes the pivot's own value, which bounds its stage sums -- position s's
  // norms are not read again otherwise).
  auto swap_labels = [&](int s, int kp) {
    const int t = sperm[s];
    sperm[s] = sperm[kp];
    sperm[kp] = t;
    const double pse = se[kp];
    sd[kp] = sd[s];
    se[kp] = se[s];
    se[s] = pse;
  };
  // In place (not in shared memory) the columns themselves are swapped.
  auto swap_columns = [&](int s, int kp) {
    if (a.smem_mode || kp == s) return;
    double* c1 = X + (size_t)s * ldx;
    double* c2 = X + (size_t)kp * ldx;
    for (int i = tid; i < nloc; i += NT) {
      const double t = c1[i];
      c1[i] = c2[i];
      c2[i] = t;
    }
  };
  // Start stage s on its own: pivot kp to position s, row s out, dots added.
  auto begin_stage = [&](int s, int kp) {
    swap_columns(s, kp);
    if (tid == 0 && kp != s) swap_labels(s, kp);
    __syncthreads();
    if (s >= r_lo && s < r_hi)
      for (int k = s + tid; k < nc; k += NT) put_row(s, k, colp(k)[s - r_lo]);
    slab_dots(s, s, s, false, nullptr);
  };

  // Initial norms over the whole panel.
  slab_dots(-1, 0, -1, false, part_w(epoch + 1));
  ++epoch;
  if (!hq_grid_barrier(a.bar, a.err, epoch, a.spin_limit, &s_flag)) return;
  reduce_parts(epoch, nc);
  for (int k = tid; k < nc; k += NT) {
    sd[k] = sw[k];
    se[k] = sw[k];
  }
  __syncthreads();
  begin_stage(0, a.pivoting ? block_argmax(0) : 0);

  for (int s = 0; s < a.ns; ++s) {
    // 1. Sums, pivot row and reflector in every CTA.
    if (!gather_sums(s)) return;
    const double tau = s_tau, scale = s_scale;
    const int i0 = max(0, s + 1 - r_lo);
    const bool own = s >= r_lo && s < r_hi;
    double* v = colp(s);
    if (cta == 0 && tid == 0) a.tau[s] = tau;

    // 2. w_k = tau * v^T X[:, k] = tau * (scale * dot_k + row_k), the new
    //    entries row_k - w_k of row s, the norm downdate and the next pivot;
    //    v = [1; scale * x] in place (rows > s), beta on the diagonal.
    int any = 0;
    long long bd = -2;
    int bk = 0x7fffffff;
    for (int k = s + 1 + tid; k < nc; k += NT) {
      const int q = k - s;
      const double thr = HQ_TOL3Z * se[k];
      const double wk = tau * fma(scale, sw[q], srow[q]);
      const double r = srow[q] - wk;
      sw[q] = wk;
      srow[q] = r;
      if (a.pivoting) {
        int flag = 0;
        double dk = sd[k];
        if (dk != 0.0) {
          const double nd = fma(-r, r, dk);
          if (hq_norm_cancelled(nd, thr)) {
            flag = 1;
          } else {
            dk = nd;
            sd[k] = dk;
          }
        }
        sflag[k] = flag;
        any |= flag;
        pick(hq_norm_key(dk), k, bd, bk);
      }
    }
    for (int i = i0 + NT - 1 - tid; i < nloc; i += NT) v[i] *= scale;
    if (tid == NT - 1 && own) v[s - r_lo] = s_beta;
    warp_pick(bd, bk);
    if (lane == 0) { s_bd[warp] = bd; s_bk[warp] = bk; }
    any = __syncthreads_or(any);

    if (any || s + 1 == a.ns || (long_slab && apart(nc - s - 1))) {
      // 3a. The last stage, norms to be recomputed, or a long slab: update the
      //     slab, X[i, k] -= v_i w_k for rows > s; the owner of row s stores its
      //     new entries.
      const int nt = nc - s - 1;
      if (nt >= NT) {
        for (int q = tid; q < nt; q += NT) {
          double* xk = colp(s + 1 + q);
          for (int i = i0; i < nloc; ++i) xk[i] = fma(-v[i], sw[q + 1], xk[i]);
          if (own) xk[s - r_lo] = srow[q + 1];
        }
      } else if (nt > 0) {
        const int groups = NT / nt, q = tid % nt, g = tid / nt;
        if (g < groups) {
          double* xk = colp(s + 1 + q);
          for (int i = i0 + g; i < nloc; i += groups) xk[i] = fma(-v[i], sw[q + 1], xk[i]);
          if (own && g == 0) xk[s - r_lo] = srow[q + 1];
        }
      }
      __syncthreads();
      if (s + 1 == a.ns) break;
      if (!any) {
        begin_stage(s + 1, next_pivot(s + 1));
        continue;
      }
      slab_dots(-1, s, s, true, part_w(epoch + 1));
      ++epoch;
      if (!hq_grid_barrier(a.bar, a.err, epoch, a.spin_limit, &s_flag)) return;
      reduce_parts(epoch, nc - s);
      for (int k = s + 1 + tid; k < nc; k += NT) {
        if (sflag[k]) {
          const double nv = (a.mp - s - 1 > 0) ? sw[k - s] : 0.0;
          sd[k] = nv;
          se[k] = nv;
          sflag[k] = 0;
        }
      }
      __syncthreads();
      begin_stage(s + 1, block_argmax(s + 1));
      continue;
    }

    // 3b. The next pivot's column, and its place.
    const int kp = next_pivot(s + 1);
    // What positions s + 1 and kp hold before they change places: one thread
    // rewrites the labels during the pass below, which takes these two
    // positions from here.
    const int s1 = s + 1;
    double* z = colp(kp);
    double* x1 = colp(s1);
    const double se_z = se[kp], se_1 = se[s1], sd_1 = sd[s1];
    const int lab_z = sperm[kp], lab_1 = sperm[s1];
    {
      const double wk = sw[kp - s];
      for (int i = i0 + tid; i < nloc; i += NT) z[i] = fma(-v[i], wk, z[i]);
      if (own && tid == NT - 1) z[s - r_lo] = srow[kp - s];
    }
    __syncthreads();
    if (kp != s1) {
      if (!a.smem_mode) {
        swap_columns(s1, kp);
        double* u = z;
        z = x1;
        x1 = u;
        __syncthreads();
      }
      if (tid == NT - 1) {
        sperm[s1] = lab_z;
        sperm[kp] = lab_1;
        sd[kp] = sd_1;
        se[kp] = se_1;
        se[s1] = se_z;
      }
    }

    // 4. One pass over the other columns (now at positions k > s + 1): the
    //    update of stage s, and the dot products of stage s + 1 over rows
    //    > s + 1; the owner of row s + 1 publishes it.
    {
      const int na = nc - s1;
      const bool own1 = s1 >= r_lo && s1 < r_hi;
      const int groups = lanes_for(na);
      const int g = tid & (groups - 1), stride = NT / groups;
      for (int q0 = 0; q0 < na; q0 += stride) {
        const int q = q0 + tid / groups, k = s1 + q;
        double t = 0.0;
        if (q < na) {
          double* xk = k == kp ? x1 : (q == 0 ? z : colp(k));
          int i = i0 + g;
          if (q == 0) {
            if (own1 && g == 0) {
              put_row(s1, k, z[i]);
              i += groups;
            }
            for (; i < nloc; i += groups) t = fma(z[i], z[i], t);
          } else {
            const int old = k == kp ? s1 : k;  // where its w and row entry are
            const double wk = sw[old - s];
            if (own1 && g == 0) {
              const double x = fma(-v[i], wk, xk[i]);
              xk[i] = x;
              put_row(s1, k, x);
              i += groups;
            }
            for (; i < nloc; i += groups) {
              const double x = fma(-v[i], wk, xk[i]);
              xk[i] = x;
              t = fma(z[i], x, t);
            }
            if (own && g == 0) xk[s - r_lo] = srow[old - s];
          }
        }
        for (int o = groups >> 1; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (g == 0 && q < na)
          fx_add(words(s1, myrep, k), t,
                 hq_fx_unit(se_z, q == 0 ? se_z : (k == kp ? se_1 : se[k]), 1));
      }
    }
  }

  // Write back, explicit unit-lower U, permutation.
  __syncthreads();
  if (a.smem_mode) {
    for (int k = warp; k < nc; k += NWARP)
      for (int i = lane; i < nloc; i += 32) a.P[r_lo + i + (size_t)k * a.ldp] = colp(k)[i];
  }
  if (a.U != nullptr) {
    for (int k = warp; k < nc; k += NWARP)
      for (int i = lane; i < nloc; i += 32) {
        const int gi = r_lo + i;
        a.U[gi + (size_t)k * a.ldu] = gi > k ? colp(k)[i] : (gi == k ? 1.0 : 0.0);
      }
  }
  if (cta == 0)
    for (int k = tid; k < nc; k += NT) a.perm[k] = sperm[k];
}

// One CTA per 16 rows up to one per SM: a stage's FP64 work is spread over
// as many SMs as the panel has 16-row slabs (64-row slabs leave SMs idle on a
// small late panel while the exchange costs about the same).  Beyond 128
// columns the slab's own work is what a stage waits for, and 8 rows pay: 641 x
// 481 takes 4.02 ms with 16 rows a CTA, 3.58 with 8 (32: 7.3, measured with an
// earlier exchange); a 2000 x 64 panel does not change.
int panel_grid(const hq_device_info* dev, int mp, int nc) {
  const int rows = nc > 128 ? 8 : 16;
  int g = (mp + rows - 1) / rows;
  if (g > dev->num_sms) g = dev->num_sms;
  if (g > MAX_G) g = MAX_G;
  return g < 1 ? 1 : g;
}

// DLARFT (Forward, Columnwise) from the Gram matrix Z = U^T U, one CTA per row:
// row r of T only involves row r itself,
// T[r, i] = -tau_i * sum_{c = r}^{i-1} T[r, c] Z[c, i] for i > r, T[r, r] =
// tau_r (zero when tau_i = 0), so the k rows are independent recurrences and
// run side by side on the SMs instead of one SM's FP64 pipe doing all of them.
// A thread holds one entry of the row and a warp 32: the warps before it hand
// theirs over in shared memory, and within the warp each entry, once known,
// is broadcast and added to the ones after it with the factors -tau_i Z[c, i]
// ready in registers -- a shuffle and a fused multiply-add a step.  (A dot
// product and a warp sum a step took 60 us for k = 64 and 132 for 128; this
// takes 9 and 16.)
__global__ void __launch_bounds__(HQ_MAX_MY) larft_rows_kernel(
    int k, const double* __restrict__ Z, int ldz, const double* __restrict__ tau,
    double* __restrict__ T, int ldt) {
  __shared__ double sx[HQ_MAX_MY];
  const int r = blockIdx.x, c = threadIdx.x, lane = c & 31, warp = c >> 5;
  const int n = k - r;  // T[r, r + c], c < n
  const bool live = c < n;
  const double t = live ? tau[r + c] : 0.0;
  const double* zc = Z + r + (size_t)(r + (live ? c : 0)) * ldz;
  double z[32];
#pragma unroll
  for (int d = 0; d < 32; ++d) z[d] = live && d < lane ? -t * zc[warp * 32 + d] : 0.0;
  double acc = 0.0, x = 0.0;
  const int nw = (n + 31) >> 5;
  for (int b = 0; b < nw; ++b) {
    double zb[32];
    if (warp > b && live) {
#pragma unroll
      for (int d = 0; d < 32; ++d) zb[d] = zc[32 * b + d];
    }
    if (warp == b) {
      const bool on = t != 0.0;
      x = c == 0 ? t : (on ? -t * acc : 0.0);
#pragma unroll
      for (int d = 0; d < 31; ++d) {
        const double xd = __shfl_sync(0xffffffffu, x, d);
        if (on && lane > d) x = fma(xd, z[d], x);
      }
      sx[c] = x;
    }
    __syncthreads();
    if (warp > b && live) {
      double acc2 = 0.0;
#pragma unroll
      for (int d = 0; d < 32; d += 2) {
        acc = fma(sx[32 * b + d], zb[d], acc);
        acc2 = fma(sx[32 * b + d + 1], zb[d + 1], acc2);
      }
      acc += acc2;
    }
  }
  if (live) T[r + (size_t)(r + c) * ldt] = x;
  for (int i = c; i < r; i += blockDim.x) T[r + (size_t)i * ldt] = 0.0;
}

}  // namespace

extern "C" size_t hq_panel_part_elems(const hq_device_info* dev, int nc) {
  // A narrower panel may spread its columns over more words.
  const size_t e = HQ_PANEL_PART_ELEMS(dev->num_sms, nc);
  const int n4 = nc < 128 ? nc : 128;
  const size_t e4 = HQ_PANEL_PART_ELEMS(dev->num_sms, n4);
  return e > e4 ? e : e4;
}

extern "C" int hq_panel_qrp(cudaStream_t stream, const hq_device_info* dev, int mp, int nc,
                            int pivoting, double* P, int ldp, double* tau,
                            double* U, int ldu, int* perm, double* part, size_t part_elems,
                            unsigned* bar, int* err, unsigned spin_limit, int ut) {
  return hq_panel_qrp_fallback(stream, dev, mp, nc, pivoting, P, ldp, tau, U, ldu, perm, part,
                               part_elems, bar, err, spin_limit, ut, nullptr);
}

extern "C" int hq_panel_qrp_fallback(cudaStream_t stream, const hq_device_info* dev, int mp,
                                     int nc, int pivoting, double* P, int ldp, double* tau,
                                     double* U, int ldu, int* perm, double* part,
                                     size_t part_elems, unsigned* bar, int* err,
                                     unsigned spin_limit, int ut, const int* gram_stat) {
  if (nc <= 0 || mp <= 0) return 0;
  if (nc > HQ_MAX_PANEL) return (int)cudaErrorInvalidValue;
  PnArgs a;
  a.mp = mp;
  a.nc = nc;
  a.ns = mp < nc ? mp : nc;
  a.pivoting = pivoting;
  a.P = P;
  a.ldp = ldp;
  a.tau = tau;
  a.U = U;
  a.ldu = ldu;
  a.perm = perm;
  a.part = part;
  a.pstride = (nc + 2) & ~1;
  a.bar = bar;
  a.err = err;
  a.spin_limit = spin_limit;
  a.ut = ut;
  a.gram_stat = gram_stat;
  const int G = panel_grid(dev, mp, nc);
  if (HQ_PANEL_PART_ELEMS(G, nc) > part_elems) return (int)cudaErrorInvalidValue;
  const int R = HQ_PANEL_R(nc);
  a.acc = reinterpret_cast<unsigned long long*>(part + (size_t)2 * G * a.pstride);
  a.rows = a.acc + (size_t)2 * R * a.pstride * FX_CS;
  a.rloc_max = (mp + G - 1) / G;
  a.ldxs = a.rloc_max | 1;
  const size_t fixed = sizeof(double) * (4 * (size_t)nc) + sizeof(int) * (2 * (size_t)nc + 2);
  const size_t with_x = fixed + sizeof(double) * (size_t)a.ldxs * nc;
  size_t smem;
  if (with_x <= dev->smem_optin) {
    a.smem_mode = 1;
    smem = with_x;
  } else {
    a.smem_mode = 0;
    smem = fixed;
    if (smem > dev->smem_optin) return (int)cudaErrorInvalidValue;
  }
  const int nt = nc <= 128 ? 256 : 512;
  const void* fn = R == 4       ? (const void*)panel_qrp_kernel<256, 1, 4>
                   : nc <= 512  ? (const void*)panel_qrp_kernel<512, 1, 2>
                                : (const void*)panel_qrp_kernel<512, 2, 2>;
  static_assert(HQ_PANEL_R(128) == 4 && HQ_PANEL_R(129) == 2 && HQ_MAX_PANEL <= 1024, "shapes");
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int z = hq_zero_words(stream, bar, 1, nullptr, 0);
  if (z) return z;
  void* args[] = {&a};
  e = hq_launch_coop(fn, dim3(G), dim3(nt), args, smem, stream);
  hq_count_launches(1);
  return (int)e;
}

extern "C" int hq_larft_from_gram(cudaStream_t stream, int k, const double* Z, int ldz,
                                  const double* tau, double* T, int ldt) {
  if (k <= 0) return 0;
  if (k > HQ_MAX_MY) return (int)cudaErrorInvalidValue;
  larft_rows_kernel<<<k, (k + 31) / 32 * 32, 0, stream>>>(k, Z, ldz, tau, T, ldt);
  hq_count_launches(1);
  return (int)cudaGetLastError();
}
