// qrp_skinny.cu -- per-block pivot selection: b stages of pivoted Householder
// QR on the (nb+pp) x N sketch Y, in one cooperative kernel.
//
// Reference: lapack_compatible_sources/NoFLA_HQRRP_WY_blk_var4.c:492-507 copies
// Y_R into V_R and runs NoFLA_QRPmod_WY_unb_var4 (:774-886) with num_stages =
// b, which per stage takes idamax of the partial column norms (:828), swaps
// the columns of V, A, Y and the labels (:831-837, :990-1036), generates and
// applies a Householder reflector (dlarfg/dlarf, :845-862) and downdates the
// norms with Drmac's LAWN 176 rule, recomputing them on cancellation
// (:864-871, :912-986).  Only the pivot sequence leaves this step: V is
// discarded and the swaps of A, Y and the labels are composed into one
// permutation that a gather kernel applies afterwards.
//
// Two kernels: one keeps the columns in registers and exchanges tagged words
// (skinny_qrp_reg_kernel, below); what does not fit it takes the one described
// here.  The N columns are split into contiguous ranges, one range per
// CTA (one CTA per SM), and a range stays in that CTA's shared memory for all
// b stages (138 x 108 doubles = 119 KB at N = 16384, nb = 128), falling back
// to an L2-resident global copy when it does not fit.  A column never changes
// owner, so swaps are bookkeeping: each CTA tracks the current position of
// each of its columns.  Per stage there is ONE grid barrier: each CTA publishes
// its best candidate (norm, position) together with that column's entries, and
// after the barrier every CTA picks the same winner (largest norm, lowest
// position on ties -- BLAS idamax's first-maximum rule) and builds the
// reflector from the published column itself, so no second exchange is needed.
#include "hq_common.cuh"

namespace {

constexpr int NT = 256;
constexpr int NWARP = NT / 32;
constexpr int HDR = 4;                // record header: norm, position, column, spare

struct SkArgs {
  int mY, N, b;
  const double* Y;
  int ldy;
  double* Xg;  // global working copy (global mode)
  int ldxg;
  int smem_mode;
  int nloc_max;
  int ldxs;
  int* pairs;
  int* npairs;
  int max_pairs;
  double* part;  // [2][P][rec]
  int rec;
  unsigned* bar;
  int* err;
  unsigned spin_limit;
};

// Candidate order: larger norm first, then lower position.
__device__ __forceinline__ bool better(double d1, int p1, double d2, int p2) {
  return d1 > d2 || (d1 == d2 && p1 < p2);
}

__global__ void __launch_bounds__(NT, 1) skinny_qrp_kernel(SkArgs a) {
  HQ_PDL_WAIT();
  extern __shared__ __align__(16) double smem[];
  const int P = gridDim.x, cta = blockIdx.x, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int mY = a.mY;
  const int c_lo = (int)((long long)cta * a.N / P);
  const int c_hi = (int)((long long)(cta + 1) * a.N / P);
  const int nloc = c_hi - c_lo;

  // Shared-memory carve-up.
  double* sX = smem;
  double* sd = sX + (a.smem_mode ? (size_t)a.nloc_max * a.ldxs : 0);
  double* se = sd + a.nloc_max;
  double* sv = se + a.nloc_max;       // reflector, HQ_MAX_MY
  double* sred = sv + HQ_MAX_MY;      // 2 * NT scratch
  int* spos = (int*)(sred + 2 * NT);  // nloc_max
  int* sint = spos + a.nloc_max;      // small ints
  __shared__ int s_flag;
  __shared__ double s_tau;
  __shared__ int s_win_pos, s_win_cta, s_win_col;

  double* X;
  int ldx;
  if (a.smem_mode) {
    X = sX;
    ldx = a.ldxs;
  } else {
    X = a.Xg + (size_t)c_lo * a.ldxg;
    ldx = a.ldxg;
  }

  // Load the range, initialise positions and full column norms.
  for (int c = warp; c < nloc; c += NWARP) {
    const double* src = a.Y + (size_t)(c_lo + c) * a.ldy;
    double* dst = X + (size_t)c * ldx;
    double q = 0.0;
    for (int r = lane; r < mY; r += 32) {
      const double v = src[r];
      dst[r] = v;
      q = fma(v, v, q);
    }
    q = hq_warp_sum(q);
    if (lane == 0) {
      sd[c] = sqrt(q);
      se[c] = sd[c];
      spos[c] = c_lo + c;
    }
  }
  __syncthreads();

  unsigned epoch = 0;
  // Publish this CTA's best candidate for stage s, entries from row s on.
  auto publish = [&](int s) {
    double bd = -2.0;
    int bp = 0x7fffffff, bc = -1;
    for (int c = tid; c < nloc; c += NT) {
      if (spos[c] < s) continue;
      double d = sd[c];
      if (d != d) d = -1.0;  // NaN never wins over a number
      if (better(d, spos[c], bd, bp)) { bd = d; bp = spos[c]; bc = c; }
    }
    // Block argmax.
    for (int o = 16; o > 0; o >>= 1) {
      const double od = __shfl_xor_sync(0xffffffffu, bd, o);
      const int op = __shfl_xor_sync(0xffffffffu, bp, o);
      const int oc = __shfl_xor_sync(0xffffffffu, bc, o);
      if (better(od, op, bd, bp)) { bd = od; bp = op; bc = oc; }
    }
    if (lane == 0) {
      sred[warp] = bd;
      sint[warp] = bp;
      sint[NWARP + warp] = bc;
    }
    __syncthreads();
    if (tid == 0) {
      for (int w = 1; w < NWARP; ++w)
        if (better(sred[w], sint[w], bd, bp)) { bd = sred[w]; bp = sint[w]; bc = sint[NWARP + w]; }
      sint[2 * NWARP] = bc;
      double* rec = a.part + ((size_t)((epoch + 1) & 1) * P + cta) * a.rec;
      rec[0] = bd;
      rec[1] = (double)bp;
      rec[2] = (double)(bc >= 0 ? c_lo + bc : -1);
    }
    __syncthreads();
    const int cbest = sint[2 * NWARP];
    if (cbest >= 0) {
      double* rec = a.part + ((size_t)((epoch + 1) & 1) * P + cta) * a.rec;
      const double* col = X + (size_t)cbest * ldx;
      for (int r = s + tid; r < mY; r += NT) rec[HDR + r] = col[r];
    }
  };

  publish(0);
  for (int s = 0; s < a.b; ++s) {
    ++epoch;
    if (!hq_grid_barrier(a.bar, a.err, epoch, a.spin_limit, &s_flag)) return;
    const double* recs = a.part + (size_t)(epoch & 1) * P * a.rec;

    // Winner: every CTA reduces the same records in the same way.
    if (warp == 0) {
      double bd = -3.0;
      int bp = 0x7fffffff, bcta = -1;
      for (int q = lane; q < P; q += 32) {
        const double d = hq_ldcg(recs + (size_t)q * a.rec);
        const int p = (int)hq_ldcg(recs + (size_t)q * a.rec + 1);
        if (d > -2.0 && better(d, p, bd, bp)) { bd = d; bp = p; bcta = q; }
      }
      for (int o = 16; o > 0; o >>= 1) {
        const double od = __shfl_xor_sync(0xffffffffu, bd, o);
        const int op = __shfl_xor_sync(0xffffffffu, bp, o);
        const int oq = __shfl_xor_sync(0xffffffffu, bcta, o);
        if (better(od, op, bd, bp)) { bd = od; bp = op; bcta = oq; }
      }
      if (lane == 0) {
        s_win_pos = bp;
        s_win_cta = bcta;
        s_win_col = bcta >= 0 ? (int)hq_ldcg(recs + (size_t)bcta * a.rec + 2) : -1;
      }
    }
    __syncthreads();
    const int wpos = s_win_pos, wcta = s_win_cta, wcol = s_win_col;
    if (wcta < 0) {  // no active column anywhere: cannot happen for b <= N
      if (tid == 0) atomicCAS(a.err, 0, HQ_ERR_BAD_SHAPE);
      return;
    }
    // Position bookkeeping for the swap of positions s and wpos.
    if (wpos != s) {
      for (int c = tid; c < nloc; c += NT)
        if (spos[c] == s) spos[c] = wpos;
    }
    __syncthreads();
    if (cta == wcta && tid == 0) spos[wcol - c_lo] = s;

    // Reflector from the published winner column (rows s..mY-1).
    const double* wrec = recs + (size_t)wcta * a.rec + HDR;
    for (int r = s + tid; r < mY; r += NT) sv[r] = hq_ldcg(wrec + r);
    __syncthreads();
    if (warp == 0) {
      double q = 0.0;
      for (int r = s + 1 + lane; r < mY; r += 32) q = fma(sv[r], sv[r], q);
      q = hq_warp_sum(q);
      if (lane == 0) {
        const HqReflector h = hq_make_reflector_sq(sv[s], q);
        s_tau = h.tau;
        sred[0] = h.scale;
      }
      __syncwarp();
      const double scale = sred[0];
      for (int r = s + 1 + lane; r < mY; r += 32) sv[r] *= scale;
      if (lane == 0) sv[s] = 1.0;
    }
    __syncthreads();
    if (s + 1 == a.b) break;  // the pivots are complete; V is discarded

    // Apply H = I - tau v v^T to every other active column and downdate its
    // norm.  One thread per column: the column's dot product, update, norm
    // test and (rare) norm recomputation need no cross-lane reduction, and no
    // FP64 work is repeated across lanes.
    const double tau = s_tau;
    for (int c = tid; c < nloc; c += NT) {
      if (spos[c] <= s) continue;
      double* x = X + (size_t)c * ldx;
      double w0 = x[s], w1 = 0.0, w2 = 0.0, w3 = 0.0;
      int r = s + 1;
      for (; r + 3 < mY; r += 4) {
        w0 = fma(sv[r], x[r], w0);
        w1 = fma(sv[r + 1], x[r + 1], w1);
        w2 = fma(sv[r + 2], x[r + 2], w2);
        w3 = fma(sv[r + 3], x[r + 3], w3);
      }
      for (; r < mY; ++r) w0 = fma(sv[r], x[r], w0);
      const double g = -tau * ((w0 + w1) + (w2 + w3));
      const double rs = x[s] + g;
      x[s] = rs;
      for (r = s + 1; r < mY; ++r) x[r] = fma(g, sv[r], x[r]);
      double dc = sd[c];
      if (dc != 0.0) {
        double t1 = fabs(rs) / dc;
        t1 = (1.0 + t1) * (1.0 - t1);
        if (0.0 > t1) t1 = 0.0;
        const double ratio = dc / se[c];
        const double t2 = t1 * ratio * ratio;
        if (t2 <= HQ_TOL3Z) {
          double q0 = 0.0, q1 = 0.0;
          for (r = s + 1; r + 1 < mY; r += 2) {
            q0 = fma(x[r], x[r], q0);
            q1 = fma(x[r + 1], x[r + 1], q1);
          }
          if (r < mY) q0 = fma(x[r], x[r], q0);
          dc = (mY - s - 1 > 0) ? sqrt(q0 + q1) : 0.0;
          sd[c] = dc;
          se[c] = dc;
        } else {
          sd[c] = dc * sqrt(t1);
        }
      }
    }
    __syncthreads();
    publish(s + 1);
  }

  // Final permutation as (dst, src) pairs for the columns that moved.
  for (int c = tid; c < nloc; c += NT) {
    if (spos[c] != c_lo + c) {
      const int i = atomicAdd(a.npairs, 1);
      if (i < a.max_pairs) {
        a.pairs[2 * i] = spos[c];
        a.pairs[2 * i + 1] = c_lo + c;
      } else {
        atomicCAS(a.err, 0, HQ_ERR_BAD_SHAPE);  // only after an aborted run
      }
    }
  }
}

// Register-resident variant, used when mY and the columns per CTA fit it (see
// launch_reg): LPC adjacent lanes hold one sketch column, rows interleaved
// (lane l has rows LPC t + l, t < RPT), so a stage reads its columns from
// registers; the reflector is staged in shared memory in the same order and
// read 16 bytes at a time, whole chunks of 16 rows above the stage's row being
// jumped over.  Scalar work is done once, not by every thread: one warp builds
// the reflector, one thread per column downdates its norm, and pivot
// candidates compare integer keys.
//
// What bounds a stage is the latency of agreeing on the pivot, so the exchange
// has neither a fence nor a counter.  A CTA writes its best candidate -- norm
// key and position, once for every CTA -- in words that carry the stage's tag
// next to the value (128- and 64-bit scalar stores, which are single-copy
// atomic), and then, as if it had won, the reflector of the candidate's column:
// its sums and square root are off the path everyone waits on, and a loser's
// cost nothing but an idle warp.  A warp of its own in each CTA polls the
// CTA's own copy of the P headers, picks the winner and polls its reflector: a
// word whose tag matches holds this stage's value, so nothing has to be
// ordered before anything else.  (With one copy of the headers for all, the
// polls of 128 CTAs queue up at the few cache lines that the headers are
// written to: 3500 clocks in that wait alone, against 1400 for 24 CTAs.)
// Headers and reflectors alternate between two buffers.  A CTA overwrites a
// buffer at stage s + 2 after it has seen every CTA's header of stage s + 1,
// which each wrote after it had read stage s.
// Tags grow over all launches of a call and the area is zeroed once per call.
//
// Measured on GB300 a stage, against two lanes a column and a counter barrier
// (release add and spin, then all headers, then the column) -> with the
// reflector built by everyone after the exchange -> this: FP32, 138 rows,
// 16384 columns 5.5 -> 3.5 -> 3.2 us, 3000 columns 5.2 -> 2.8 -> 2.6; FP64, 74
// rows, 2000 columns 9.7 -> 4.2 -> 3.5.
//
// T is the arithmetic of the reflector applications (the bulk of the FP64
// work): double for the plain path, float for the mixed path, whose sketch is
// formed from two-digit BF16 operands (~16 significant bits) and only steers
// pivots.  Norms, their LAWN 176 downdate and recomputation, and in the plain
// path the reflector scalars are FP64.  Norms are kept squared:
// d^2 <- d^2 - r^2, recomputed when d^2 - r^2 <= tol3z e^2 -- LAPACK's test
// t2 = (d^2 - r^2) / e^2 <= tol3z without its two divisions and square root
// (~2.2k clocks of FP64 a stage on this GPU); the argmax of d^2 is the argmax
// of d.  In FP32 a column's dot product is four chains (rows modulo 4) added
// as (0 + 2) + (1 + 3), whatever the launch shape.
struct RegArgs {
  int mY, N, b;
  const double* Y;
  int ldy;
  int* pairs;
  int* npairs;
  int max_pairs;
  unsigned char* hdrs;  // [2][MAX_P copies][MAX_P] 16-byte headers
  unsigned char* recs;  // [2][MAX_P] reflectors
  unsigned tag0;        // stage s's tag is tag0 + s + 1
  int* err;
  unsigned spin_limit;
};
constexpr int MAX_P = 160;               // CTAs
constexpr int HDR_LANE = MAX_P / 32;     // headers per polling lane

// One entry of a published column and its tag: 8 bytes in FP32, 16 in FP64.
template <typename T>
struct Tagged;
template <>
struct Tagged<float> {
  static constexpr int BYTES = 8;
  static __device__ __forceinline__ void put(unsigned char* p, float x, unsigned tag) {
    hq_st_word(p, ((unsigned long long)tag << 32) | __float_as_uint(x));
  }
  static __device__ __forceinline__ bool get(const unsigned char* p, unsigned tag, float& x) {
    unsigned long long v;
    hq_ld_word(p, v);
    x = __uint_as_float((unsigned)v);
    return (unsigned)(v >> 32) == tag;
  }
};
template <>
struct Tagged<double> {
  static constexpr int BYTES = 16;
  static __device__ __forceinline__ void put(unsigned char* p, double x, unsigned tag) {
    hq_st_word(p, (unsigned long long)__double_as_longlong(x), tag);
  }
  static __device__ __forceinline__ bool get(const unsigned char* p, unsigned tag, double& x) {
    unsigned long long lo, hi;
    hq_ld_word(p, lo, hi);
    x = __longlong_as_double((long long)lo);
    return hi == tag;
  }
};

__device__ __forceinline__ bool better_key(long long k1, int p1, long long k2, int p2) {
  return k1 > k2 || (k1 == k2 && p1 < p2);
}

// Best (key, position) of the warp in every lane: largest key, then lowest
// position; keys are >= -3.  Three integer reductions instead of five rounds
// of shuffles.
__device__ __forceinline__ void warp_best(long long& key, int& pos) {
  const unsigned long long u = (unsigned long long)(key + 4);
  const unsigned hi = (unsigned)(u >> 32);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = hi == mh ? (unsigned)u : 0u;
  const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
  const bool mine = hi == mh && (unsigned)u == ml;
  pos = __reduce_min_sync(0xffffffffu, mine ? pos : 0x7fffffff);
  key = (long long)(((unsigned long long)mh << 32) | ml) - 4;
}

// case i of a switch over 16-row chunks: do it, and fall through to the next.
#define HQ_CHUNKS(DO)                                                                        \
  case 0: DO(0) case 1: DO(1) case 2: DO(2) case 3: DO(3) case 4: DO(4) case 5: DO(5)        \
  case 6: DO(6) case 7: DO(7) case 8: DO(8) case 9: DO(9) case 10: DO(10) case 11: DO(11)    \
  case 12: DO(12) case 13: DO(13) case 14: DO(14) case 15: DO(15)

template <int CNT, int RPT, int LPC, typename T>
__global__ void __launch_bounds__(CNT + 32, 1) skinny_qrp_reg_kernel(RegArgs a) {
  HQ_PDL_WAIT();
  constexpr int POLLER = CNT / 32;     // the warp that exchanges; it holds no columns
  constexpr bool F32 = sizeof(T) == 4;
  constexpr int NC = CNT / LPC;        // columns per CTA
  constexpr int CE = 16 / LPC;         // entries of a lane per 16-row chunk
  constexpr int NCH = RPT / CE;
  constexpr int STR = RPT + 16 / (int)sizeof(T) * ((RPT * (int)sizeof(T)) % 128 == 0);  // no bank conflicts
  constexpr int RLANE = (LPC * RPT + 31) / 32;  // rows per lane of one warp
  // The reflector stays in registers between its two uses where they suffice.
  constexpr bool KEEP = CNT <= 256 && RPT * (int)sizeof(T) <= 144;
  static_assert(RPT % CE == 0 && CE * sizeof(T) % 16 == 0 && NCH <= 16, "chunks");
  static_assert(NC % 32 == 0, "downdating threads fill whole warps");
  __shared__ __align__(16) T sv[LPC * STR];  // the reflector v, lane-major
  __shared__ T sraw[LPC * RPT];              // the candidate's column, by rows
  __shared__ long long s_bk[NC / 32];
  __shared__ int s_bp[NC / 32];
  __shared__ int sflag[NC];
  __shared__ T srs[NC];        // the columns' new entries of row s
  __shared__ double snrm[NC];  // (re)computed squared norms
  __shared__ int s_win_pos, s_dead;
  __shared__ T s_tau;
  const int P = gridDim.x, cta = blockIdx.x, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5, l = lane & (LPC - 1);
  const int mY = a.mY;
  const int c_lo = (int)((long long)cta * a.N / P);
  const int c_hi = (int)((long long)(cta + 1) * a.N / P);
  const int nloc = c_hi - c_lo;
  const int c = tid / LPC;  // this lane group's local column
  const bool have = c < nloc;
  const size_t rec_bytes = (size_t)mY * Tagged<T>::BYTES;

  T x[RPT];
  // FP32 registers hold the column times 2^-ec (ec from its norm), so FP32's
  // range never limits the input; 2^ec converts back (exact).
  int ec = 0;
  {
    const double* src = a.Y + (size_t)(c_lo + (have ? c : 0)) * a.ldy;
    double q = 0.0;
#pragma unroll
    for (int t = 0; t < RPT; ++t) {
      const int r = LPC * t + l;
      const double y = (have && r < mY) ? src[r] : 0.0;
      if constexpr (!F32) x[t] = y;
      q = fma(y, y, q);
    }
#pragma unroll
    for (int o = LPC / 2; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    if constexpr (F32) {
      int eq = (int)((__double_as_longlong(q) >> 52) & 0x7FF) - 1023;  // q >= 0
      if (eq < -1022) eq = -1022;
      ec = eq / 2;
      const double sc = __longlong_as_double((long long)(1023 - ec) << 52);
#pragma unroll
      for (int t = 0; t < RPT; ++t) {
        const int r = LPC * t + l;
        x[t] = (have && r < mY) ? (T)(src[r] * sc) : (T)0;
      }
    }
    if (l == 0 && c < NC) {
      snrm[c] = q;
      sflag[c] = ec;
    }
  }
  for (int r = tid; r < LPC * STR; r += CNT + 32) sv[r] = (T)0;
  if (tid == 0) s_dead = 0;
  __syncthreads();

  int mypos = have ? c_lo + c : -1;  // position of the group's column
  const bool dd = tid < nloc;        // this thread downdates column tid
  int dpos = dd ? c_lo + tid : -1;
  double dn = dd ? snrm[tid] : 0.0;
  double thr = HQ_TOL3Z * dn;  // recompute at or below this
  const double unscale = __longlong_as_double((long long)(1023 + (tid < NC ? sflag[tid] : 0)) << 52);

  // This warp's best candidate for stage s (warps of downdating threads).
  auto local_best = [&](int s) {
    if (tid < NC) {
      long long k = -2;
      int p = 0x7fffffff;
      if (dd && dpos >= s) {
        k = hq_norm_key(dn);
        p = dpos;
      }
      warp_best(k, p);
      if (lane == 0) {
        s_bk[warp] = k;
        s_bp[warp] = p;
      }
    }
  };
  // Write this CTA's best candidate for stage s (s_bk and s_bp complete) and
  // then the reflector it would give, by the warp that holds the column (a
  // header alone, by warp 0, when no column is active).  Entry s of the record
  // is tau, the entries below v's.
  auto publish = [&](int s) {
    long long k = s_bk[0];
    int p = s_bp[0];
#pragma unroll
    for (int w = 1; w < NC / 32; ++w)
      if (better_key(s_bk[w], s_bp[w], k, p)) { k = s_bk[w]; p = s_bp[w]; }
    const unsigned tag = a.tag0 + (unsigned)s + 1u;
    const bool mine = k > -2 && have && mypos == p;
    const bool here = __any_sync(0xffffffffu, mine);
    if (!here && !(k <= -2 && warp == 0)) return;
    unsigned char* h = a.hdrs + ((size_t)(s & 1) * MAX_P * MAX_P + cta) * 16;
    const unsigned long long w1 = ((unsigned long long)tag << 32) | (unsigned)p;
#pragma unroll
    for (int j = 0; j < HDR_LANE; ++j) {
      const int q = lane + 32 * j;
      if (32 * j < P && q < P) hq_st_word(h + (size_t)q * MAX_P * 16, (unsigned long long)k, w1);
    }
    if (!here) return;
    if (mine) {
#pragma unroll
      for (int t = 0; t < RPT; ++t) sraw[LPC * t + l] = x[t];
    }
    __syncwarp();
    // Tail norm, reflector, v = [1; scale * tail].  In FP32 the reflector of
    // the scaled column is built directly (it does not depend on the column's
    // scale): beta = -sign(alpha) sqrt(alpha^2 + q), tau = (beta - alpha) /
    // beta, scale = 1 / (alpha - beta); tau = 0 for a zero tail.
    const T al = sraw[s];
    T z[RLANE], q = (T)0;
#pragma unroll
    for (int i = 0; i < RLANE; ++i) {
      const int r = s + 1 + lane + 32 * i;
      z[i] = r < mY ? sraw[r] : (T)0;
    }
#pragma unroll
    for (int i = 0; i < RLANE; ++i)
      if (s + 1 + 32 * i < mY) q = fma(z[i], z[i], q);
    q = hq_warp_sum(q);
    T tau, scale;
    if constexpr (F32) {
      tau = 0.f;
      scale = 0.f;
      if (q > 0.f) {
        const float beta = -copysignf(sqrtf(fmaf(al, al, q)), al);
        tau = (beta - al) / beta;
        scale = 1.f / (al - beta);
      }
    } else {
      const HqReflector hr = hq_make_reflector_sq(al, q);
      tau = hr.tau;
      scale = hr.scale;
    }
    unsigned char* rec = a.recs + ((size_t)(s & 1) * MAX_P + cta) * rec_bytes;
    if (lane == 0) Tagged<T>::put(rec + (size_t)s * Tagged<T>::BYTES, tau, tag);
#pragma unroll
    for (int i = 0; i < RLANE; ++i) {
      const int r = s + 1 + lane + 32 * i;
      if (r < mY) Tagged<T>::put(rec + (size_t)r * Tagged<T>::BYTES, scale * z[i], tag);
    }
  };

  local_best(0);
  __syncthreads();
  publish(0);
  for (int s = 0; s < a.b; ++s) {
    if (warp == POLLER) {
      const unsigned tag = a.tag0 + (unsigned)s + 1u;
      // Winner: every CTA reduces the same headers in the same way.
      const unsigned char* h0 = a.hdrs + ((size_t)(s & 1) * MAX_P + cta) * MAX_P * 16;
      long long kk[HDR_LANE];
      int pp[HDR_LANE];
      bool ok = false;
      unsigned it = 0;
      for (;;) {
        ok = true;
#pragma unroll
        for (int j = 0; j < HDR_LANE; ++j) {
          const int q = lane + 32 * j;
          kk[j] = -3;
          pp[j] = 0x7fffffff;
          if (32 * j < P && q < P) {
            unsigned long long k0, w;
            hq_ld_word(h0 + (size_t)q * 16, k0, w);
            kk[j] = (long long)k0;
            pp[j] = (int)(unsigned)w;
            ok = ok && (unsigned)(w >> 32) == tag;
          }
        }
        ok = __all_sync(0xffffffffu, ok);
        if (ok || ++it >= a.spin_limit) break;
        if ((it & 15u) == 0u && __any_sync(0xffffffffu, hq_ld_volatile(a.err) != 0)) break;
      }
      long long bk = kk[0];
      int bp = pp[0], bq = lane;
#pragma unroll
      for (int j = 1; j < HDR_LANE; ++j)
        if (better_key(kk[j], pp[j], bk, bp)) {
          bk = kk[j];
          bp = pp[j];
          bq = lane + 32 * j;
        }
      long long wk = bk;
      int wp = bp;
      warp_best(wk, wp);
      const unsigned who = __ballot_sync(0xffffffffu, bk == wk && bp == wp);
      const int wcta = __shfl_sync(0xffffffffu, bq, __ffs((int)who) - 1);
      const bool none = ok && wk <= -2;  // no active column anywhere: cannot happen for b <= N
      // The winner's tau, and v in rows s + 1 + lane + 32 i.
      T tau = (T)0, z[RLANE];
      if (ok && !none) {
        const unsigned char* rec = a.recs + ((size_t)(s & 1) * MAX_P + wcta) * rec_bytes;
        for (;;) {
          bool got = Tagged<T>::get(rec + (size_t)s * Tagged<T>::BYTES, tag, tau);
#pragma unroll
          for (int i = 0; i < RLANE; ++i) {
            const int r = s + 1 + lane + 32 * i;
            z[i] = (T)0;
            if (r < mY) got = Tagged<T>::get(rec + (size_t)r * Tagged<T>::BYTES, tag, z[i]) && got;
          }
          ok = __all_sync(0xffffffffu, got);
          if (ok || ++it >= a.spin_limit) break;
          if ((it & 15u) == 0u && __any_sync(0xffffffffu, hq_ld_volatile(a.err) != 0)) break;
        }
      }
      if (!ok || none) {
        if (lane == 0) {
          atomicCAS(a.err, 0, none ? HQ_ERR_BAD_SHAPE : HQ_ERR_BARRIER_TIMEOUT);
          s_dead = 1;
        }
      } else {
        if (lane == 0) s_win_pos = wp;
        auto put = [&](int r, T v) { sv[(r & (LPC - 1)) * STR + r / LPC] = v; };
#pragma unroll
        for (int i = 0; i < RLANE; ++i) {
          const int r = s + 1 + lane + 32 * i;
          if (r < mY) put(r, z[i]);
        }
        if (lane == 0) {
          s_tau = tau;
          put(s, (T)1);
          if (s > 0) put(s - 1, (T)0);
        }
      }
    }
    __syncthreads();
    if (s_dead != 0) return;  // an exchange gave up; the other CTAs see the error word
    // Position bookkeeping for the swap of positions s and wpos (columns are
    // never moved).
    const int wpos = s_win_pos;
    if (have) mypos = mypos == wpos ? s : (mypos == s ? wpos : mypos);
    if (dd) dpos = dpos == wpos ? s : (dpos == s ? wpos : dpos);
    if (s + 1 == a.b) break;  // the pivots are complete; V is discarded

    // Apply H = I - tau v v^T to the group's column (if still active); the
    // new entry of row s goes to srs for the downdate.
    const bool active = have && mypos > s;
    if (__any_sync(0xffffffffu, active)) {
      const int sch = s >> 4;  // first chunk holding a row >= s
      const T* vl = sv + l * STR;
      __align__(16) T v[RPT];
      auto load_chunk = [&](int ch) {
#pragma unroll
        for (int j = 0; j < CE * (int)sizeof(T) / 16; ++j)
          reinterpret_cast<int4*>(v + CE * ch)[j] = reinterpret_cast<const int4*>(vl + CE * ch)[j];
      };
      T w = (T)0;
#define HQ_DOT(I)                                                                   \
  if constexpr (I < NCH) {                                                          \
    load_chunk(I);                                                                  \
    _Pragma("unroll") for (int j = 0; j < CE; ++j) w = fma(v[CE * I + j], x[CE * I + j], w); \
  }
      switch (sch) { HQ_CHUNKS(HQ_DOT) }
#undef HQ_DOT
#pragma unroll
      for (int o = LPC / 2; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
      if (active) {
        const T g = (T)(-s_tau) * w;
        T xs = (T)0;  // the new entry of row s, in the lane that holds it
        const int ts = s / LPC;
#define HQ_UPD(I)                                                                    \
  if constexpr (I < NCH) {                                                           \
    if constexpr (!KEEP) load_chunk(I);                                              \
    _Pragma("unroll") for (int j = 0; j < CE; ++j)                                   \
      x[CE * I + j] = fma(g, v[CE * I + j], x[CE * I + j]);                          \
  }
        switch (sch) { HQ_CHUNKS(HQ_UPD) }
#undef HQ_UPD
#define HQ_PICK(I)                                                                  \
  if constexpr (I < NCH) {                                                          \
    _Pragma("unroll") for (int j = 0; j < CE; ++j) if (CE * I + j == ts) xs = x[CE * I + j]; \
  }                                                                                 \
  break;
        switch (sch) { HQ_CHUNKS(HQ_PICK) }
#undef HQ_PICK
        if (l == (s & (LPC - 1))) srs[c] = xs;
      }
    }
    __syncthreads();
    // Norm downdate, one thread per column (LAWN 176 on squared norms); flagged
    // norms are recomputed from the registers.
    int flag = 0;
    if (dd && dpos > s && dn != 0.0) {
      const double r = F32 ? (double)srs[tid] * unscale : (double)srs[tid];
      const double nd = fma(-r, r, dn);
      if (hq_norm_cancelled(nd, thr)) flag = 1;
      else dn = nd;
    }
    if (tid < NC) sflag[tid] = flag;
    local_best(s + 1);
    if (__syncthreads_or(flag)) {
      if (active && sflag[c]) {
        T f = (T)0;
#pragma unroll
        for (int t = 0; t < RPT; ++t)
          if (LPC * t + l > s) f = fma(x[t], x[t], f);
        const unsigned gmask = ((1u << LPC) - 1u) << (lane & ~(LPC - 1));
#pragma unroll
        for (int o = LPC / 2; o > 0; o >>= 1) f += __shfl_xor_sync(gmask, f, o);
        if (l == 0) {
          const double up = __longlong_as_double((long long)(1023 + ec) << 52);
          snrm[c] = mY - s - 1 > 0 ? (double)f * (up * up) : 0.0;
        }
      }
      __syncthreads();
      if (flag) {
        dn = snrm[tid];
        thr = HQ_TOL3Z * dn;
      }
      local_best(s + 1);
      __syncthreads();
    }
    publish(s + 1);
  }

  // Final permutation as (dst, src) pairs for the columns that moved.
  if (have && l == 0 && mypos != c_lo + c) {
    const int i = atomicAdd(a.npairs, 1);
    if (i < a.max_pairs) {
      a.pairs[2 * i] = mypos;
      a.pairs[2 * i + 1] = c_lo + c;
    } else {
      atomicCAS(a.err, 0, HQ_ERR_BAD_SHAPE);  // only after an aborted run
    }
  }
}
#undef HQ_CHUNKS

// A launch shape of the register kernel: entry, threads, columns a CTA holds,
// rows it takes.
struct RegShape {
  const void* fn;
  int threads, cols, rows;
};
template <int CNT, int RPT, int LPC, typename T>
RegShape reg_shape() {
  return {(const void*)skinny_qrp_reg_kernel<CNT, RPT, LPC, T>, CNT, CNT / LPC, LPC * RPT};
}

int skinny_grid(const hq_device_info* dev, int N) {
  int p = (N + 15) / 16;
  if (p > dev->num_sms) p = dev->num_sms;
  return p < 1 ? 1 : p;
}

}  // namespace

extern "C" size_t hq_skinny_part_elems(const hq_device_info* dev, int mY) {
  const int rec = HDR + ((mY + 1) & ~1);
  return (size_t)2 * dev->num_sms * rec;
}

// The register kernel's exchange area: fixed places for MAX_P CTAs, so a word
// never changes its meaning from one launch of a call to the next.
extern "C" size_t hq_skinny_xch_bytes(int mY, int fp32) {
  return (size_t)2 * MAX_P * (MAX_P * 16 + (size_t)mY * (fp32 ? 8 : 16));
}

// The register kernel, if a shape holds the sketch; cudaErrorNotSupported
// otherwise.
static int launch_reg(cudaStream_t stream, const hq_device_info* dev, const SkArgs& s, void* xch,
                      unsigned* tag, int fp32) {
  // Shapes by rows and columns per CTA, the first that holds the sketch on one
  // CTA per SM.  FP32: four lanes a column, 64 columns a CTA, else 128 (3000
  // columns: 128 a CTA 9.3 ms a factorization, 64 8.2, 32 8.2).  FP64: eight
  // lanes and 32 columns, else four and 64, or two and 128.
  constexpr int N_SHAPES = 14, F32_SHAPES = 6;
  static const RegShape shapes[N_SHAPES] = {
      reg_shape<256, 20, 4, float>(),  reg_shape<256, 36, 4, float>(),
      reg_shape<256, 64, 4, float>(),  reg_shape<512, 20, 4, float>(),
      reg_shape<512, 36, 4, float>(),  reg_shape<512, 64, 4, float>(),
      reg_shape<256, 10, 8, double>(), reg_shape<256, 18, 8, double>(),
      reg_shape<256, 32, 8, double>(), reg_shape<256, 20, 4, double>(),
      reg_shape<256, 36, 4, double>(), reg_shape<256, 64, 4, double>(),
      reg_shape<256, 40, 2, double>(), reg_shape<256, 72, 2, double>()};
  const int max_p = dev->num_sms < MAX_P ? dev->num_sms : MAX_P;
  for (int i = fp32 ? 0 : F32_SHAPES; i < (fp32 ? F32_SHAPES : N_SHAPES); ++i) {
    const RegShape& sh = shapes[i];
    const int hold = (s.N + sh.cols - 1) / sh.cols;
    if (s.mY > sh.rows || hold > max_p) continue;
    // CTAs: in FP32 as few as hold the columns (the stage is latency, and
    // fewer headers are polled); in FP64 one per 16 columns, up to one per
    // SM: the FP64 work of its columns is what a stage costs a CTA (2000
    // columns of 74 rows: 16 a CTA 9.1 ms a factorization, 32 9.8).
    int P = fp32 ? hold : (s.N + 15) / 16;
    if (P > max_p) P = max_p;
    if (P < hold) P = hold;
    RegArgs a;
    a.mY = s.mY;
    a.N = s.N;
    a.b = s.b;
    a.Y = s.Y;
    a.ldy = s.ldy;
    a.pairs = s.pairs;
    a.npairs = s.npairs;
    a.max_pairs = s.max_pairs;
    a.hdrs = static_cast<unsigned char*>(xch);
    a.recs = a.hdrs + (size_t)2 * MAX_P * MAX_P * 16;
    a.tag0 = *tag;
    *tag += (unsigned)s.b;
    a.err = s.err;
    a.spin_limit = s.spin_limit;
    const int z = hq_zero_words(stream, s.npairs, 1, nullptr, 0);
    if (z) return z;
    void* args[] = {&a};
    const cudaError_t e = hq_launch_coop(sh.fn, dim3(P), dim3(sh.threads + 32), args, 0, stream);
    hq_count_launches(1);
    return (int)e;
  }
  return (int)cudaErrorNotSupported;
}

extern "C" int hq_skinny_qrp(cudaStream_t stream, const hq_device_info* dev, int mY, int N,
                             int b, const double* Y, int ldy, double* V, int ldv, int* pairs,
                             int* npairs, double* part, size_t part_elems, void* xch,
                             unsigned* tag, unsigned* bar, int* err, unsigned spin_limit,
                             int fp32) {
  if (mY > HQ_MAX_MY || b > mY || b > N || b <= 0) return (int)cudaErrorInvalidValue;
  SkArgs a;
  a.mY = mY;
  a.N = N;
  a.b = b;
  a.Y = Y;
  a.ldy = ldy;
  a.Xg = V;
  a.ldxg = ldv;
  a.pairs = pairs;
  a.npairs = npairs;
  a.max_pairs = 2 * b;
  a.part = part;
  a.rec = HDR + ((mY + 1) & ~1);
  a.bar = bar;
  a.err = err;
  a.spin_limit = spin_limit;
  const int reg = launch_reg(stream, dev, a, xch, tag, fp32);
  if (reg != (int)cudaErrorNotSupported) return reg;
  // More columns than the registers of the grid hold: the shared-memory
  // kernel, one CTA per 16 columns up to one per SM.
  const int P = skinny_grid(dev, N);
  if ((size_t)2 * P * a.rec > part_elems) return (int)cudaErrorInvalidValue;
  a.nloc_max = (N + P - 1) / P;
  a.ldxs = mY | 1;
  const size_t fixed = sizeof(double) * (2 * (size_t)a.nloc_max + HQ_MAX_MY + 2 * NT) +
                       sizeof(int) * ((size_t)a.nloc_max + 4 * NWARP + 8);
  const size_t with_x = fixed + sizeof(double) * (size_t)a.nloc_max * a.ldxs;
  size_t smem;
  if (with_x <= dev->smem_optin) {
    a.smem_mode = 1;
    smem = with_x;
  } else {
    a.smem_mode = 0;
    smem = fixed;
    if (V == nullptr || smem > dev->smem_optin) return (int)cudaErrorInvalidValue;
  }
  const int z = hq_zero_words(stream, bar, 1, npairs, 1);
  if (z) return z;
  void* args[] = {&a};
  cudaError_t e = cudaFuncSetAttribute(skinny_qrp_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  e = hq_launch_coop((const void*)skinny_qrp_kernel, dim3(P), dim3(NT), args, smem, stream);
  hq_count_launches(1);
  return (int)e;
}
