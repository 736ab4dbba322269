// qrp_wide.cu -- pivoted Householder QR of a matrix of at most 1024 rows (any
// number of columns), one cooperative kernel.
//
// Reference: the small-matrix branch of dgeqp4
// (lapack_compatible_sources/NoFLA_HQRRP_WY_blk_var4.c:189-199) hands every
// matrix with min(m, n) < 1000 to LAPACK's dgeqpf or dgeqp3, whatever n is.
// Both pick, at stage s, the remaining column of largest partial norm (first
// maximum in column order, like idamax), swap it into position s (the norms
// follow their column), apply dlarfg/dlarf, and downdate the partial norms
// with the LAWN 176 test, recomputing a norm when cancellation is detected
// (the same rule as the reference's own QRPmod, :774-886 and :912-986).
//
// GB300 layout: the columns are dealt out cyclically, one CTA per SM at most; a
// column never moves and never leaves its CTA, staged in shared memory when
// the CTA's columns fit.  Swaps are bookkeeping -- each CTA keeps the position
// of its own columns -- and the final order is applied afterwards by one
// gather of the displaced columns (at most two per stage).  Per stage there is
// one exchange.  One warp of every CTA writes the CTA's best candidate's norm
// and position, once for every CTA, in words that carry the stage's number,
// and polls the others' (as in pivot selection, qrp_skinny.cu).  The other
// warps meanwhile build the candidate's reflector and write it out behind a
// flag, as if it had won: its square root and sums are then off the path that
// everyone waits on, and a loser's cost nothing but idle units.  Each CTA takes
// the winner's reflector and updates its columns by whole warps, so the norm
// downdate (squared norms) and the rare recomputation need no communication.
//
// The row-partitioned panel kernel (qrp_panel.cu) takes more than 1024 rows,
// and up to 512 columns of any number of rows, where it is the faster one
// (a stage here costs ~7 us whatever the width: 641 x 481 3.5 ms there, 3.6
// here; 999 x 998 11.4 and 7.9).  Measured on GB300 against one column range a
// CTA, a counter barrier and the reflector built by everyone after the
// exchange: 300 x 2000 5.6 -> 2.3 ms, 100 x 3000 2.6 -> 0.8, 999 x 5000 39.6 ->
// 17.8.
#include "hq_columns.cuh"

namespace {

constexpr int WT = 512;
constexpr int WW = WT / 32;
constexpr int ND = 128, NDW = ND / 32;  // threads with one FP64 value each: a warp per quarter
constexpr int MAX_P = 160, HDR_LANE = MAX_P / 32;

struct WdArgs {
  int m, n, ns;
  double* A;
  int lda;
  double* tau;
  int* pairs;          // out: (dst, src) pairs of the final order
  int* npairs;         // out: their count (zeroed by the launcher)
  unsigned char* hdrs; // [2][P copies][P] 16-byte headers
  unsigned long long* flags;  // [2][P] the tag of the reflector in
  double* cols;               // [2][P][m + 1] reflectors, then tau
  int* err;
  unsigned spin_limit;
  int cpc;             // most columns any CTA owns
  int staged;
  double* state;       // the columns' norms and positions, where they outgrow shared memory
};

__global__ void __launch_bounds__(WT, 1) wide_qrp_kernel(WdArgs a) {
  HQ_PDL_WAIT();
  extern __shared__ __align__(16) double wsm[];
  const int P = gridDim.x, cta = blockIdx.x, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int m = a.m, nl = (a.n - cta + P - 1) / P;
  double* sc = wsm;             // [m] the reflector of this CTA's candidate
  double* sv = sc + m;          // [m] the winner's, when it is another CTA's
  double* sd = a.state ? a.state + (size_t)4 * a.cpc * cta : sv + m;  // [cpc] squared partial norms of the CTA's columns
  double* sthr = sd + a.cpc;    // [cpc] recompute at or below
  double* srs = sthr + a.cpc;   // [cpc] the stage's new entries of row s
  int* spos = (int*)(srs + a.cpc);  // [cpc] positions (<= s: factored)
  int* sact = spos + a.cpc;     // [cpc] columns not yet factored
  double* sX = sv + m + 4 * a.cpc;  // [cpc][m] the columns, when staged
  __shared__ double s_red[NDW];
  __shared__ long long s_bk[NDW], s_at[NDW];
  __shared__ long long s_k, s_w;
  __shared__ double s_tau, s_scale, s_beta;
  __shared__ int s_wpos, s_wcta, s_bad;

  auto colp = [&](int q) {
    return a.staged ? sX + (size_t)q * m : a.A + (size_t)(cta + P * q) * a.lda;
  };
  for (int q = warp; q < nl; q += WW) {
    const double* g = a.A + (size_t)(cta + P * q) * a.lda;
    double* x = colp(q);
    double t = 0.0;
#pragma unroll 4
    for (int i = lane; i < m; i += 32) {
      const double v = g[i];
      if (a.staged) x[i] = v;
      t = fma(v, v, t);
    }
    t = hq_warp_sum(t);
    if (lane == 0) {
      sd[q] = t;
      sthr[q] = HQ_TOL3Z * t;
      spos[q] = cta + P * q;
      sact[q] = q;
    }
  }
  if (tid == 0) s_bad = 0;
  __syncthreads();
  int cnt = nl;
  auto best_of_columns = [&]() {
    if (tid >= ND) return;
    long long k = -2, at = 0x7fffffffLL << 32;
    for (int j = tid; j < cnt; j += ND) {
      const int q = sact[j];
      const long long kj = hq_norm_key(sd[q]);
      const long long aj = ((long long)spos[q] << 32) | (unsigned)q;
      if (better(kj, aj, k, at)) { k = kj; at = aj; }
    }
    warp_best(k, at, s_bk + warp, s_at + warp);
  };
  best_of_columns();
  __syncthreads();
  // The warps that build reflectors (all but warp 0).
  auto worker_barrier = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(WT - 32) : "memory"); };

  for (int s = 0; s < a.ns; ++s) {
    // 1. This CTA's candidate; the winner of all.
    const unsigned tag = (unsigned)s + 1u;
    long long bk = s_bk[0], at = s_at[0];
#pragma unroll
    for (int w = 1; w < NDW; ++w)
      if (better(s_bk[w], s_at[w], bk, at)) { bk = s_bk[w]; at = s_at[w]; }
    const int lq = (int)(unsigned)at;
    int wpos = (int)(at >> 32), wcta = cta;
    double* rec = a.cols + ((size_t)(s & 1) * P + cta) * (m + 1);
    if (warp == 0) {
      if (P > 1) {
        unsigned char* h = a.hdrs + ((size_t)(s & 1) * P * P + cta) * 16;
        const unsigned long long w1 = ((unsigned long long)tag << 32) | (unsigned)wpos;
#pragma unroll
        for (int j = 0; j < HDR_LANE; ++j) {
          const int q = lane + 32 * j;
          if (32 * j < P && q < P) hq_st_word(h + (size_t)q * P * 16, (unsigned long long)bk, w1);
        }
        const unsigned char* h0 = a.hdrs + ((size_t)(s & 1) * P + cta) * P * 16;
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
        if (ok) {
          long long k = kk[0], w = ((long long)pp[0] << 32) | (unsigned)lane;
#pragma unroll
          for (int j = 1; j < HDR_LANE; ++j) {
            const long long w2 = ((long long)pp[j] << 32) | (unsigned)(lane + 32 * j);
            if (better(kk[j], w2, k, w)) { k = kk[j]; w = w2; }
          }
          warp_best(k, w, &s_k, &s_w);
          __syncwarp();
          wpos = (int)(s_w >> 32);
          wcta = (int)(unsigned)s_w;
          if (lane == 0) {
            s_wpos = wpos;
            s_wcta = wcta;
          }
          if (wcta != cta) {  // its reflector is out
            const unsigned long long* f = a.flags + (size_t)(s & 1) * P + wcta;
            for (;;) {
              unsigned long long t;
              hq_ld_word(f, t);
              ok = t == tag;
              if (ok || ++it >= a.spin_limit) break;
              if ((it & 15u) == 0u && hq_ld_volatile(a.err) != 0) break;
            }
            ok = __all_sync(0xffffffffu, ok);
            __threadfence();  // flag, then reflector
          }
        }
        if (!ok && lane == 0) {
          atomicCAS(a.err, 0, HQ_ERR_BARRIER_TIMEOUT);
          s_bad = 1;
        }
      }
    } else if (bk > -2) {
      // The candidate's reflector, v = [1; scale x] from row s on.
      const double* x = colp(lq);
      const int wt = tid - 32;
      if (wt < ND) {
        const double t = tail_squares(x, s, m, wt, ND);
        if (lane == 0) s_red[warp - 1] = t;
      }
      worker_barrier();
      if (warp == 1) {
        double q = s_red[lane & (NDW - 1)];
#pragma unroll
        for (int o = NDW / 2; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
        if (lane == 0) {
          const HqReflector h = hq_make_reflector_sq(x[s], m - s > 1 ? q : 0.0);
          s_tau = h.tau;
          s_scale = h.scale;
          s_beta = h.beta;
        }
      }
      worker_barrier();
      const double scale = s_scale;
      for (int i = s + wt; i < m; i += WT - 32) {
        const double v = i == s ? 1.0 : x[i] * scale;
        sc[i] = v;
        if (P > 1) rec[i] = v;
      }
      if (P > 1) {
        if (wt == 0) rec[m] = s_tau;
        worker_barrier();
        if (wt == 0) {
          __threadfence();  // reflector, then flag
          hq_st_word(a.flags + (size_t)(s & 1) * P + cta, (unsigned long long)tag);
        }
      }
    }
    __syncthreads();
    if (s_bad) return;  // an exchange gave up; the other CTAs see the error word
    if (P > 1) {
      wpos = s_wpos;
      wcta = s_wcta;
    }
    const bool own = wcta == cta;
    // 2. Bookkeeping: the winner goes to position s, what was there to the
    //    winner's.  The winner's reflector; its owner puts it in place.
    for (int j = tid; j < cnt; j += WT) {
      const int q = sact[j], p = spos[q];
      if (own && q == lq) {
        spos[q] = s;
        sact[j] = -1;  // replaced by the last one below
      } else if (p == s) {
        spos[q] = wpos;
      }
    }
    double tau;
    if (own) {
      tau = s_tau;
      double* x = colp(lq);
      for (int i = s + tid; i < m; i += WT) x[i] = i == s ? s_beta : sc[i];
      if (tid == 0) a.tau[s] = tau;
    } else {
      const double* from = a.cols + ((size_t)(s & 1) * P + wcta) * (m + 1);
      tau = hq_ldcg(from + m);
      for (int i = s + tid; i < m; i += WT) sv[i] = hq_ldcg(from + i);
    }
    __syncthreads();
    if (own) {
      --cnt;
      if (warp == 0)  // the list without the pivot
        for (int j = lane; j < cnt; j += 32)
          if (sact[j] < 0) sact[j] = sact[cnt];
      __syncthreads();
    }

    // 3. Update the CTA's remaining columns; LAWN 176 downdate of the squared
    //    norms, one thread per column; norms to be recomputed, a warp each.
    apply_columns<WW>(own ? sc : sv, tau, s, m, cnt, sact, srs, colp, warp, lane);
    __syncthreads();
    int any = 0;
    for (int j = tid; tid < ND && j < cnt; j += ND) {
      const int q = sact[j];
      const double d = sd[q];
      int flag = 0;
      if (d != 0.0) {
        const double r = srs[q];
        const double nd = fma(-r, r, d);
        if (hq_norm_cancelled(nd, sthr[q])) flag = 1;
        else sd[q] = nd;
      }
      if (flag) sd[q] = -1.0;
      any |= flag;
    }
    best_of_columns();
    if (__syncthreads_or(any)) {
      for (int j = warp; j < cnt; j += WW) {
        const int q = sact[j];
        if (sd[q] != -1.0) continue;  // uniform across the warp
        const double* x = colp(q);
        double t = 0.0;
        for (int i = s + 1 + lane; i < m; i += 32) t = fma(x[i], x[i], t);
        t = hq_warp_sum(t);
        __syncwarp();
        if (lane == 0) {
          sd[q] = t;
          sthr[q] = HQ_TOL3Z * t;
        }
      }
      __syncthreads();
      best_of_columns();
      __syncthreads();
    }
  }

  // The way out: the columns where they were, and the order as pairs.
  if (a.staged)
    for (int q = warp; q < nl; q += WW) {
      const double* x = colp(q);
      double* g = a.A + (size_t)(cta + P * q) * a.lda;
      for (int i = lane; i < m; i += 32) g[i] = x[i];
    }
  for (int q = tid; q < nl; q += WT) {
    const int c = cta + P * q;
    if (spos[q] != c) {
      const int i = atomicAdd(a.npairs, 1);
      if (i < 2 * a.ns) {
        a.pairs[2 * i] = spos[q];
        a.pairs[2 * i + 1] = c;
      } else {
        atomicCAS(a.err, 0, HQ_ERR_BAD_SHAPE);  // cannot happen: at most two move per stage
      }
    }
  }
}

// CTAs: as many as bring a stage's FP64 work (2 FMAs a clock on one SM) to ~700
// clocks on average, one column each at least, one per SM at most.  (350 and
// 1500 measured within 2 %.)
int wide_grid(const hq_device_info* dev, int m, int n) {
  const double k = m < n ? m : n, l = m < n ? n : m;
  const double clocks = (2.0 * l * k * k - 2.0 * k * k * k / 3.0) / (4.0 * k);
  int p = (int)(clocks / 700.0) + 1;
  if (p > dev->num_sms) p = dev->num_sms;
  if (p > MAX_P) p = MAX_P;
  if (p > n) p = n;
  return p;
}

}  // namespace

// Bytes of the exchange, and of the columns' state kept in global memory (a
// matrix of millions of columns).
static size_t wide_words(size_t P) { return 2 * P * (P * 16 + 8); }  // that carry tags
static size_t wide_exchange(size_t P, int m) { return wide_words(P) + 2 * P * ((size_t)m + 1) * 8; }
static size_t wide_state(const hq_device_info* dev, size_t P, int m, int n) {
  const size_t cpc = ((size_t)n + P - 1) / P;
  return sizeof(double) * (2 * (size_t)m + 4 * cpc) > dev->smem_optin ? sizeof(double) * 4 * cpc * P : 0;
}

extern "C" size_t hq_wide_xch_bytes(const hq_device_info* dev, int m, int n) {
  const size_t P = (size_t)wide_grid(dev, m, n);
  return wide_exchange(P, m) + wide_state(dev, P, m, n);
}

extern "C" int hq_wide_qrp(cudaStream_t stream, const hq_device_info* dev, int m, int n,
                           double* A, int lda, double* tau, void* xch, int* pairs, int* npairs,
                           int* err, unsigned spin_limit) {
  if (m <= 0 || n <= 0) return 0;
  if (m > HQ_WIDE_MAX_ROWS || lda < m) return (int)cudaErrorInvalidValue;
  WdArgs a;
  a.m = m;
  a.n = n;
  a.ns = m < n ? m : n;
  a.A = A;
  a.lda = lda;
  a.tau = tau;
  a.pairs = pairs;
  a.npairs = npairs;
  a.err = err;
  a.spin_limit = spin_limit;
  const int P = wide_grid(dev, m, n);
  a.hdrs = static_cast<unsigned char*>(xch);
  a.flags = reinterpret_cast<unsigned long long*>(a.hdrs + (size_t)2 * P * P * 16);
  a.cols = reinterpret_cast<double*>(a.flags + 2 * P);
  a.cpc = (n + P - 1) / P;
  const bool in_smem = wide_state(dev, (size_t)P, m, n) == 0;
  a.state = in_smem ? nullptr : reinterpret_cast<double*>(a.hdrs + wide_exchange((size_t)P, m));
  const size_t fixed = sizeof(double) * (2 * (size_t)m + (in_smem ? 4 * (size_t)a.cpc : 0));
  const size_t with_x = fixed + sizeof(double) * (size_t)m * a.cpc;
  a.staged = in_smem && with_x <= dev->smem_optin;
  const size_t smem = a.staged ? with_x : fixed;
  if (smem > dev->smem_optin) return (int)cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(wide_qrp_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  // The tags start from zero.
  const size_t words = P > 1 ? wide_words((size_t)P) / 4 : 0;
  const int z = hq_zero_words(stream, npairs, 1, words ? xch : nullptr, words);
  if (z) return z;
  void* args[] = {&a};
  e = hq_launch_coop((const void*)wide_qrp_kernel, dim3(P), dim3(WT), args, smem, stream);
  hq_count_launches(1);
  return (int)e;
}
