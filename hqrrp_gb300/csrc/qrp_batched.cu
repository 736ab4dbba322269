// qrp_batched.cu -- thousands of independent small pivoted QRs in one
// persistent launch.
//
// dgeqp4 hands every matrix with min(m, n) < 1000 to LAPACK's dgeqpf / dgeqp3
// (lapack_compatible_sources/NoFLA_HQRRP_WY_blk_var4.c:189-199); both produce
// the Businger-Golub column-pivoted Householder QR with LAWN 176 norm
// downdating, the algorithm restated per matrix here.  A batch is scheduled
// through device work queues: the host orders the matrices by cost (largest
// first), and whoever is free takes the next index with an atomic until the
// queue is empty, so uneven sizes balance across the SMs.
//
// One SM runs 2 FP64 FMAs per clock, so a 1024 x 512 matrix alone holds it for
// 55 ms and bounds a batch of any size.  The launch is therefore made of
// clusters of T CTAs (T = 1, 2, 4 or 8, part of the launch shape).  The
// largest matrices go through a first queue to whole clusters, columns dealt
// out cyclically; the CTAs then take the rest one by one from a second queue.
// In a team, every CTA pushes its best candidate into the shared memory of the
// others, one cluster barrier per stage, and each reads the winning column
// from its owner -- shared memory over the cluster's network, or L2 -- and
// builds the reflector itself.
//
// Columns never move: a pivot is bookkeeping (each column's position), and the
// final order is made once, on the way out.  A matrix is staged in shared
// memory when its CTA's columns fit the launch's staging budget and worked on
// in place (L2-resident) otherwise.  FP64 instructions are the time (an SM
// issues one per 16 clocks), so a warp takes four columns together: their dot
// products' partial sums are reduced by six additions instead of twenty, and
// norms are kept squared, without divisions or square roots, one thread per
// column.
//
// The launch shape -- threads per CTA, the staging budget, T -- is chosen by
// the host autotuner (hqrrp_driver.c) per batch signature.  Measured on GB300
// against one CTA per matrix, swapped columns and a column per warp: 1024
// matrices of the benchmark's sizes 90 -> 28.5 ms (FP64 alone: 16), 4096 of them
// 139 -> 95 (63).
//
// All columns are free (LAPACK jpvt = 0 input); on return jpvt[k] is the
// 1-based original index of column k, tau[0..min(m,n)) the reflector scalars,
// R and the reflectors overwrite A.
#include "hq_columns.cuh"

namespace {

constexpr int T_MAX = 8;        // CTAs per cluster (the portable limit)
constexpr int TEAM_ROWS = HQ_BATCHED_TEAM_ROWS;  // rows of a matrix a team takes
constexpr unsigned LAYER_NS = 4000;  // more than what CTAs of one layer start apart

struct BatchArgs {
  int batch;
  const int* m;
  const int* n;
  double* const* A;
  const int* lda;
  int* const* jpvt;
  double* const* tau;
  int* info;
  const int* order;   // schedule: matrix indices, largest first
  int* next;          // queue heads: [0] single CTAs, [1] teams (zeroed before the launch)
  const int* n_team;  // the first *n_team of the schedule are the teams' (T > 1)
  int stage_bytes;    // dynamic shared memory available for staging a matrix
  int max_n;
};

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Every thread of every CTA of the cluster; what was written before, to any of
// the cluster's shared memories or to global memory, is read after.
__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}
__device__ __forceinline__ unsigned cluster_addr(const void* smem, unsigned rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((unsigned)__cvta_generic_to_shared(smem)), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_st(unsigned addr, long long a, long long b) {
  asm volatile("st.shared::cluster.v2.b64 [%0], {%1, %2};" ::"r"(addr), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ double cluster_ld(unsigned addr) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  return v;
}

// LEAN: 1024 threads an SM and the registers that leaves each, for batches of
// long or narrow columns, which wait for loads and stages more than for the FP64
// pipe (batches of 1200, best launch shape without and with it: 600 x 20 1.15 ->
// 0.88 ms, 1100 x 64 16.5 -> 13.0, 10000 x 30 61 -> 43).
template <int NT, bool LEAN>
__global__ void __launch_bounds__(NT, (LEAN ? 1024 : 512) / NT) qrp_batched_kernel(BatchArgs a) {
  extern __shared__ __align__(16) double smem[];
  constexpr int NW = NT / 32;
  // FP64 work that is one value per thread goes to four warps, one per quarter
  // of the SM: more would only queue up for the same pipes.
  constexpr int ND = 128, NDW = ND / 32;
  __shared__ __align__(16) long long s_cand[2][T_MAX][2];  // the team's candidates, by stage parity
  __shared__ __align__(16) long long s_item[2][2];
  __shared__ double s_red[NW];
  __shared__ long long s_bk[NDW], s_at[NDW];
  __shared__ double s_tau, s_scale, s_beta;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned rank = cluster_rank();
  const int T_all = (int)cluster_size();
  double* sd = smem;                  // squared partial norms of this CTA's columns, max_n
  double* sthr = sd + a.max_n;        // recompute at or below, max_n
  double* srs = sthr + a.max_n;       // the stage's new entries of row s, max_n
  int* spos = (int*)(srs + a.max_n);  // positions, max_n
  int* sact = spos + a.max_n;         // columns not yet factored, max_n
  double* sv = srs + 2 * a.max_n;     // a team's reflector, TEAM_ROWS
  double* sX = sv + (T_all > 1 ? TEAM_ROWS : 0);

  // Every CTA of the cluster has started before its shared memory is written.
  if (T_all > 1) cluster_barrier();
  // CTAs that share an SM take their first matrix one after the other, a layer
  // of the whole GPU at a time: else the two largest, the next in the queue, often
  // meet on one SM and take twice as long as they need (1024 matrices of up to
  // 1024 x 512, two CTAs an SM, single / teams of two / of four: 115 / 58 / 31.4
  // ms, so 71 / 42 / 28.5).  The warp's slot on the SM tells the layer; should it
  // not, only the balance suffers.
  if (tid == 0) {
    unsigned slot;
    asm volatile("mov.u32 %0, %%warpid;" : "=r"(slot));
    __nanosleep(slot / NW * LAYER_NS);
  }
  bool teams = T_all > 1;
  for (int turn = 0;; ++turn) {
    // The next matrix: of the teams' queue while it lasts, then of the CTAs'.
    int item;
    if (teams) {
      if (rank == 0 && tid == 0) {
        const int q = atomicAdd(a.next + 1, 1);
        const long long it = q < min(*a.n_team, a.batch) ? a.order[q] : -1;
        for (int r = 0; r < T_all; ++r) cluster_st(cluster_addr(s_item[turn & 1], r), it, 0);
      }
      cluster_barrier();
      item = (int)s_item[turn & 1][0];
      if (item < 0) {
        teams = false;
        continue;
      }
    } else {
      __syncthreads();
      if (tid == 0) {
        const int q = atomicAdd(a.next, 1) + (T_all > 1 ? *a.n_team : 0);
        s_item[turn & 1][0] = q < a.batch ? a.order[q] : -1;
      }
      __syncthreads();
      item = (int)s_item[turn & 1][0];
      if (item < 0) break;
    }
    const int m = a.m[item], n = a.n[item], lda = a.lda[item];
    // The plan gives no matrix of more than TEAM_ROWS rows to a team; one that
    // has them now is the first CTA's alone, the others go on to the next
    // turn's barrier.
    const bool alone = teams && m > TEAM_ROWS;
    if (alone && rank != 0) continue;
    const int T = teams && !alone ? T_all : 1, me = T > 1 ? (int)rank : 0;
    double* Ag = a.A[item];
    // A size the kernel cannot take (negative, lda < max(1, m), more than
    // max_n columns) is flagged and left untouched; an empty matrix is done.
    const bool bad = m < 0 || n < 0 || n > a.max_n || lda < max(1, m);
    if (bad || m == 0 || n == 0) {
      if (tid == 0 && me == 0 && a.info) a.info[item] = bad ? HQ_ERR_BAD_SHAPE : 0;
      continue;
    }
    // This CTA's columns are me, me + T, ...: local index q, column me + T q.
    const int nl = (n - me + T - 1) / T;
    const bool staged = (long long)m * ((n + T - 1) / T) * 8 <= a.stage_bytes;
    auto colp = [&](int q) { return staged ? sX + (size_t)q * m : Ag + (size_t)(me + T * q) * lda; };
    // Load, initial norms (warp per column, fixed lane order).
    for (int q = warp; q < nl; q += NW) {
      const double* g = Ag + (size_t)(me + T * q) * lda;
      double* x = colp(q);
      double t = 0.0;
#pragma unroll 4
      for (int i = lane; i < m; i += 32) {
        const double v = g[i];
        if (staged) x[i] = v;
        t = fma(v, v, t);
      }
      t = hq_warp_sum(t);
      if (lane == 0) {
        sd[q] = t;
        sthr[q] = HQ_TOL3Z * t;
        spos[q] = me + T * q;
        sact[q] = q;
      }
    }
    __syncthreads();
    int cnt = nl;  // columns in sact
    // Each warp's best of the columns not yet factored; at = position << 32 |
    // column.
    auto best_of_columns = [&]() {
      if (tid >= ND) return;
      long long k = -2, at = 0x7fffffffLL << 32;
      for (int j = tid; j < cnt; j += ND) {
        const int q = sact[j];
        const long long kj = hq_norm_key(sd[q]);
        const long long aj = ((long long)spos[q] << 32) | (unsigned)(me + T * q);
        if (better(kj, aj, k, at)) { k = kj; at = aj; }
      }
      warp_best(k, at, s_bk + warp, s_at + warp);
    };
    best_of_columns();
    __syncthreads();

    const int mn = min(m, n);
    int pend = -1;  // a team's own pivot column, to be written after the next barrier
    double pend_beta = 0.0;
    auto flush = [&](int s_of) {  // v (still in sv) below row s_of, beta on it
      if (pend < 0) return;
      double* x = colp(pend);
      for (int i = s_of + 1 + tid; i < m; i += NT) x[i] = sv[i];
      if (tid == 0) x[s_of] = pend_beta;
      pend = -1;
    };
    for (int s = 0; s < mn; ++s) {
      // 1. The pivot.
      long long bk = s_bk[0], at = s_at[0];
#pragma unroll
      for (int w = 1; w < NDW; ++w)
        if (better(s_bk[w], s_at[w], bk, at)) { bk = s_bk[w]; at = s_at[w]; }
      if (T > 1) {
        if (tid < T) cluster_st(cluster_addr(s_cand[s & 1][me], (unsigned)tid), bk, at);
        cluster_barrier();
        bk = s_cand[s & 1][0][0];
        at = s_cand[s & 1][0][1];
        for (int r = 1; r < T; ++r)
          if (better(s_cand[s & 1][r][0], s_cand[s & 1][r][1], bk, at)) {
            bk = s_cand[s & 1][r][0];
            at = s_cand[s & 1][r][1];
          }
        flush(s - 1);
      }
      const int wpos = (int)(at >> 32), wcol = (int)(unsigned)at;
      const int owner = wcol % T, wq = wcol / T;
      for (int j = tid; j < cnt; j += NT) {
        const int q = sact[j];
        const int p = spos[q];
        if (owner == me && q == wq) {
          spos[q] = s;
          sact[j] = -1;  // replaced by the last one below
        } else if (p == s) {
          spos[q] = wpos;
        }
      }
      if (T > 1) __syncthreads();  // sv is rewritten below

      // 2. The pivot column and its reflector; v in place (one CTA), or in sv.
      double* v = T > 1 ? sv : colp(wq);
      {
        if (T > 1) {
          const double* g = Ag + (size_t)wcol * lda;
          const unsigned r0 = cluster_addr(sX + (size_t)wq * m, (unsigned)owner);
          for (int i = s + tid; i < m; i += NT)
            sv[i] = staged ? cluster_ld(r0 + 8u * (unsigned)i) : hq_ldcg(g + i);
          __syncthreads();
        }
        // (All warps load a long column.)
        const int nd = m > TEAM_ROWS ? NT : ND;
        if (tid < nd) {
          const double t = tail_squares(v, s, m, tid, nd);
          if (lane == 0) s_red[warp] = t;
        }
        __syncthreads();
        if (warp == 0) {
          const int parts = nd / 32;  // a power of two
          double q = s_red[lane & (parts - 1)];
          for (int o = parts / 2; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
          if (lane == 0) {
            const HqReflector h = hq_make_reflector_sq(v[s], m - s > 1 ? q : 0.0);
            s_tau = h.tau;
            s_scale = h.scale;
            s_beta = h.beta;
            if (me == 0) a.tau[item][s] = h.tau;
          }
        } else if (warp == 1) {
          // The list without the pivot: its place takes the last column.
          if (owner == me) {
            for (int j = lane; j < cnt - 1; j += 32)
              if (sact[j] < 0) sact[j] = sact[cnt - 1];
          }
        }
        if (owner == me) --cnt;
        __syncthreads();
        const double scale = s_scale;
        for (int i = s + 1 + tid; i < m; i += NT) v[i] *= scale;
        if (tid == 0) v[s] = 1.0;  // restored to beta after the update
        if (T > 1 && owner == me) {
          pend = wq;
          pend_beta = s_beta;
        }
        __syncthreads();
      }

      // 3. X[s:, k] -= tau v (v^T X[s:, k]).
      apply_columns<NW, LEAN>(v, s_tau, s, m, cnt, sact, srs, colp, warp, lane);
      __syncthreads();

      // 4. LAWN 176 downdate of the squared norms, one thread per column; the
      //    next pivot.  Norms to be recomputed (rare): a warp per column.
      if (T == 1 && tid == 0) v[s] = s_beta;
      int any = 0;
      for (int jj = tid; tid < ND && jj < cnt; jj += ND) {
        const int q = sact[jj];
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
        for (int jj = warp; jj < cnt; jj += NW) {
          const int q = sact[jj];
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
    if (T > 1) {
      cluster_barrier();  // every CTA has read the last pivot column
      flush(mn - 1);
      __syncthreads();
    }

    // The way out: jpvt, and the columns in their final order.
    for (int q = tid; q < nl; q += NT) a.jpvt[item][spos[q]] = me + T * q + 1;
    if (staged) {
      // Every CTA of a team has loaded its columns long before (a barrier ago).
      for (int q = warp; q < nl; q += NW) {
        const double* x = colp(q);
        double* g = Ag + (size_t)spos[q] * lda;
        for (int i = lane; i < m; i += 32) g[i] = x[i];
      }
      __syncthreads();
      if (T > 1) cluster_barrier();  // s_cand, sv and sX may be reused
    } else {
      // In place: rows are dealt out over the threads, and each walks the
      // cycles of the permutation (position p takes the column jpvt[p]).
      if (T > 1) cluster_barrier();  // jpvt and the columns are written
      else __syncthreads();
      int* from = spos;  // column that position p takes; then marked by its complement
      int* seq = sact;   // the cycles one after the other, a cycle's first entry complemented
      __shared__ int s_len;
      for (int p = tid; p < n; p += NT) from[p] = __ldcg(a.jpvt[item] + p) - 1;
      __syncthreads();
      if (tid == 0) {
        int len = 0;
        for (int p = 0; p < n; ++p) {
          if (from[p] < 0 || from[p] == p) continue;
          int c = p;
          bool first = true;
          while (from[c] >= 0) {
            const int nx = from[c];
            seq[len++] = first ? ~c : c;
            first = false;
            from[c] = ~nx;
            c = nx;
          }
        }
        s_len = len;
      }
      __syncthreads();
      const int len = s_len;
      for (int i = me * NT + tid; i < m; i += T * NT) {
        double* x = Ag + i;
        double first = 0.0;  // value of the current cycle's first entry
        constexpr int B = 8;  // loads in flight along a cycle
        for (int e = 0; e < len; e += B) {
          // Entry e receives the next one's value; the last of a cycle its
          // first's.  All loads of a batch precede its stores, and a batch's
          // stores only reach entries whose values are already loaded.
          double val[B];
#pragma unroll
          for (int u = 0; u < B; ++u) {
            if (e + u < len) {
              const int c = seq[e + u];
              if (c < 0) first = __ldcg(x + (size_t)(~c) * lda);
              const int nx = e + u + 1 < len ? seq[e + u + 1] : -1;
              val[u] = nx < 0 ? first : __ldcg(x + (size_t)nx * lda);
            }
          }
#pragma unroll
          for (int u = 0; u < B; ++u) {
            if (e + u < len) {
              const int c = seq[e + u];
              x[(size_t)(c < 0 ? ~c : c) * lda] = val[u];
            }
          }
        }
      }
      __syncthreads();
      if (T > 1) cluster_barrier();
    }
    if (tid == 0 && me == 0 && a.info) a.info[item] = 0;
  }
}

template <int NT, bool LEAN = false>
int launch_t(cudaStream_t st, const hq_device_info* dev, BatchArgs a, int ctas_per_sm,
             int team) {
  const size_t fixed = sizeof(double) * 4 * (size_t)a.max_n +
                       (team > 1 ? sizeof(double) * TEAM_ROWS : 0);
  if (fixed > dev->smem_optin) return (int)cudaErrorInvalidValue;
  if ((size_t)a.stage_bytes > dev->smem_optin - fixed) a.stage_bytes = (int)(dev->smem_optin - fixed);
  const size_t smem = fixed + (size_t)a.stage_bytes;
  auto kernel = qrp_batched_kernel<NT, LEAN>;
  cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, NT, smem);
  if (e != cudaSuccess) return (int)e;
  if (per_sm < 1) return (int)cudaErrorInvalidConfiguration;
  if (ctas_per_sm < per_sm) per_sm = ctas_per_sm;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)team;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = team > 1 ? 1 : 0;
  int grid = dev->num_sms * per_sm;
  if (team > 1) {
    int ncl = 0;
    cfg.gridDim = dim3((unsigned)team);
    e = cudaOccupancyMaxActiveClusters(&ncl, kernel, &cfg);
    if (e != cudaSuccess) return (int)e;
    if (ncl < 1) return (int)cudaErrorInvalidConfiguration;
    if (grid > ncl * team) grid = ncl * team;
    grid = grid / team * team;
    if (grid < team) grid = team;
  } else if (grid > a.batch) {
    grid = a.batch;
  }
  cfg.gridDim = dim3((unsigned)grid);
  e = cudaLaunchKernelEx(&cfg, kernel, a);
  hq_count_launches(1);
  return (int)e;
}

}  // namespace

// Workspace: queue heads, the teams' counts, schedule.
extern "C" size_t hq_qrp_batched_workspace(int batch) {
  return sizeof(int) * (size_t)(batch + 64);
}

extern "C" int hq_qrp_batched(cudaStream_t stream, const hq_device_info* dev, int batch,
                              const int* d_m, const int* d_n, double* const* d_A,
                              const int* d_lda, int* const* d_jpvt, double* const* d_tau,
                              int* d_info, void* d_work, int max_n, int threads, int stage_kb,
                              int ctas_per_sm, int team) {
  if (batch <= 0) return 0;
  if (max_n <= 0 || max_n > 4096) return (int)cudaErrorInvalidValue;
  if (team != 1 && team != 2 && team != 4 && team != T_MAX) return (int)cudaErrorInvalidValue;
  if (ctas_per_sm < 1 || ctas_per_sm > 7) return (int)cudaErrorInvalidValue;
  BatchArgs a;
  a.batch = batch;
  a.m = d_m;
  a.n = d_n;
  a.A = d_A;
  a.lda = d_lda;
  a.jpvt = d_jpvt;
  a.tau = d_tau;
  a.info = d_info;
  a.next = static_cast<int*>(d_work);
  a.n_team = static_cast<const int*>(d_work) + HQ_BATCHED_TEAM_SLOT + ctas_per_sm;
  a.order = static_cast<const int*>(d_work) + 32;
  a.stage_bytes = stage_kb * 1024;
  a.max_n = max_n;
  cudaError_t e = cudaMemsetAsync(a.next, 0, 2 * sizeof(int), stream);
  if (e != cudaSuccess) return (int)e;
  switch (threads) {
    case 128: return launch_t<128>(stream, dev, a, ctas_per_sm, team);
    case 256:
      return ctas_per_sm > 2 ? launch_t<256, true>(stream, dev, a, ctas_per_sm, team)
                             : launch_t<256>(stream, dev, a, ctas_per_sm, team);
    case 512:
      return ctas_per_sm > 1 ? launch_t<512, true>(stream, dev, a, ctas_per_sm, team)
                             : launch_t<512>(stream, dev, a, ctas_per_sm, team);
    default: return (int)cudaErrorInvalidValue;
  }
}
