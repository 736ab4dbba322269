// qrp_gram.cu -- the mixed-precision path's panel without a grid-wide
// reduction per column (sm_103a).
//
// The reference factors each block's panel column by column
// (NoFLA_QRPmod_WY_unb_var4, NoFLA_HQRRP_WY_blk_var4.c:774-886): every column
// needs the norms and dot products of the whole panel, which on a GPU is one
// grid-wide reduction and barrier per column.  Here a panel Ap (mp x b,
// b <= 128), pivoted within its b columns, is factored as
//   1. G = Ap^T Ap, a split-BF16 tensor-core product (FP64-accurate);
//   2. pivoted Cholesky of G, column-scaled to unit diagonal, in FP32 on one
//      SM: P and a preconditioner R1 with (Ap P)^T (Ap P) ~ R1^T R1.  The
//      Schur complement's diagonal holds the squared norms of the columns'
//      residuals, so taking the largest (first on ties) is the pivot rule of
//      column-pivoted Householder QR;
//   3. CholeskyQR2 (Fukaya, Nakatsukasa, Yanagisawa, Yamamoto, 2014), the
//      first pass preconditioned in FP32 (Yamazaki, Tomov, Dongarra, 2015):
//      Q1 = Ap P R1^{-1}, G2 = Q1^T Q1 = R2^T R2 with R2 in FP64,
//      Q = Q1 R2^{-1}, R = R2 R1; the FP64 second pass restores
//      orthogonality to working precision;
//   4. Householder reconstruction (Ballard, Demmel, Grigori, Jacquelin,
//      Nguyen, Solomonik, IPDPS 2014): the LU factorization without pivoting
//      Q - [D; 0] = V U, with D_kk = -sign of the k-th Schur pivot, gives the
//      unit lower trapezoidal V of Householder QR with LAPACK's sign choice
//      (beta = -sign(alpha) ||x||), tau_k = -D_kk U_kk, and R_H = D R.
// The steps over the panel's rows (G, Q1, G2, Q, V2 = Q2 U^{-1}) are
// tensor-core products issued by the host driver; the b x b steps are the
// kernels of this file.  FP64 runs at about two lanes per clock on a GB300
// SM, so one SM is slow for them: the FP64 Cholesky and LU run on a cluster
// of eight CTAs (each owns every eighth column, or group of four; the pivot
// columns travel through distributed shared memory), the triangular inverses and products
// and the first pass's scaling with one CTA per column, and only the pivoted
// first pass itself on one SM, in FP32.
//
// A step that meets a panel it cannot factor accurately sets a bit in a
// status word: a first-pass pivot below 1e-5 of the column's own squared
// norm (the column lies within about 0.3 % of the span of the earlier ones:
// the panel is too ill-conditioned for an FP32 preconditioner), a
// second-pass pivot below 1e-10 of its diagonal entry (G2 far from the
// identity), or an LU pivot outside [0.5, 2.5] (|U_kk| = tau_k lies in
// [1, 2] for an orthonormal Q).  The commit kernel then leaves
// the panel untouched, and the cooperative pivoted panel kernel, which reads
// the same word, factors it instead.

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>

#include "hq_common.cuh"
#include "hq_internal.h"

namespace cg = cooperative_groups;

namespace {

constexpr int GN = HQ_GRAM_MAX;  // widest panel
constexpr int LDS = GN + 1;      // shared-memory column stride of the b x b kernels
constexpr int CT = 256;          // threads of the one-SM kernel
constexpr int CW = CT / 32;
constexpr int TW = 4;            // warps per CTA of the second pass's kernel (one column per CTA)
constexpr float PIVOT32_REL_MIN = 1e-5f;  // first pass: scaled pivot floor
constexpr double CHOL2_REL_MIN = 1e-10;   // cluster Cholesky: pivot floor, relative to the diagonal
constexpr double NEARID_MAX = 2e-4;       // second pass: largest max|G2 - I| it converges from
constexpr int NEARID_ITERS = 4;           // second pass: fixed-point steps
constexpr int CL = 8;                     // CTAs of the cluster kernels
constexpr int CLT = 256;                  // threads per CTA of the cluster kernels
constexpr int CLW = CLT / 32;
constexpr int OWN = GN / CL;              // columns per CTA (column j lives in CTA j % CL)
static_assert(OWN == 2 * CLW, "each warp of a cluster CTA updates two own columns");

// Pass 1: pivoted Cholesky of the n x n Gram matrix G scaled to unit diagonal,
// in FP32 on one SM, the matrix held in registers.  The FP64 arithmetic around
// it -- S_ij = G_ij / sqrt(G_ii G_jj) before, R = Rs diag(sqrt(G_pp)) after --
// runs on one CTA per column (gram_scale_kernel, gram_unscale_kernel): on the
// one SM it took 28 of 97 us.
//
// What the three kernels hand on, in the memory of R (in) and of G (out):
struct PcholIn {
  float S[GN * GN];  // scaled Gram matrix, column-major
  double rt[GN];     // sqrt(G_jj)
  float key[GN];     // G_jj relative to the largest
};
struct PcholOut {
  float Rs[GN * GN];  // Rs[k * GN + i]: row k of the scaled factor at source column i
  double rt[GN];
  float r[GN];        // its diagonal
  int ord[GN];        // source column of position k
};
static_assert(sizeof(PcholIn) <= sizeof(double) * GN * GN &&
                  sizeof(PcholOut) <= sizeof(double) * GN * GN,
              "they fit a GN x GN FP64 matrix");

__global__ void __launch_bounds__(GN)
    gram_scale_kernel(int n, const double* __restrict__ G, int ldg, PcholIn* __restrict__ in) {
  HQ_PDL_WAIT();
  __shared__ double s_scj;
  __shared__ float s_max[GN / 32];
  const int i = threadIdx.x, j = blockIdx.x;
  const double d = i < n ? G[i + (size_t)i * ldg] : 0.0;
  const double v = i < n && j < n ? G[i + (size_t)j * ldg] : 0.0;
  const int ok = d > 0.0 && d <= 1.7e308;
  const double rt = ok ? sqrt(d) : 0.0;
  const double sc = ok ? 1.0 / rt : 0.0;
  if (i == j) s_scj = sc;
  __syncthreads();
  in->S[i + j * GN] = (float)(v * sc * s_scj);
  if (j != 0) return;
  const float l = ok ? (float)log2(d) : -4096.0f;  // squared norm, scaled below
  float m = l;
#pragma unroll
  for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((i & 31) == 0) s_max[i >> 5] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < GN / 32; ++w) m = fmaxf(m, s_max[w]);
  in->rt[i] = rt;
  in->key[i] = exp2f(l - m);
}

// Thread (warp w, lane t) holds the 64 entries (i, j) with i = t + 32 a
// (a < 4) and j = 16 w + c (c < 16) of the full symmetric matrix.  Columns are
// not moved: step k picks the active column p with the largest residual norm
// (scaled Schur diagonal times the column's original squared norm relative to
// the largest; the lowest index among residuals equal to 2^-15), the warp
// holding column p publishes it over the active rows (0 elsewhere), every warp
// scales it to l = S[:, p] / sqrt(S[p][p]), and every thread updates its
// entries by S_ij -= l_i l_j -- a no-op on eliminated rows and columns, so the
// update needs no masks.  Every warp keeps the whole diagonal (four entries a
// lane, updated as the matrix's) and finds the pivot itself with one warp
// maximum, so a step takes one barrier, and only the diagonal stands between a
// published column and the next pivot.  What every warp does for itself is
// what the SM issues most: 8 warps.  (16 warps, the diagonal passed through
// shared memory, the FP64 scaling on the same SM: 102 us for n = 128; the
// three kernels now take 70.)
// Sets *stat = 0, or `bit` when a scaled pivot is not above PIVOT32_REL_MIN;
// *alt (the second pass's choice of method) and *emax (its max|E|) := 0.
__global__ void __launch_bounds__(CT, 1)
    gram_pchol32_kernel(int n, const PcholIn* __restrict__ in, PcholOut* __restrict__ out,
                        int* __restrict__ stat, int bit, int* __restrict__ alt,
                        unsigned long long* __restrict__ emax) {
  HQ_PDL_WAIT();
  __shared__ __align__(16) float s_l[2][GN];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int CPW = GN / CW;  // columns a warp
  static_assert(CPW == 16 && GN == 128, "register layout: 8 warps x 16 columns, 32 lanes x 4 rows");
  float S[4][CPW];
#pragma unroll
  for (int c = 0; c < CPW; ++c)
#pragma unroll
    for (int a = 0; a < 4; ++a) S[a][c] = in->S[lane + 32 * a + (CPW * warp + c) * GN];
  // Per lane: the keys (negative once eliminated) and diagonal entries of
  // columns lane + 32 q.
  float keyr[4], dq[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int j = lane + 32 * q;
    keyr[q] = j < n ? in->key[j] : -1.0f;
    dq[q] = in->S[j + j * GN];
  }
  for (int j = tid; j < GN; j += CT) out->rt[j] = in->rt[j];
  int fail = 0;
  for (int k = 0; k < n; ++k) {
    // Every warp finds the pivot: one 32-bit key per column, the residual's
    // FP32 bits above the low 8 (positive floats order like their bits) and
    // 255 - j below them, so one warp maximum gives the largest residual
    // and, among residuals equal to 2^-15, the lowest column.  Residuals below
    // zero and eliminated columns are negative; a NaN, the largest, fails.
    int best = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      best = max(best, (__float_as_int(keyr[q] * dq[q]) & ~255) | (255 - (lane + 32 * q)));
    best = __reduce_max_sync(0xffffffffu, best);
    const int p = 255 - (best & 255);
    const int pq = (p >> 5) & 3;
    float dsel = dq[0];
#pragma unroll
    for (int q = 1; q < 4; ++q)
      if (q == pq) dsel = dq[q];
    const float dp = __shfl_sync(0xffffffffu, dsel, p & 31);
    if (best == 0 || !(dp > PIVOT32_REL_MIN)) {  // also NaN and a zero column
      fail = 1;
      break;
    }
    if ((p & 31) == lane) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (q == pq) keyr[q] = -1.0f;
    }
    // The warp holding column p publishes it over the active rows (row
    // lane + 32 a is this lane's column slot a); every warp takes the root
    // and the quotient meanwhile and scales for itself.
    const bool owner = warp == p / CPW;
    if (owner) {
      const int cp = p % CPW;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        float v = S[a][0];
#pragma unroll
        for (int c = 1; c < CPW; ++c)
          if (c == cp) v = S[a][c];
        s_l[k & 1][lane + 32 * a] = keyr[a] >= 0.0f ? v : 0.0f;
      }
    }
    const float r = sqrtf(dp);
    const float rinv = 1.0f / r;
    __syncthreads();
    float li[4], lj[CPW];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      li[a] = s_l[k & 1][lane + 32 * a] * rinv;
      dq[a] = fmaf(-li[a], li[a], dq[a]);
    }
    const float4* l4 = reinterpret_cast<const float4*>(&s_l[k & 1][CPW * warp]);
#pragma unroll
    for (int c = 0; c < CPW; c += 4) {
      const float4 f = l4[c / 4];
      lj[c] = f.x * rinv;
      lj[c + 1] = f.y * rinv;
      lj[c + 2] = f.z * rinv;
      lj[c + 3] = f.w * rinv;
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < CPW; ++c) S[a][c] = fmaf(-li[a], lj[c], S[a][c]);
    if (owner) {
#pragma unroll
      for (int a = 0; a < 4; ++a) out->Rs[k * GN + lane + 32 * a] = li[a];
      if (lane == 0) {
        out->r[k] = r;
        out->ord[k] = p;
      }
    }
  }
  if (tid == 0) {
    *stat = fail ? bit : 0;
    *alt = 0;
    *emax = 0ull;
  }
}

// perm[m] (source column of position m) and R = Rs diag(sqrt(G_pp)) in FP64
// (upper, zeros below); R = I and perm the identity when *stat has `bit`.
__global__ void __launch_bounds__(GN)
    gram_unscale_kernel(int n, const PcholOut* __restrict__ out, const int* __restrict__ stat,
                        int bit, double* __restrict__ R, int ldr, int* __restrict__ perm) {
  HQ_PDL_WAIT();
  const int k = threadIdx.x, m = blockIdx.x;
  const int fail = *stat & bit;
  const int p = fail ? m : out->ord[m];
  if (k < n) {
    double v = fail ? (k == m ? 1.0 : 0.0) : 0.0;
    if (!fail && k <= m)
      v = (double)(k < m ? out->Rs[k * GN + p] : out->r[m]) * out->rt[p];
    R[k + (size_t)m * ldr] = v;
  }
  if (k == 0) perm[m] = p;
}

// An FP32 approximation of 1 / x as an FP64, for |x| well inside FP32's range
// (LU: 0.5 .. 2.5; Cholesky: the root of a diagonal entry of a scaled Gram
// matrix).  Both conversions take integer instructions: x's bits are cut to
// FP32's, the quotient's widened.
__device__ __forceinline__ double seed_inverse(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned f =
      (hi & 0x80000000u) | ((((hi & 0x7FFFFFFFu) - 0x38000000u) << 3) | (lo >> 29));
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(f)));
  const unsigned r = __float_as_uint(y);
  return __hiloint2double((int)((r & 0x80000000u) | (((r & 0x7FFFFFFFu) >> 3) + 0x38000000u)),
                          (int)(r << 29));
}

// 1 / x from that seed y and one third-order correction: with e = 1 - x y,
// 1 / x = y (1 + e + e^2 + ...), so y + y (e + e^2) leaves e^3 ~ 2^-66: three
// dependent FMAs instead of the longer FP64 division sequence.
__device__ __forceinline__ double quick_inverse(double x) {
  const double y = seed_inverse(x);
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// Unpivoted FP64 Cholesky factorization of the symmetric n x n matrix A (lda,
// lower triangle read) on a cluster of CL CTAs: F := R (upper, zeros below)
// with R^T R = A.  Column j lives in the shared memory of CTA j % CL.  Step k:
// every CTA updates its columns right of k from the published, scaled column k;
// the owner of column k + 1 updates that column first, takes its root, scales
// it and writes it into every CTA's receive buffer (distributed shared memory,
// double-buffered by the parity of the step).  One cluster barrier per step,
// split into arrive and wait around the update of the remaining own columns;
// it also orders the receive buffers' reuse.  A pivot q <= 1e-10 d0 is recorded
// and replaced by 1, so every CTA takes the same barriers; the output is then
// the identity and `bit` is set in *stat.  (Only panels without pivoting, and
// second passes far from the identity, come here.)
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(CLT, 1)
    cluster_chol_kernel(int n, const double* __restrict__ A, int lda, double* __restrict__ F,
                        int ldf, int* __restrict__ stat, int bit, const int* __restrict__ gate) {
  HQ_PDL_WAIT();
  if (gate != nullptr && *gate == 0) return;  // every CTA of the cluster reads the same word
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  __shared__ double Xc[OWN * LDS];
  __shared__ double colbuf[2][GN];
  __shared__ int s_bad[2];
  __shared__ double s_pub[2];  // root, 1 / root
  __shared__ int s_pubbad;
  __shared__ double s_d0[OWN];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nown = rank < n ? (n - 1 - rank) / CL + 1 : 0;
  for (int c = warp; c < nown; c += CLW) {
    const int j = rank + CL * c;
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = lane + 32 * q;
      v[q] = (i < n && i >= j) ? A[i + (size_t)j * lda] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = lane + 32 * q;
      if (i < n) Xc[i + c * LDS] = v[q];
    }
  }
  __syncthreads();
  for (int c = tid; c < nown; c += CLT) s_d0[c] = Xc[(rank + CL * c) + c * LDS];

  // Publish own column kk (local c): root, final diagonal, scaled rows below
  // it, into every CTA's buffers of parity par.  Thread 0 wrote the column's
  // diagonal entry itself (it updates row kk), so it takes the root before
  // the barrier that orders the other rows' updates.
  auto publish = [&](int kk, int par) {
    const int c = kk / CL;
    if (tid == 0) {
      const double q = Xc[kk + c * LDS];
      const int bad = !(q > CHOL2_REL_MIN * s_d0[c]);
      const double piv = bad ? 1.0 : sqrt(q);
      s_pub[0] = piv;
      s_pub[1] = quick_inverse(piv);
      s_pubbad = bad;
      Xc[kk + c * LDS] = piv;
    }
    __syncthreads();
    const double inv = s_pub[1];
    for (int i = kk + 1 + tid; i < n; i += CLT) {
      const double l = Xc[i + c * LDS] * inv;
      Xc[i + c * LDS] = l;
#pragma unroll
      for (int r = 0; r < CL; ++r) *cl.map_shared_rank(&colbuf[par][i], r) = l;
    }
    if (tid < CL) *cl.map_shared_rank(&s_bad[par], tid) = s_pubbad;
  };

  if (rank == 0 && n > 0) publish(0, 0);
  cl.sync();
  int bad = 0;
  for (int k = 0; k < n; ++k) {
    const int b = k & 1;
    const int nx = k + 1;
    if (nx < n && nx % CL == rank) {
      const int c1 = nx / CL;
      const double lj = colbuf[b][nx];
      for (int i = nx + tid; i < n; i += CLT) Xc[i + c1 * LDS] -= colbuf[b][i] * lj;
      publish(nx, b ^ 1);
    }
    // The other own columns right of k: warp w takes local columns w and
    // w + CLW together, their four row chunks unrolled.  Everything read
    // from the receive buffer is in registers before this CTA arrives at the
    // step's barrier (after which the buffer may be refilled two steps on),
    // so the barrier's latency overlaps the update; the wait comes last.
    {
      double xa[2][4], lb[2][4], mult[2];
      int act[2], base[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int c = warp + CLW * u, j = rank + CL * c;
        act[u] = c < nown && j > k && j != nx;
        mult[u] = act[u] ? colbuf[b][j] : 0.0;
        base[u] = j;
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int c = warp + CLW * u, i = base[u] + lane + 32 * q;
          const int live = act[u] && i < n;
          xa[u][q] = live ? Xc[i + c * LDS] : 0.0;
          lb[u][q] = live ? colbuf[b][i] : 0.0;
        }
      bad |= s_bad[b];
      cl.barrier_arrive();
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int c = warp + CLW * u, i = base[u] + lane + 32 * q;
          if (act[u] && i < n) Xc[i + c * LDS] = xa[u][q] - lb[u][q] * mult[u];
        }
    }
    __syncthreads();  // the CTA's own updates (after its arrive) before the next step reads them
    cl.barrier_wait();
  }
  // R[g][i] = L[i][g]; R[i][g] = 0 below the diagonal
  for (int c = warp; c < nown; c += CLW) {
    const int g = rank + CL * c;
    for (int i = g + lane; i < n; i += 32) {
      F[g + (size_t)i * ldf] = bad ? (i == g ? 1.0 : 0.0) : Xc[i + c * LDS];
      if (i > g) F[i + (size_t)g * ldf] = 0.0;
    }
  }
  if (bad && rank == 0 && tid == 0) atomicOr(stat, bit);
}

// Unpivoted FP64 LU of A - D (n x n), D_kk = -1 if the k-th Schur pivot is >= 0
// else +1 (Householder reconstruction), on a cluster of CL CTAs: F := L
// strictly below the diagonal and U on and above it, dsgn := D, tau :=
// -D U_kk.
//
// Columns go in groups of LUG: group g lives in the shared memory of CTA
// g % CL.  Step g: the owner of group g + 1 brings it up to date with group g,
// factors its diagonal block in one warp (registers and shuffles) while the
// other warps update the rows below, solves those rows for L, and writes L's
// four columns into every CTA's receive buffer (distributed shared memory);
// the other columns are updated between the arrive and the wait of the step's
// cluster barrier.  Three receive buffers: group g's is read until a CTA
// arrives at step g + 1 and written again during step g + 2.  (A barrier and
// an exchange per column instead of per group took 152 us for n = 128; this
// takes 105, most of it the diagonal blocks' chains of a quotient, a product
// and an update per column.)  A pivot |u| outside [0.5, 2.5] is recorded and
// replaced by 1; the output is then the identity (and tau 0) and `bit` is set
// in *stat.
constexpr int LUG = 4;
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(CLT, 1)
    cluster_lu_kernel(int n, const double* __restrict__ A, int lda, double* __restrict__ F,
                      int ldf, double* __restrict__ dsgn, double* __restrict__ tau,
                      int* __restrict__ stat, int bit) {
  HQ_PDL_WAIT();
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  __shared__ double Xc[OWN * LDS];
  // Row i of the published group's L (zeros on and above the diagonal).
  __shared__ __align__(16) double Lb[3][GN][LUG];
  __shared__ int s_badb[3];
  __shared__ __align__(16) double s_l44[LUG][LUG];
  __shared__ double s_u44[LUG][LUG], s_inv[LUG], s_u[LUG][LUG], s_D[OWN];
  __shared__ int s_bad;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  static_assert(OWN % LUG == 0 && OWN == 2 * CLW && CLT == 256, "layout");
  const int ng = (n + LUG - 1) / LUG;
  auto column = [&](int c) { return ((c / LUG) * CL + rank) * LUG + c % LUG; };
  for (int c = warp; c < OWN; c += CLW) {
    const int j = column(c);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = lane + 32 * q;
      Xc[i + c * LDS] = (i < n && j < n) ? A[i + (size_t)j * lda] : 0.0;
    }
  }
  __syncthreads();

  // U's entries x[k .. k + 3] of a column against group buffer L, k its first row.
  auto solve4 = [&](const double (*L)[LUG], int k, const double* x, double (&u)[LUG]) {
    u[0] = x[k];
    u[1] = fma(-L[k + 1][0], u[0], x[k + 1]);
    u[2] = fma(-L[k + 2][1], u[1], fma(-L[k + 2][0], u[0], x[k + 2]));
    u[3] = fma(-L[k + 3][2], u[2],
               fma(-L[k + 3][1], u[1], fma(-L[k + 3][0], u[0], x[k + 3])));
  };

  // Bring own group gg up to date with group gg - 1, factor and publish it.
  auto factor = [&](int gg) {
    const int k0 = LUG * gg, kp = k0 - LUG, lc = LUG * (gg / CL);
    const double (*L)[LUG] = Lb[(gg + 2) % 3];
    double* X = Xc + lc * LDS;
    if (warp == 0) {
      const int r = (lane >> 2) & 3, cc = lane & 3;
      double v = X[min(k0 + r, GN - 1) + cc * LDS];
      if (gg > 0) {
        double u[LUG];
        solve4(L, kp, X + cc * LDS, u);
        const double* lr = L[min(k0 + r, GN - 1)];
        v = fma(-lr[1], u[1], fma(-lr[0], u[0], v)) - fma(lr[3], u[3], lr[2] * u[2]);
      }
      int bad = 0;
#pragma unroll
      for (int kk = 0; kk < LUG; ++kk) {
        if (k0 + kk >= n) break;
        const double q = __shfl_sync(0xffffffffu, v, kk * 4 + kk);
        const double a = __shfl_sync(0xffffffffu, v, r * 4 + kk);
        const double uk = __shfl_sync(0xffffffffu, v, kk * 4 + cc);
        // The comparisons are of the bits: an FP64 one holds the chain up.
        const long long qb = __double_as_longlong(q);
        const double D = qb >= 0 || qb == LLONG_MIN ? -1.0 : 1.0;
        double piv = q - D;
        const long long ub = __double_as_longlong(piv) & LLONG_MAX;
        if (!(ub >= 0x3FE0000000000000LL && ub <= 0x4004000000000000LL)) {  // 0.5, 2.5
          bad = 1;
          piv = 1.0;
        }
        // quick_inverse, and a / piv beside it.
        const double y = seed_inverse(piv);
        const double e = fma(-piv, y, 1.0), ay = a * y;
        const double t = fma(e, e, e);
        const double l = fma(ay, t, ay);
        if (r > kk && cc > kk) v = fma(-l, uk, v);
        if (r > kk && cc == kk) v = l;
        if (r == kk && cc == kk) v = piv;
        if (lane == 0) {
          s_inv[kk] = fma(y, t, y);
          s_D[lc + kk] = D;
        }
      }
      if (lane < 16) {
        if (k0 + r < n) X[k0 + r + cc * LDS] = v;
        s_l44[r][cc] = r > cc ? v : 0.0;
        s_u44[r][cc] = v;
      }
      if (lane == 0) s_bad = bad;
    } else if (gg > 0) {
      if (warp == 1 && lane < LUG) {
        double u[LUG];
        solve4(L, kp, X + lane * LDS, u);
#pragma unroll
        for (int s = 0; s < LUG; ++s) s_u[lane][s] = u[s];
      }
      __syncwarp();
      asm volatile("bar.sync 1, %0;" ::"n"(CLT - 32) : "memory");  // warps 1 on
      // (Warp 4 would share its FP64 pipe with warp 0.)
      for (int it = warp < 4 ? warp - 1 : warp == 4 ? 4 * LUG : warp - 2; it < 4 * LUG;
           it += CLW - 2) {
        const int cc = it & 3, i = k0 + LUG + lane + 32 * (it >> 2);
        if (i < n) {
          const double2 l01 = *reinterpret_cast<const double2*>(&L[i][0]);
          const double2 l23 = *reinterpret_cast<const double2*>(&L[i][2]);
          double x = X[i + cc * LDS];
          x = fma(-l01.x, s_u[cc][0], x);
          x = fma(-l01.y, s_u[cc][1], x);
          x = fma(-l23.x, s_u[cc][2], x);
          X[i + cc * LDS] = fma(-l23.y, s_u[cc][3], x);
        }
      }
    }
    __syncthreads();
    const int par = gg % 3;
    if (tid < GN) {
      const int i = k0 + LUG + tid;
      if (i < n) {  // then the group is full
        double a0 = X[i], a1 = X[i + LDS], a2 = X[i + 2 * LDS], a3 = X[i + 3 * LDS];
        double2 l01, l23;
        l01.x = a0 * s_inv[0];
        a1 = fma(-l01.x, s_u44[0][1], a1);
        a2 = fma(-l01.x, s_u44[0][2], a2);
        a3 = fma(-l01.x, s_u44[0][3], a3);
        l01.y = a1 * s_inv[1];
        a2 = fma(-l01.y, s_u44[1][2], a2);
        a3 = fma(-l01.y, s_u44[1][3], a3);
        l23.x = a2 * s_inv[2];
        a3 = fma(-l23.x, s_u44[2][3], a3);
        l23.y = a3 * s_inv[3];
        X[i] = l01.x;
        X[i + LDS] = l01.y;
        X[i + 2 * LDS] = l23.x;
        X[i + 3 * LDS] = l23.y;
#pragma unroll
        for (int d = 0; d < CL; ++d) {
          double* p = cl.map_shared_rank(&Lb[par][i][0], d);
          *reinterpret_cast<double2*>(p) = l01;
          *reinterpret_cast<double2*>(p + 2) = l23;
        }
      }
    } else if (warp == 4) {
      const int d = lane >> 2, r = lane & 3;
      if (k0 + r < n) {
        double* p = cl.map_shared_rank(&Lb[par][k0 + r][0], d);
        *reinterpret_cast<double2*>(p) = *reinterpret_cast<const double2*>(&s_l44[r][0]);
        *reinterpret_cast<double2*>(p + 2) = *reinterpret_cast<const double2*>(&s_l44[r][2]);
      }
    } else if (warp == 5) {
      if (lane < CL) *cl.map_shared_rank(&s_badb[par], lane) = s_bad;
    } else if (warp == 6 && gg > 0 && lane < LUG * LUG) {
      X[kp + (lane >> 2) + (lane & 3) * LDS] = s_u[lane & 3][lane >> 2];
    }
  };

  if (rank == 0) factor(0);
  cl.sync();
  int bad = 0;
  for (int g = 0; g < ng; ++g) {
    const double (*L)[LUG] = Lb[g % 3];
    const int k0 = LUG * g;
    bad |= s_badb[g % 3];
    if (g + 1 < ng && (g + 1) % CL == rank) factor(g + 1);
    __syncwarp();
    cl.barrier_arrive();
    // The other own columns right of the group: warp w takes local columns w
    // and w + CLW.
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = warp + CLW * h, gc = (c / LUG) * CL + rank;
      if (gc <= g + (((g + 1) % CL) == rank ? 1 : 0) || column(c) >= n) continue;
      double* x = Xc + c * LDS;
      double u[LUG];
      solve4(L, k0, x, u);
      __syncwarp();
      if (lane < LUG) x[k0 + lane] = lane == 0 ? u[0] : lane == 1 ? u[1] : lane == 2 ? u[2] : u[3];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = k0 + LUG + lane + 32 * q;
        if (i < n) {
          const double2 l01 = *reinterpret_cast<const double2*>(&L[i][0]);
          const double2 l23 = *reinterpret_cast<const double2*>(&L[i][2]);
          double v = x[i];
          v = fma(-l01.x, u[0], v);
          v = fma(-l01.y, u[1], v);
          v = fma(-l23.x, u[2], v);
          x[i] = fma(-l23.y, u[3], v);
        }
      }
    }
    __syncthreads();
    cl.barrier_wait();
  }
  // Output of the own columns.
  for (int c = warp; c < OWN; c += CLW) {
    const int j = column(c);
    if (j >= n) continue;
    for (int i = lane; i < n; i += 32)
      F[i + (size_t)j * ldf] = bad ? (i == j ? 1.0 : 0.0) : Xc[i + c * LDS];
  }
  for (int c = tid; c < OWN; c += CLT) {
    const int j = column(c);
    if (j >= n) continue;
    dsgn[j] = bad ? -1.0 : s_D[c];
    tau[j] = bad ? 0.0 : -s_D[c] * Xc[j + c * LDS];
  }
  if (bad && rank == 0 && tid == 0) atomicOr(stat, bit);
}

// Fixed-point steps the second pass needs from max|E|: the error of R^{-1}
// after m steps is about max|E|^(m+1) (measured on FP32-preconditioned
// panels), below 2^-53 after 2 steps up to 4e-6, 3 up to 5e-5, 4 up to
// NEARID_MAX.
__device__ __forceinline__ int nearid_steps(double emax) {
  return emax <= 4e-6 ? 2 : (emax <= 5e-5 ? 3 : NEARID_ITERS);
}

// One step of the second CholeskyQR pass for G = I + E near the identity:
// R2 = I + X (X upper with its diagonal) and R2^{-1} = I + Z are the fixed
// points of
//   X <- Uh(E - X^T X),   Z <- -X (I + Z),
// Uh = strict upper part plus half the diagonal (X + X^T + X^T X = E is
// R2^T R2 = G).  Both converge linearly at a rate of about ||E||_2, so
// NEARID_ITERS steps from X = Uh(E), Z = -X reach working precision when
// max|E| <= NEARID_MAX (first pass in FP32: max|E| ~ 1e-6 .. 1e-4 for
// panels with condition numbers 10 .. 300); fewer suffice for smaller
// max|E| (nearid_steps), and the later launches then only copy.  Every product is a column of a
// b x b product, so the pass needs no sequential factorization: one CTA per
// column c stages X's columns 0..c (asynchronous copies, all in flight at once)
// and each thread accumulates one row (13 us for n = 128; with
// the copies through registers and an atomic maximum per entry 30).
// Step 0: X, Z are Uh(E), -Uh(E) (Xin, Zin unused), and the CTA checks its
// column of E against NEARID_MAX, setting *alt when it is exceeded (the
// later steps then return at once and the cluster Cholesky and a triangular
// inverse, gated on *alt, take the pass) and raising *emax; the last step
// writes I + X and I + Z.
__global__ void __launch_bounds__(TW * 32)
    nearid_kernel(int n, const double* __restrict__ G, int ldg, const double* __restrict__ Xin,
                  const double* __restrict__ Zin, int ld, double* __restrict__ Xout,
                  double* __restrict__ Zout, int it, int* __restrict__ alt,
                  unsigned long long* __restrict__ emax) {
  HQ_PDL_WAIT();
  extern __shared__ double sX[];  // LDS * n: X's columns 0..c, rows <= column
  __shared__ double s_z[GN];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c = blockIdx.x;
  const int first = it == 0, last = it == NEARID_ITERS - 1;
  if (!first) {
    if (*alt != 0) return;  // too far from the identity: the cluster Cholesky runs
    if (it >= nearid_steps(__longlong_as_double((long long)*emax))) {
      // converged: pass X and Z through (adding I after the last step)
      for (int i = tid; i < n; i += TW * 32) {
        const double d = (last && i == c) ? 1.0 : 0.0;
        Xout[i + (size_t)c * ld] = Xin[i + (size_t)c * ld] + d;
        Zout[i + (size_t)c * ld] = Zin[i + (size_t)c * ld] + d;
      }
      return;
    }
  }
  {
    const double* src = first ? G : Xin;
    const int lds = first ? ldg : ld;
    for (int j = warp; j <= c; j += TW)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = lane + 32 * q;
        if (i <= j)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                           (unsigned)__cvta_generic_to_shared(sX + i + j * LDS)),
                       "l"(src + i + (size_t)j * lds)
                       : "memory");
      }
  }
  static_assert(TW * 32 == GN, "one row a thread");
  // E's entry of this row (diagonal: minus 1) and Z's.
  const int i = tid;
  const double gi = i <= c ? G[i + (size_t)c * ldg] : 0.0;
  const double ei = i == c ? gi - 1.0 : gi;
  const double zi = !first && i <= c ? Zin[i + (size_t)c * ld] : 0.0;
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (first) {
    if (i <= c) sX[i + i * LDS] = 0.5 * (sX[i + i * LDS] - 1.0);
    // The CTA's largest |E|; non-negative doubles order like their bits.
    const double ae = fabs(ei);
    const int ok = i > c || ae <= NEARID_MAX;  // not for NaN
    unsigned long long m = ok && i <= c ? (unsigned long long)__double_as_longlong(ae) : 0ull;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const unsigned long long om = __shfl_xor_sync(0xffffffffu, m, o);
      m = om > m ? om : m;
    }
    if (lane == 0 && m != 0ull) atomicMax(emax, m);
    if (__syncthreads_or(!ok) && tid == 0) atomicOr(alt, 1);
  }
  if (i <= c) s_z[i] = first ? -sX[i + c * LDS] : zi;
  __syncthreads();
  if (i < n) {
    double xn = 0.0, zn = 0.0;
    if (i <= c) {
      double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
      int k = 0;
      for (; k + 3 <= i; k += 4) {
        a0 = fma(sX[k + i * LDS], sX[k + c * LDS], a0);
        a1 = fma(sX[k + 1 + i * LDS], sX[k + 1 + c * LDS], a1);
        a2 = fma(sX[k + 2 + i * LDS], sX[k + 2 + c * LDS], a2);
        a3 = fma(sX[k + 3 + i * LDS], sX[k + 3 + c * LDS], a3);
      }
      for (; k <= i; ++k) a0 = fma(sX[k + i * LDS], sX[k + c * LDS], a0);
      const double r = ei - ((a0 + a1) + (a2 + a3));
      xn = i < c ? r : 0.5 * r;
      double b0 = 0.0, b1 = 0.0, b2 = 0.0, b3 = 0.0;
      k = i;
      for (; k + 3 <= c; k += 4) {
        b0 = fma(sX[i + k * LDS], s_z[k], b0);
        b1 = fma(sX[i + (k + 1) * LDS], s_z[k + 1], b1);
        b2 = fma(sX[i + (k + 2) * LDS], s_z[k + 2], b2);
        b3 = fma(sX[i + (k + 3) * LDS], s_z[k + 3], b3);
      }
      for (; k <= c; ++k) b0 = fma(sX[i + k * LDS], s_z[k], b0);
      zn = -sX[i + c * LDS] - ((b0 + b1) + (b2 + b3));
      if (last && i == c) {
        xn += 1.0;
        zn += 1.0;
      }
    }
    Xout[i + (size_t)c * ld] = xn;
    Zout[i + (size_t)c * ld] = zn;
  }
}

// One triangular job: X = A^{-1} (mode 0) or X = diag(rs) A B (mode 1; rs
// may be null), A and B upper triangular n x n (only their upper triangles
// are read), X upper triangular with zeros below.
struct TriJob {
  int mode;
  const double* A;
  int lda;
  const double* B;
  int ldb;
  const double* rs;
  double* X;
  int ldx;
};

// One CTA per column c of X (and per job: blocks [0, n) run j0, [n, 2n)
// j1), one thread per entry.  The inverse is a back substitution: a warp holds
// 32 entries and, once the warps after it have handed theirs over in shared
// memory, broadcasts each entry as it becomes known and adds it to the ones
// before it with the factors -A_ik / A_ii ready in registers: a shuffle and a
// multiply-add a step.  The product is a sum per entry.  (One warp walking
// the column took 33 us for n = 128; this takes 17.)
__global__ void __launch_bounds__(GN)
    tri_kernel(int n, TriJob j0, TriJob j1, const int* __restrict__ gate) {
  HQ_PDL_WAIT();
  __shared__ double sx[GN];
  if (gate != nullptr && *gate == 0) return;
  const int i = threadIdx.x, lane = i & 31, warp = i >> 5;
  const TriJob J = blockIdx.x < (unsigned)n ? j0 : j1;
  const int c = (int)(blockIdx.x % (unsigned)n);
  const int lda = J.lda;
  const double* __restrict__ Ai = J.A + i;  // row i
  const bool live = i <= c;
  double x = 0.0;
  if (J.mode == 0) {
    const double dinv = live ? 1.0 / Ai[(size_t)i * lda] : 0.0;
    double z[32];
#pragma unroll
    for (int d = 0; d < 32; ++d) {
      const int k = warp * 32 + d;
      z[d] = (k > i && k <= c) ? -Ai[(size_t)k * lda] * dinv : 0.0;
    }
    double acc = i == c ? 1.0 : 0.0;
    for (int b = c >> 5; b >= 0; --b) {
      double zb[32];
      if (warp < b) {
#pragma unroll
        for (int d = 0; d < 32; ++d) {
          const int k = 32 * b + d;
          zb[d] = k <= c ? Ai[(size_t)k * lda] : 0.0;
        }
      }
      if (warp == b) {
        x = acc * dinv;
#pragma unroll
        for (int d = 31; d > 0; --d) {
          const double xd = __shfl_sync(0xffffffffu, x, d);
          if (lane < d && 32 * b + d <= c) x = fma(xd, z[d], x);
        }
        sx[i] = x;
      }
      __syncthreads();
      if (warp < b) {
        double a1 = 0.0;
#pragma unroll
        for (int d = 0; d < 32; d += 2) {
          acc = fma(-zb[d], sx[32 * b + d], acc);
          a1 = fma(-zb[d + 1], sx[32 * b + d + 1], a1);
        }
        acc += a1;
      }
    }
  } else {
    sx[i] = live ? J.B[i + (size_t)c * J.ldb] : 0.0;
    __syncthreads();
    double a1 = 0.0;
    int k = i;
#pragma unroll 4
    for (; k < c; k += 2) {
      x = fma(Ai[(size_t)k * lda], sx[k], x);
      a1 = fma(Ai[(size_t)(k + 1) * lda], sx[k + 1], a1);
    }
    if (k == c) x = fma(Ai[(size_t)k * lda], sx[k], x);
    x += a1;
    if (J.rs && live) x *= J.rs[i];
  }
  if (i < n) J.X[i + (size_t)c * J.ldx] = live ? x : 0.0;
}

// When *stat == 0: the panel P (mp x n, ldp) gets R on and above the
// diagonal and the Householder vectors below it (L's strict lower part in
// the top n rows, V2 below from U's rows >= n, where the V2 product wrote
// them); U's top n rows become the explicit unit-lower V1; tau and the
// panel permutation (identity: the Gram path's pivots were applied to the
// columns before the products) are written.  Otherwise nothing.
__global__ void gram_commit_kernel(int mp, int n, double* __restrict__ P, int ldp,
                                   double* __restrict__ U, int ldu, const double* __restrict__ RH,
                                   int ldr, const double* __restrict__ LU, int ldlu,
                                   const double* __restrict__ tau_in, double* __restrict__ tau,
                                   int* __restrict__ perm, const int* __restrict__ stat,
                                   int* __restrict__ count) {
  HQ_PDL_WAIT();
  const int st = *stat;
  if (count != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
    atomicAdd(&count[st != 0 ? 1 : 0], 1);
  if (st != 0) return;
  const int k = blockIdx.y;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < mp; i += gridDim.x * blockDim.x) {
    double pv;
    if (i < n) {
      double uv;
      if (i < k) {
        pv = RH[i + (size_t)k * ldr];
        uv = 0.0;
      } else if (i == k) {
        pv = RH[i + (size_t)k * ldr];
        uv = 1.0;
      } else {
        pv = LU[i + (size_t)k * ldlu];
        uv = pv;
      }
      U[i + (size_t)k * ldu] = uv;
    } else {
      pv = U[i + (size_t)k * ldu];
    }
    P[i + (size_t)k * ldp] = pv;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    tau[k] = tau_in[k];
    perm[k] = k;
  }
}

}  // namespace

extern "C" int hq_gram_pchol32(cudaStream_t stream, int n, double* G, int ldg, double* R,
                               int ldr, int* perm, int* stat, int bit, int* alt,
                               unsigned long long* emax) {
  if (n <= 0 || n > GN || ldg != GN || ldr != GN) return (int)cudaErrorInvalidValue;
  PcholIn* in = reinterpret_cast<PcholIn*>(R);
  PcholOut* out = reinterpret_cast<PcholOut*>(G);
  hq_launch(gram_scale_kernel, GN, GN, 0, stream, n, G, ldg, in);
  hq_launch(gram_pchol32_kernel, 1, CT, 0, stream, n, in, out, stat, bit, alt, emax);
  hq_launch(gram_unscale_kernel, n, GN, 0, stream, n, out, stat, bit, R, ldr, perm);
  hq_count_launches(3);
  return (int)cudaGetLastError();
}

extern "C" int hq_cluster_fact(cudaStream_t stream, int n, int mode, const double* A, int lda,
                               double* F, int ldf, double* dsgn, double* tau, int* stat, int bit,
                               const int* gate) {
  if (n <= 0 || n > GN || mode < 0 || mode > 1) return (int)cudaErrorInvalidValue;
  if (mode == 0)
    hq_launch(cluster_chol_kernel, CL, CLT, 0, stream, n, A, lda, F, ldf, stat, bit, gate);
  else
    hq_launch(cluster_lu_kernel, CL, CLT, 0, stream, n, A, lda, F, ldf, dsgn, tau, stat, bit);
  hq_count_launches(1);
  return (int)cudaGetLastError();
}

extern "C" int hq_nearid_chol(cudaStream_t stream, int n, const double* G, int ldg, double* R,
                              double* Rinv, double* wX, double* wZ, int ld, int* alt,
                              unsigned long long* emax) {
  if (n <= 0 || n > GN) return (int)cudaErrorInvalidValue;
  const size_t smem = sizeof(double) * (size_t)LDS * (size_t)n;
  cudaError_t e =
      cudaFuncSetAttribute(nearid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  static_assert(NEARID_ITERS % 2 == 0, "the last step writes R and Rinv");
  for (int it = 0; it < NEARID_ITERS; ++it) {
    // ping-pong: odd steps write the work pair, even steps the output pair
    const double* xi = (it & 1) ? wX : R;
    const double* zi = (it & 1) ? wZ : Rinv;
    double* xo = (it & 1) ? R : wX;
    double* zo = (it & 1) ? Rinv : wZ;
    hq_launch(nearid_kernel, n, TW * 32, smem, stream, n, G, ldg, xi, zi, ld, xo, zo, it, alt, emax);
  }
  hq_count_launches(NEARID_ITERS);
  return (int)cudaGetLastError();
}

extern "C" int hq_tri(cudaStream_t stream, int n, int mode, const double* A, int lda,
                      const double* B, int ldb, const double* rs, double* X, int ldx,
                      const int* gate) {
  return hq_tri2g(stream, n, mode, A, lda, B, ldb, rs, X, ldx, -1, nullptr, 0, nullptr, 0,
                  nullptr, nullptr, 0, gate);
}

extern "C" int hq_tri2(cudaStream_t stream, int n, int mode0, const double* A0, int lda0,
                       const double* B0, int ldb0, const double* rs0, double* X0, int ldx0,
                       int mode1, const double* A1, int lda1, const double* B1, int ldb1,
                       const double* rs1, double* X1, int ldx1) {
  return hq_tri2g(stream, n, mode0, A0, lda0, B0, ldb0, rs0, X0, ldx0, mode1, A1, lda1, B1, ldb1,
                  rs1, X1, ldx1, nullptr);
}

extern "C" int hq_tri2g(cudaStream_t stream, int n, int mode0, const double* A0, int lda0,
                        const double* B0, int ldb0, const double* rs0, double* X0, int ldx0,
                        int mode1, const double* A1, int lda1, const double* B1, int ldb1,
                        const double* rs1, double* X1, int ldx1, const int* gate) {
  if (n <= 0) return 0;
  if (n > GN || mode0 < 0 || mode0 > 1 || mode1 < -1 || mode1 > 1)
    return (int)cudaErrorInvalidValue;
  const TriJob j0 = {mode0, A0, lda0, B0, ldb0, rs0, X0, ldx0};
  const TriJob j1 = {mode1 < 0 ? 0 : mode1, A1, lda1, B1, ldb1, rs1, X1, ldx1};
  hq_launch(tri_kernel, mode1 < 0 ? n : 2 * n, GN, 0, stream, n, j0, j1, gate);
  hq_count_launches(1);
  return (int)cudaGetLastError();
}

extern "C" int hq_gram_commit(cudaStream_t stream, int mp, int n, double* P, int ldp, double* U,
                              int ldu, const double* RH, int ldr, const double* LU, int ldlu,
                              const double* tau_in, double* tau, int* perm, const int* stat,
                              int* count) {
  if (mp <= 0 || n <= 0) return 0;
  int bx = (mp + 255) / 256;
  if (bx > 64) bx = 64;
  hq_launch(gram_commit_kernel, dim3(bx, n), 256, 0, stream, mp, n, P, ldp, U, ldu, RH, ldr, LU, ldlu,
                                                      tau_in, tau, perm, stat, count);
  hq_count_launches(1);
  return (int)cudaGetLastError();
}
