// gemm_f64.cu -- FP64 GEMM for the plain-precision path.
//
// C = alpha * op(A) * op(B) + beta * C, column-major, op in {N, T}.  GB300's
// FP64 rate (2 DFMA per clock per SM, the same for DMMA and the FP64 pipe: a
// warp instruction occupies its quarter of the SM for 64 cycles) bounds every
// FP64 product in HQRRP, and by so much that nothing else about a tile
// matters: a 32 x 32 tile asks for 1 byte per clock per SM.  What is left to
// lose is pipe time: multiplications by padding, and SMs without work.  So the
// tiles are small -- 32 x 32, four warps of 16 x 16 each, a warp whose part
// lies outside the matrix (or, for a Gram matrix, below the diagonal) issuing
// no FP64 at all -- and K is cut wherever that levels the load of the SMs
// (plan_split).  Partial products are summed in a fixed order by a second
// kernel, so results do not depend on scheduling.
//
// Measured on GB300 against 64 x 64 tiles with slices of at least 128 of K
// (time at 1.24 TFLOP/s in brackets): 74 x 64 x 2000, the sketch downdate of
// a 2000^2 factorization, 154 -> 34 us (15); its Gram matrix 64 x 64 x 2000,
// 154 -> 28 (13); W1 = U^T C, 64 x 1936 x 2000, 553 -> 439 (400);
// C -= U W2 of 500 x 436 x 64, 74 -> 40 (23), of 2000 x 1936 x 64, 475 -> 435
// (400), of 8000 x 7872 x 128, 13.28 -> 13.21 ms.
#include "hq_common.cuh"

namespace {

constexpr int BM = 32, BN = 32, BK = 16, NT = 128;

// upper: only the tiles that reach the upper triangle are formed (C's strictly
// lower triangle below them keeps its values).
template <bool TA, bool TB>
__global__ void __launch_bounds__(NT, 8)
    dgemm_tile(int M, int N, int K, int kchunk, double alpha, const double* __restrict__ A,
               int lda, const double* __restrict__ B, int ldb, double beta,
               double* __restrict__ Cm, int ldc, double* __restrict__ ws, int upper) {
  HQ_PDL_WAIT();
  __shared__ double As[BK][BM + 1];
  __shared__ double Bs[BK][BN + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  if (upper && m0 >= n0 + BN) return;  // every row of the tile below every column
  const int kbeg = blockIdx.z * kchunk;
  const int kend = min(K, kbeg + kchunk);
  // This warp's 16 x 16 part; lane (lx, ly) has rows lx + 8 i, columns ly + 4 j.
  const int wm = (warp & 1) * 16, wn = (warp >> 1) * 16;
  const int lx = lane & 7, ly = lane >> 3;
  const bool live = m0 + wm < M && n0 + wn < N && !(upper && m0 + wm >= n0 + wn + 16);

  double ra[4], rb[4];
  auto load_a = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int idx = tid + NT * q;
      int i, k;
      if (!TA) { i = idx & (BM - 1); k = idx >> 5; }
      else     { k = idx & (BK - 1); i = idx >> 4; }
      const int gi = m0 + i, gk = k0 + k;
      double v = 0.0;
      if (gi < M && gk < kend)
        v = TA ? A[gk + (size_t)gi * lda] : A[gi + (size_t)gk * lda];
      ra[q] = v;
    }
  };
  auto load_b = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int idx = tid + NT * q;
      int j, k;
      if (!TB) { k = idx & (BK - 1); j = idx >> 4; }
      else     { j = idx & (BN - 1); k = idx >> 5; }
      const int gj = n0 + j, gk = k0 + k;
      double v = 0.0;
      if (gj < N && gk < kend)
        v = TB ? B[gj + (size_t)gk * ldb] : B[gk + (size_t)gj * ldb];
      rb[q] = v;
    }
  };
  auto store_tiles = [&]() {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int idx = tid + NT * q;
      if (!TA) As[idx >> 5][idx & (BM - 1)] = ra[q];
      else     As[idx & (BK - 1)][idx >> 4] = ra[q];
      if (!TB) Bs[idx & (BK - 1)][idx >> 4] = rb[q];
      else     Bs[idx >> 5][idx & (BN - 1)] = rb[q];
    }
  };

  double acc[2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;

  if (kbeg < kend) {
    load_a(kbeg);
    load_b(kbeg);
    for (int k0 = kbeg; k0 < kend; k0 += BK) {
      __syncthreads();
      store_tiles();
      __syncthreads();
      if (k0 + BK < kend) {
        load_a(k0 + BK);
        load_b(k0 + BK);
      }
      if (live) {
        const int kn = min(BK, kend - k0);
        auto step = [&](int k) {
          double a[2], b[4];
#pragma unroll
          for (int i = 0; i < 2; ++i) a[i] = As[k][wm + lx + 8 * i];
#pragma unroll
          for (int j = 0; j < 4; ++j) b[j] = Bs[k][wn + ly + 4 * j];
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        };
        if (kn == BK) {
#pragma unroll
          for (int k = 0; k < BK; ++k) step(k);
        } else {
          for (int k = 0; k < kn; ++k) step(k);
        }
      }
    }
  }
  if (!live) return;

  double* out = ws != nullptr ? ws + (size_t)blockIdx.z * M * N : Cm;
  const size_t ldo = ws != nullptr ? (size_t)M : (size_t)ldc;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int gj = n0 + wn + ly + 4 * j;
    if (gj >= N) continue;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int gi = m0 + wm + lx + 8 * i;
      if (gi >= M) continue;
      double* c = out + gi + (size_t)gj * ldo;
      if (ws != nullptr) *c = acc[i][j];
      else *c = (beta == 0.0) ? alpha * acc[i][j] : fma(alpha, acc[i][j], beta * *c);
    }
  }
}

// The slices' sum, in a fixed order: 32 elements per CTA, eight threads per
// element each adding every eighth slice (a single thread walking up to 256
// slices of a small output would take as long as the product), the eight
// partial sums then added in order.
constexpr int SUM_E = 32, SUM_G = 8;
__global__ void __launch_bounds__(SUM_E* SUM_G)
    dgemm_splitk_sum(int M, int N, int splits, double alpha, const double* __restrict__ ws,
                     double beta, double* __restrict__ Cm, int ldc, int upper) {
  HQ_PDL_WAIT();
  __shared__ double part[SUM_G][SUM_E];
  const size_t total = (size_t)M * N;
  const int x = threadIdx.x & (SUM_E - 1), g = threadIdx.x / SUM_E;
  for (size_t e0 = blockIdx.x * (size_t)SUM_E; e0 < total; e0 += (size_t)gridDim.x * SUM_E) {
    const size_t e = e0 + x;
    const int i = (int)(e % M), j = (int)(e / M);
    // upper: the 16 x 16 parts wholly below the diagonal were not formed.
    const bool live = e < total && !(upper && (i & ~15) >= (j & ~15) + 16);
    double s = 0.0;
    if (live) {
#pragma unroll 4
      for (int z = g; z < splits; z += SUM_G) s += ws[e + (size_t)z * total];
    }
    part[g][x] = s;
    __syncthreads();
    if (g == 0 && live) {
#pragma unroll
      for (int h = 1; h < SUM_G; ++h) s += part[h][x];
      double* c = Cm + i + (size_t)j * ldc;
      *c = (beta == 0.0) ? alpha * s : fma(alpha, s, beta * *c);
    }
    __syncthreads();
  }
}

__global__ void dgemm_scale(int M, int N, double beta, double* __restrict__ Cm, int ldc) {
  HQ_PDL_WAIT();
  const size_t total = (size_t)M * N;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(e % M), j = (int)(e / M);
    double* c = Cm + i + (size_t)j * ldc;
    *c = (beta == 0.0) ? 0.0 : beta * *c;
  }
}

// Slices of K (multiples of BK) that make the product end soonest: the SM with
// the most tiles takes ceil(tiles x slices / SMs) x (its slice of K + ~8 steps
// to start and store a tile); the slices cost a launch (~8 steps) and two
// passes over M x N x slices at ~4 TB/s.  In steps of one K of a 32 x 32 tile
// (0.25 us).  At most 256 slices, and as many as ws holds.
int plan_split(long tiles, int M, int N, int K, size_t ws_elems, int num_sms, int* kchunk) {
  int best_s = 1, best_kc = K;
  double best = 1e300;
  const int steps = (K + BK - 1) / BK;
  for (int s = 1; s <= steps && s <= 256; ++s) {
    if (s > 1 && (size_t)s * M * N > ws_elems) break;
    const int kc = (steps + s - 1) / s * BK;
    const int ss = (K + kc - 1) / kc;  // slices this chunk really gives
    const long per_sm = (tiles * ss + num_sms - 1) / num_sms;
    double cost = (double)per_sm * ((kc < K ? kc : K) + 8.0);
    if (ss > 1) cost += 8.0 + 16.0 * ss * (double)M * N / (4e6 * 0.25);
    if (cost < best) {
      best = cost;
      best_s = ss;
      best_kc = kc;
    }
    if (tiles * s > 64L * num_sms) break;  // already level
  }
  *kchunk = best_s > 1 ? best_kc : K;
  return best_s;
}

}  // namespace

extern "C" int hq_dgemm_part(cudaStream_t stream, const hq_device_info* dev, char transa,
                             char transb, int M, int N, int K, double alpha, const double* A,
                             int lda, const double* B, int ldb, double beta, double* Cm, int ldc,
                             double* ws, size_t ws_elems, int upper) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || alpha == 0.0) {
    if (beta == 1.0) return 0;
    hq_launch(dgemm_scale, dev->num_sms * 4, 256, 0, stream, M, N, beta, Cm, ldc);
    hq_count_launches(1);
    return (int)cudaGetLastError();
  }
  const bool ta = (transa == 'T' || transa == 't'), tb = (transb == 'T' || transb == 't');
  const int gm = (M + BM - 1) / BM, gn = (N + BN - 1) / BN;
  constexpr int MAX_GY = 65535;  // grid.y's limit: wider outputs take several launches
  int kchunk = K, splits = 1;
  if (ws != nullptr && gn <= MAX_GY)
    splits = plan_split((long)gm * gn, M, N, K, ws_elems, dev->num_sms, &kchunk);
  double* out_ws = splits > 1 ? ws : nullptr;
  for (int g0 = 0; g0 < gn; g0 += MAX_GY) {
    const int gw = gn - g0 < MAX_GY ? gn - g0 : MAX_GY;
    const int nw = N - g0 * BN < gw * BN ? N - g0 * BN : gw * BN;
    const double* Bw = B + (tb ? (size_t)g0 * BN : (size_t)g0 * BN * ldb);
    double* Cw = Cm + (size_t)g0 * BN * ldc;
    dim3 grid(gm, gw, splits);
    if (!ta && !tb)
      hq_launch(dgemm_tile<false, false>, grid, NT, 0, stream, M, nw, K, kchunk, alpha, A, lda, Bw,
                ldb, beta, Cw, ldc, out_ws, upper);
    else if (ta && !tb)
      hq_launch(dgemm_tile<true, false>, grid, NT, 0, stream, M, nw, K, kchunk, alpha, A, lda, Bw,
                ldb, beta, Cw, ldc, out_ws, upper);
    else if (!ta && tb)
      hq_launch(dgemm_tile<false, true>, grid, NT, 0, stream, M, nw, K, kchunk, alpha, A, lda, Bw,
                ldb, beta, Cw, ldc, out_ws, upper);
    else
      hq_launch(dgemm_tile<true, true>, grid, NT, 0, stream, M, nw, K, kchunk, alpha, A, lda, Bw,
                ldb, beta, Cw, ldc, out_ws, upper);
    hq_count_launches(1);
  }
  if (splits > 1) {
    const long total = (long)M * N;
    long blocks = (total + SUM_E - 1) / SUM_E;
    if (blocks > dev->num_sms * 32L) blocks = dev->num_sms * 32L;
    hq_launch(dgemm_splitk_sum, (unsigned)blocks, SUM_E * SUM_G, 0, stream, M, N, splits, alpha, ws,
              beta, Cm, ldc, upper);
    hq_count_launches(1);
  }
  return (int)cudaGetLastError();
}

extern "C" int hq_dgemm(cudaStream_t stream, const hq_device_info* dev, char transa, char transb,
                        int M, int N, int K, double alpha, const double* A, int lda,
                        const double* B, int ldb, double beta, double* Cm, int ldc, double* ws,
                        size_t ws_elems) {
  return hq_dgemm_part(stream, dev, transa, transb, M, N, K, alpha, A, lda, B, ldb, beta, Cm, ldc,
                       ws, ws_elems, 0);
}
