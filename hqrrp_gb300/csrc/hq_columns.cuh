// hq_columns.cuh -- device code shared by the kernels that keep whole columns of
// a pivoted Householder QR in one CTA (qrp_batched.cu, qrp_wide.cu): pivot
// candidates, and the application of a reflector to a CTA's columns.
#pragma once
#include "hq_common.cuh"

namespace {

// Larger key first, then the lower position (the upper word of at).
__device__ __forceinline__ bool better(long long k1, long long at1, long long k2, long long at2) {
  return k1 > k2 || (k1 == k2 && at1 < at2);
}

// Sums over the lanes of NY values per lane, in the lanes [32 / NY c, 32 / NY
// (c + 1)) for value c: each halving of the lanes that share a value also
// halves the values a lane keeps, so four take 2 + 1 + 3 additions.
template <int NY>
__device__ __forceinline__ double lanes_sum(const double (&d)[NY], int lane) {
  double t;
  if constexpr (NY == 4) {
    const bool up = lane & 16;
    const double a = (up ? d[2] : d[0]) + __shfl_xor_sync(0xffffffffu, up ? d[0] : d[2], 16);
    const double b = (up ? d[3] : d[1]) + __shfl_xor_sync(0xffffffffu, up ? d[1] : d[3], 16);
    const bool up8 = lane & 8;
    t = (up8 ? b : a) + __shfl_xor_sync(0xffffffffu, up8 ? a : b, 8);
  } else if constexpr (NY == 2) {
    const bool up = lane & 16;
    t = (up ? d[1] : d[0]) + __shfl_xor_sync(0xffffffffu, up ? d[0] : d[1], 16);
    t += __shfl_xor_sync(0xffffffffu, t, 8);
  } else {
    t = d[0] + __shfl_xor_sync(0xffffffffu, d[0], 16);
    t += __shfl_xor_sync(0xffffffffu, t, 8);
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// y_c -= tau (v^T y_c) v over rows s..m-1 for NY columns y_c of one warp; the
// new entries of row s go to rs[c].  CH > 0: CH steps of 32 rows cover them,
// without a branch (so every load can be issued ahead), and the columns stay in
// registers between the two uses; CH = 0: any number of rows, read twice, eight
// loads ahead (four or sixteen: 2 to 18 % slower batches).
template <int NY, int CH>
__device__ __forceinline__ void apply_warp(const double* __restrict__ v, double* const (&y)[NY],
                                           double tau, int s, int m, int lane, double* (&rs)[NY]) {
  double d[NY];
#pragma unroll
  for (int c = 0; c < NY; ++c) d[c] = 0.0;
  if constexpr (CH > 0) {
    double x[NY][CH];
#pragma unroll
    for (int t = 0; t < CH; ++t) {
      const int i = s + lane + 32 * t;
#pragma unroll
      for (int c = 0; c < NY; ++c) x[c][t] = i < m ? y[c][i] : 0.0;
    }
#pragma unroll
    for (int t = 0; t < CH; ++t) {
      const int i = s + lane + 32 * t;
      const double vi = i < m ? v[i] : 0.0;
#pragma unroll
      for (int c = 0; c < NY; ++c) d[c] = fma(vi, x[c][t], d[c]);
    }
    const double t = lanes_sum<NY>(d, lane) * -tau;
    double w[NY];
#pragma unroll
    for (int c = 0; c < NY; ++c) w[c] = __shfl_sync(0xffffffffu, t, 32 / NY * c);
#pragma unroll
    for (int t2 = 0; t2 < CH; ++t2) {
      const int i = s + lane + 32 * t2;
      const double vi = i < m ? v[i] : 0.0;
#pragma unroll
      for (int c = 0; c < NY; ++c) {
        const double z = fma(vi, w[c], x[c][t2]);
        if (i < m) y[c][i] = z;
        if (t2 == 0 && lane == 0) *rs[c] = z;
      }
    }
  } else {
#pragma unroll 8
    for (int i = s + lane; i < m; i += 32) {
      const double vi = v[i];
#pragma unroll
      for (int c = 0; c < NY; ++c) d[c] = fma(vi, y[c][i], d[c]);
    }
    const double t = lanes_sum<NY>(d, lane) * -tau;
    double w[NY];
#pragma unroll
    for (int c = 0; c < NY; ++c) w[c] = __shfl_sync(0xffffffffu, t, 32 / NY * c);
#pragma unroll 8
    for (int i = s + lane; i < m; i += 32) {
      const double vi = v[i];
#pragma unroll
      for (int c = 0; c < NY; ++c) {
        const double z = fma(vi, w[c], y[c][i]);
        y[c][i] = z;
        if (i == s) *rs[c] = z;
      }
    }
  }
}

template <int NY, int CH>
struct Take {
  static constexpr int ny = NY, ch = CH;
};

// Columns act[0..cnt) (local indices; colp gives a column's address) of a CTA
// of NW warps: X[s:, k] -= tau v (v^T X[s:, k]), the new entries of row s to
// row.  A warp takes four, two or one column together, as its registers hold
// of this many rows (256, 512, 1024).  More together need fewer FP64
// instructions -- with S steps of 32 rows 8 S + 7 for four, 4 S + 6 for two, 2 S
// + 6 for one -- but spread over fewer quarters of the SM, each of which issues
// one every 64 clocks: the choice is what the busiest quarter issues.  Longer
// columns are read twice, and one at a time: the second reading of one column a
// warp still finds it in the L1 cache, of four it does not (400 matrices of 2000
// x 64: 12.0 ms, with four a warp 16.6; 150 of 4000 x 40: 3.9 and 7.3).  LEAN:
// few registers a thread, every column is read twice.
template <int NW, bool LEAN = false, typename ColP>
__device__ __forceinline__ void apply_columns(const double* v, double tau, int s, int m, int cnt,
                                              const int* act, double* row, ColP colp, int warp,
                                              int lane) {
  auto apply = [&](auto take, int j) {
    constexpr int NY = decltype(take)::ny;
    double* y[NY];
    double* rs[NY];
#pragma unroll
    for (int c = 0; c < NY; ++c) {
      const int q = act[j + c];
      y[c] = colp(q);
      rs[c] = row + q;
    }
    apply_warp<NY, decltype(take)::ch>(v, y, tau, s, m, lane, rs);
  };
  // Groups of NY columns to warps 0, 1, ...; what is left singly to the next.
  auto apply_all = [&](auto many, auto single) {
    constexpr int NY = decltype(many)::ny;
    const int groups = cnt / NY;
    for (int g = warp; g < groups; g += NW) apply(many, NY * g);
    if constexpr (NY > 1) {
      const int j = groups * NY + (warp - groups % NW + NW) % NW;
      if (j < cnt) apply(single, j);
    }
  };
  if constexpr (LEAN) {
    apply_all(Take<1, 0>{}, Take<1, 0>{});
    return;
  }
#define HQ_MANY(NY, CH) apply_all(Take<NY, CH>{}, Take<1, CH>{}); break;
  const int S = (m - s + 31) >> 5;
  const int t1 = ((cnt + 3) >> 2) * (2 * S + 6);
  const int t2 = S > 16 ? t1 : (((cnt >> 1) + (cnt & 1) + 3) >> 2) * (4 * S + 6);
  const int t4 = S > 8 ? t1 : (((cnt >> 2) + (cnt & 3) + 3) >> 2) * (8 * S + 7);
  if (S > 32) {
    apply_all(Take<1, 0>{}, Take<1, 0>{});
  } else if (t4 < t1 && t4 <= t2) {
    switch (S) {
      case 1: HQ_MANY(4, 1)
      case 2: HQ_MANY(4, 2)
      case 3: HQ_MANY(4, 3)
      case 4: HQ_MANY(4, 4)
      case 5: HQ_MANY(4, 5)
      case 6: HQ_MANY(4, 6)
      case 7: HQ_MANY(4, 7)
      default: HQ_MANY(4, 8)
    }
  } else if (t2 < t1) {
    switch ((S + 1) >> 1) {
      case 1: HQ_MANY(2, 2)
      case 2: HQ_MANY(2, 4)
      case 3: HQ_MANY(2, 6)
      case 4: HQ_MANY(2, 8)
      case 5: HQ_MANY(2, 10)
      case 6: HQ_MANY(2, 12)
      case 7: HQ_MANY(2, 14)
      default: HQ_MANY(2, 16)
    }
  } else {
    switch ((S - 1) >> 1) {
      case 0: HQ_MANY(1, 2)
      case 1: HQ_MANY(1, 4)
      case 2: HQ_MANY(1, 6)
      case 3: HQ_MANY(1, 8)
      case 4: case 5: HQ_MANY(1, 12)
      case 6: case 7: HQ_MANY(1, 16)
      case 8: case 9: HQ_MANY(1, 20)
      case 10: case 11: HQ_MANY(1, 24)
      case 12: case 13: HQ_MANY(1, 28)
      default: HQ_MANY(1, 32)
    }
  }
#undef HQ_MANY
}

// Sum of squares of x over rows (s, m) by the threads t < nd of some warps: each
// warp's part in every lane of it.
__device__ __forceinline__ double tail_squares(const double* x, int s, int m, int t, int nd) {
  double sum = 0.0;
  for (int i0 = s + 1 + t; i0 - t < m; i0 += 8 * nd) {
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = i0 + k * nd < m ? x[i0 + k * nd] : 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (i0 - t + k * nd < m) sum = fma(v[k], v[k], sum);  // uniform
  }
  return hq_warp_sum(sum);
}

// The warp's best candidate (largest key, then lowest position, the upper word
// of at) to *bk, *ba; keys are >= -3.  Three integer reductions.
__device__ __forceinline__ void warp_best(long long k, long long at, long long* bk,
                                          long long* ba) {
  const unsigned long long u = (unsigned long long)(k + 4);
  const unsigned hi = (unsigned)(u >> 32);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = hi == mh ? (unsigned)u : 0u;
  const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
  const bool mine = hi == mh && (unsigned)u == ml;
  const int p = (int)(at >> 32);
  const int bp = __reduce_min_sync(0xffffffffu, mine ? p : 0x7fffffff);
  if (mine && p == bp) {
    *bk = k;
    *ba = at;
  }
}

}  // namespace
