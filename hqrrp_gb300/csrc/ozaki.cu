// ozaki.cu -- FP64 products on the BF16 tensor cores (tcgen05), split-digit
// ("Ozaki scheme I") emulation, for the mixed-precision block updates.
//
// Each operand row r (a row of the M-side matrix, or a column of the output
// on the N side) gets a power-of-two scale 2^e_r >= max |x|, and every entry
// is written as S balanced base-256 digits:
//     x = 2^e_r * sum_s d_s * 2^(-7-8s) (+ a remainder below 2^(e_r - 8S)),
// with integer digits |d_s| <= 128, each exact in BF16.  The product of a
// digit pair is an integer of at most 2^14 in the pair's unit, so a tensor-
// core FP32 accumulation of up to 2^24 / (2^14 * pairs) terms is exact.  Pairs
// are grouped by level L = s + t (unit 2^(-14-8L)), and only pairs with
// L <= S-1 are formed (the rest are below the dropped remainder).  Digit s is
// stored pre-scaled by 2^(-8s) (exact in BF16), so every product already
// carries its level's weight.  Levels 0..3 each get a TMEM accumulator, exact
// per 256-deep slice of K (integers below 2^24 in their unit); level 4 gets its
// own; levels 5 and 6 need at most 2^-12 relative precision and share one.
// All are drained every 256 K into running sums: float-float (FP32 pairs, ~48
// bits), or 64-bit integers where K is at most 256.  (Folding level 4 in as well measured 2^-47.5 instead of 2^-52: the
// tensor core's FP32 accumulation loses more than IEEE rounding when products
// of very different magnitude meet in one accumulator.)  Six accumulators
// instead of seven leave TMEM room for 80-column tiles.  The
// result is recombined in FP64.  With S = 7 the product is accurate to about
// 2^-52 relative to |A| |B| row/column-wise.
//
// Layout: the split writes each operand as the tiles the MMA descriptors
// read: for each row tile and block of 32 K, S digit tiles of (tile rows) x 64
// bytes one after the other, 64-byte swizzled (16-byte chunk c of row r at
// chunk c ^ ((r >> 1) & 3); 8-row atoms of 512 B).  So a pipeline stage is one
// contiguous bulk copy per operand; a tensor-map box of 64-byte rows out of
// plain K-major digit matrices took a tenth longer per tile of a short product.
// M tile 128 rows, N tile 80, K block 32.
//
// The GEMM kernels are warp-specialised: warp 20 issues the bulk copies into a
// 3-stage (2 for seven digits) ring, one thread of warp 21 issues tcgen05.mma
// (cta_group::1, kind::f16, 128 x 80..240 x 16) into TMEM, warps 0-19 drain TMEM
// (tcgen05.ld, five warps per 32-lane quadrant, 16 columns each) and write
// the output.  Every wait is bounded; on expiry the
// kernel records an error, waits (bounded) for its in-flight copies and MMAs,
// frees its TMEM and returns.
#include <cuda.h>
#include <cudaTypedefs.h>

#include "hq_common.cuh"

namespace {

constexpr int TM = 128, TN = 80, TK = 32;  // six accumulators x 80 = 480 TMEM columns
constexpr int TN_SHORT = TN;  // the short-K kernel uses the same N tiles
constexpr int MAX_STAGES = 3;
constexpr int KB_PER_DRAIN = 8;  // 256 K elements
constexpr int MAX_ACC = 6;  // levels 0..4 alone (0..3 exact), 5 and 6 shared

__host__ __device__ constexpr int n_acc(int S) { return S < MAX_ACC ? S : MAX_ACC; }
__host__ __device__ inline uint32_t tmem_pow2(uint32_t c) {
  return c <= 32 ? 32u : (c <= 64 ? 64u : (c <= 128 ? 128u : (c <= 256 ? 256u : 512u)));
}
// Warps 0-19 epilogue (five per TMEM lane quadrant, each a fifth of the
// tile's columns), warp 20 producer, warp 21 MMA.  The epilogue is latency-
// bound (FP64 adds, C loads, TMEM loads): five warps per quadrant instead of
// two hide it -- 257 -> 206 ms of tensor-phase time per 16384^2 mixed
// factorization -- at 80 registers per thread.
constexpr int NT = 704;
constexpr int NEPI = 640;
constexpr int PRODUCER_WARP = 20, MMA_WARP = 21;
constexpr int EPI_COLS = TN / 5;  // columns per epilogue thread (a multiple of 8)
static_assert(TN % 5 == 0 && EPI_COLS % 8 == 0, "epilogue columns come in TMEM loads of 8");
constexpr int A_TILE = TM * TK * 2;  // 8 KB per digit tile
constexpr int B_TILE = TN * TK * 2;  // 5 KB per digit tile

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// ---------------------------------------------------------------------------
// Split

// One FP64 entry's balanced base-256 digits in one word: W = V + 128 *
// sum_p 256^p, where V = round(x * 2^(8S - 1 - e)) is the fixed-point integer
// of a row of scale 2^e, |V| <= 2^(8S-1) (zeros, subnormals, infinities and
// NaNs give V = 0).  Digit p < S-1 is byte p of W minus 128 and the top digit
// W >> 8(S-1) minus 128 -- the same digits as peeling them from the bottom.
// shift_base = 8S - 1076 - e, so V = mantissa * 2^(exponent field + shift_base);
// the shift left by 3 leaves only right shifts, and one bit more than V to
// round by.  The integer pipe is what bounds the conversions (the products
// that cut their digits themselves spend as long on this as on their MMAs), so
// this and digit_pair are written for few of its instructions.
template <int S>
__device__ __forceinline__ unsigned long long digit_word(double x, int shift_base) {
  constexpr unsigned long long BIAS = 0x8080808080808080ULL >> (8 * (8 - S));
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  const int ex = (hi >> 20) & 0x7FF;
  unsigned r = (unsigned)(2 - shift_base - ex);
  if ((unsigned)(ex - 1) >= 2046u || r > 63u) r = 63u;
  const unsigned mh = ((unsigned)hi & 0xFFFFFu) | 0x100000u;
  const unsigned long long m = ((unsigned long long)((mh << 3) | (lo >> 29)) << 32) | (lo << 3);
  const unsigned long long v = ((m >> r) + 1ull) >> 1;
  const long long neg = hi >> 31;
  return (v ^ (unsigned long long)neg) + (BIAS - (unsigned long long)neg);
}

// Digits S-1-s of two words, times 2^(-8s), as a pair of BF16: the FP32
// pattern with exponent 23 - 8s and mantissa u is 2^(23-8s) + u 2^(-8s)
// exactly, and subtracting 2^(23-8s) + 128 2^(-8s) (exact in FP32) leaves
// (u - 128) 2^(-8s), exact in BF16, in one byte permutation and one addition.
template <int S>
__device__ __forceinline__ uint32_t digit_pair(unsigned long long w0, unsigned long long w1,
                                               int s) {
  const int p = S - 1 - s;
  const uint32_t base = (uint32_t)(150 - 8 * s) << 23;  // only its top byte is set
  uint32_t f0, f1;
  if (s == 0) {  // the top digit: up to 9 bits
    f0 = base | (uint32_t)(w0 >> (8 * p));
    f1 = base | (uint32_t)(w1 >> (8 * p));
  } else {
    f0 = __byte_perm((uint32_t)(w0 >> (32 * (p / 4))), base, 0x7540 | (p & 3));
    f1 = __byte_perm((uint32_t)(w1 >> (32 * (p / 4))), base, 0x7540 | (p & 3));
  }
  const float off = __uint_as_float(base | 128u);
  const uint32_t d0 = __float_as_uint(__fsub_rn(__uint_as_float(f0), off));
  const uint32_t d1 = __float_as_uint(__fsub_rn(__uint_as_float(f1), off));
  return __byte_perm(d0, d1, 0x7632);
}

// The S digits of entries 8 ch .. 8 ch + 7 of row r, one 16-byte store each,
// in the tile layout.
template <int S>
__device__ __forceinline__ void put_digits(const unsigned long long (&W)[8], uint8_t* tiles, int r,
                                           int ch, int TR, int KB) {
  const int rt = r / TR, ri = r - rt * TR;
  uint8_t* base = tiles + ((long long)rt * KB + (ch >> 2)) * (S * TR * (TK * 2)) + ri * (TK * 2) +
                  (((ch & 3) ^ ((ri >> 1) & 3)) << 4);
#pragma unroll
  for (int s = 0; s < S; ++s)
    *reinterpret_cast<uint4*>(base + s * (TR * (TK * 2))) =
        make_uint4(digit_pair<S>(W[0], W[1], s), digit_pair<S>(W[2], W[3], s),
                   digit_pair<S>(W[4], W[5], s), digit_pair<S>(W[6], W[7], s));
}

// Rows r < R of X (element (r, k) at X[r*rs + k*ks], k < K) -> S digit tiles.
// One warp per row; each lane takes 8-element chunks (one 16-byte group of a
// tile row), so every digit is written with one 16-byte store.  Rows
// R..RT*TR-1 and k >= K are written as zeros.  Slice s holds digit p = S-1-s,
// the most significant first.
template <int S>
__global__ void ozk_split_kernel(const double* __restrict__ X, long long rs, long long ks, int R,
                                 int K, int TR, int KB, int rows_total,
                                 uint8_t* __restrict__ tiles, int* __restrict__ exps) {
  HQ_PDL_WAIT();
  const int lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5;
  const int nchunk = KB * (TK / 8);
  for (int r = blockIdx.x * warps + (threadIdx.x >> 5); r < rows_total;
       r += gridDim.x * warps) {
    const bool live = r < R;
    const double* xr = X + (live ? (long long)r * rs : 0);
    // Largest magnitude from the bit patterns (integer compares).
    long long mb = 0;
    if (live)
      for (int k = lane; k < K; k += 32) {
        const long long bb = __double_as_longlong(xr[(long long)k * ks]) & 0x7FFFFFFFFFFFFFFFLL;
        mb = bb > mb ? bb : mb;
      }
    for (int o = 16; o > 0; o >>= 1) {
      const long long ob = __shfl_xor_sync(0xffffffffu, mb, o);
      mb = ob > mb ? ob : mb;
    }
    // 2^e > max |x| >= 2^(e-1); 0 for zero or subnormal rows.
    const int bexp = (int)(mb >> 52);
    const int e = bexp == 0 ? 0 : bexp - 1022;
    if (lane == 0) exps[r] = e;
    const int shift_base = 8 * S - 1076 - e;
    for (int ch = lane; ch < nchunk; ch += 32) {
      const int k0 = ch * 8;
      unsigned long long W[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        W[j] = digit_word<S>((live && k0 + j < K) ? xr[(long long)(k0 + j) * ks] : 0.0, shift_base);
      }
      put_digits<S>(W, tiles, r, ch, TR, KB);
    }
  }
}

// Column-major operand with short rows (row stride 1, K <= CM_KMAX, e.g. a
// panel's rows with K = its columns): reading a row walks a column stride
// per entry, so a CTA first stages 32 consecutive rows x K in shared memory
// with coalesced loads (one warp load = 32 consecutive rows of one column),
// then splits each row exactly as ozk_split_kernel does (same digits and
// exponents), the maxima one warp per row, the digits four lanes a tile row.
constexpr int CM_KMAX = 128;
template <int S>
__global__ void __launch_bounds__(256) ozk_split_cm_kernel(const double* __restrict__ X,
                                                           long long ks, int R, int K, int TR,
                                                           int KB, int rows_total,
                                                           uint8_t* __restrict__ tiles,
                                                           int* __restrict__ exps) {
  HQ_PDL_WAIT();
  __shared__ double tile[CM_KMAX][33];
  __shared__ int s_e[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r0 = blockIdx.x * 32;
  for (int k = warp; k < K; k += 8) {
    const int r = r0 + lane;
    tile[k][lane] = r < R ? X[(long long)r + (long long)k * ks] : 0.0;
  }
  __syncthreads();
  for (int rr = warp; rr < 32; rr += 8) {
    const int r = r0 + rr;
    if (r >= rows_total) break;
    long long mb = 0;
    for (int k = lane; k < K; k += 32) {
      const long long bb = __double_as_longlong(tile[k][rr]) & 0x7FFFFFFFFFFFFFFFLL;
      mb = bb > mb ? bb : mb;
    }
    for (int o = 16; o > 0; o >>= 1) {
      const long long ob = __shfl_xor_sync(0xffffffffu, mb, o);
      mb = ob > mb ? ob : mb;
    }
    const int bexp = (int)(mb >> 52);
    const int e = bexp == 0 ? 0 : bexp - 1022;
    if (lane == 0) exps[r] = s_e[rr] = e;
  }
  __syncthreads();
  for (int it = threadIdx.x; it < KB * 128; it += 256) {
    const int rr = (it >> 2) & 31, ch = (it >> 7) * 4 + (it & 3), r = r0 + rr;
    if (r >= rows_total) continue;
    const int shift_base = 8 * S - 1076 - s_e[rr];
    unsigned long long W[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      W[j] = digit_word<S>(ch * 8 + j < K ? tile[ch * 8 + j][rr] : 0.0, shift_base);
    put_digits<S>(W, tiles, r, ch, TR, KB);
  }
}

// Largest exponent field of each row, several CTAs per row (ROWMAX_SPAN
// entries each, eight loads in flight per thread) raising raw[r] -- zeroed
// before -- with an integer atomicMax: the first pass of the split of long
// rows.
constexpr int ROWMAX_SPAN = 2048;
__global__ void __launch_bounds__(256) ozk_rowmax_atomic_kernel(const double* __restrict__ X,
                                                                long long rs, long long ks, int K,
                                                                int* __restrict__ raw) {
  HQ_PDL_WAIT();
  __shared__ long long s_max[8];
  const int r = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int k0 = blockIdx.y * ROWMAX_SPAN;
  const double* xr = X + (long long)r * rs;
  long long v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int k = k0 + tid + 256 * i;
    v[i] = k < K ? (__double_as_longlong(xr[(long long)k * ks]) & 0x7FFFFFFFFFFFFFFFLL) : 0;
  }
  long long mb = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) mb = v[i] > mb ? v[i] : mb;
  for (int o = 16; o > 0; o >>= 1) {
    const long long ob = __shfl_xor_sync(0xffffffffu, mb, o);
    mb = ob > mb ? ob : mb;
  }
  if (lane == 0) s_max[warp] = mb;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < 8; ++w) mb = s_max[w] > mb ? s_max[w] : mb;
    mb = s_max[0] > mb ? s_max[0] : mb;
    if (mb != 0) atomicMax(raw + r, (int)(mb >> 52));
  }
}

// The same for column-major operands (row stride 1): 32 rows a CTA, a row a
// lane, so that a warp's loads are contiguous.
constexpr int ROWMAX_CM_SPAN = 512;
__global__ void __launch_bounds__(256) ozk_rowmax_cm_kernel(const double* __restrict__ X,
                                                            long long ks, int R, int K,
                                                            int* __restrict__ raw) {
  HQ_PDL_WAIT();
  __shared__ int s_max[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = blockIdx.x * 32 + lane;
  const int k1 = min(K, (int)(blockIdx.y + 1) * ROWMAX_CM_SPAN);
  int m = 0;
  if (r < R) {
    const int* xr = reinterpret_cast<const int*>(X + r) + 1;  // the upper word
#pragma unroll 8
    for (int k = blockIdx.y * ROWMAX_CM_SPAN + warp; k < k1; k += 8)
      m = max(m, (xr[(long long)k * ks * 2] >> 20) & 0x7FF);
  }
  s_max[warp][lane] = m;
  __syncthreads();
  if (warp == 0 && r < R) {
#pragma unroll
    for (int w = 1; w < 8; ++w) m = max(m, s_max[w][lane]);
    if (m != 0) atomicMax(raw + r, m);
  }
}

// Long rows: with the rows' largest exponent fields known (from the kernels
// above, or from the epilogue of the update that wrote X), every 8-element
// chunk independently -- a warp takes a K block of 8 rows: 256-byte loads (64
// down a column), 512-byte digit stores per slice.
template <int S>
__global__ void __launch_bounds__(256) ozk_split_chunk_kernel(
    const double* __restrict__ X, long long rs, long long ks, int R, int K, int TR, int KB,
    int rows_total, uint8_t* __restrict__ tiles, int* __restrict__ exps,
    const int* __restrict__ raw) {
  HQ_PDL_WAIT();
  static_assert(TK == 32, "four chunks a K block");
  const long long total = (long long)rows_total * KB * (TK / 8);
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long grp = idx >> 5;  // K block kb of 8 rows
    const int kb = (int)(grp % KB), r = (int)(grp / KB) * 8 + (((int)idx >> 2) & 7);
    const int ch = kb * 4 + ((int)idx & 3), k0 = ch * 8;
    const bool live = r < R;
    const double* xr = X + (live ? (long long)r * rs : 0);
    const int bexp = live ? raw[r] : 0;
    const int e = bexp == 0 ? 0 : bexp - 1022;
    if (ch == 0) exps[r] = e;
    const int shift_base = 8 * S - 1076 - e;
    double v[8];
    if (live && ks == 1 && k0 + 8 <= K && ((reinterpret_cast<uintptr_t>(xr + k0) & 15) == 0)) {
      const double2* p2 = reinterpret_cast<const double2*>(xr + k0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double2 d = p2[j];
        v[2 * j] = d.x;
        v[2 * j + 1] = d.y;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = (live && k0 + j < K) ? xr[(long long)(k0 + j) * ks] : 0.0;
    }
    unsigned long long W[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) W[j] = digit_word<S>(v[j], shift_base);
    put_digits<S>(W, tiles, r, ch, TR, KB);
  }
}

// ---------------------------------------------------------------------------
// GEMM

struct OzkArgs {
  const uint8_t* A;  // M-side tiles [MT][KB][S][TM x TK], 16-byte aligned
  const uint8_t* B;  // N-side tiles [NTL][KB][S][TN x TK], 16-byte aligned
  const int* ea;
  const int* eb;
  int M, N, S, KB;
  int kb_per_z;  // K blocks per grid.z slice (multiple of KB_PER_DRAIN)
  int mode;      // 0: out = sign * A B^T (per z slice); 1: C += sign * A B^T
  double* C;
  long long crs, ccs;  // element (r, c) at C[r*crs + c*ccs]
  long long zstride;   // mode 0, gridDim.z > 1: slice z writes at C + z*zstride
  double sign;
  int stages;  // 2 or 3, whatever fits in shared memory
  int* err;
  unsigned spin_limit;
  // Short kernel, mode 1: when set, colexp[c] gets the largest exponent field
  // of the new C over rows >= row_lo of column c (atomicMax; zeroed before).
  int* colexp;
  int row_lo;
  // FP64 N-side operand (ozk_gemm_c64_kernel): eb_raw[n] is column n's
  // largest exponent field, from which its scale exponent follows (eb unused).
  const int* eb_raw;
};

// The scale exponent of a row whose largest exponent field is raw: 2^e >
// max |x| >= 2^(e-1), 0 for a zero row.
__device__ __forceinline__ int scale_of_raw(int raw) { return raw == 0 ? 0 : raw - 1022; }

__device__ __forceinline__ void mbar_init(uint64_t* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count));
}

__device__ __forceinline__ bool mbar_wait(uint64_t* b, unsigned parity, unsigned limit,
                                          volatile int* abort_flag) {
  for (unsigned it = 0; it < limit; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    if (ok) return true;
    if (abort_flag && *abort_flag) return false;
  }
  return false;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}

// mbar_wait by a whole warp, with one outcome.
__device__ __forceinline__ bool warp_wait(uint64_t* b, unsigned parity, unsigned limit,
                                          volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait(b, parity, limit, abort_flag));
}

// The warp's index, known to be the same in all its lanes.
__device__ __forceinline__ int uniform_warp() {
  return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
}

// One arrival for the warp, after all its lanes.
__device__ __forceinline__ void warp_arrive(uint64_t* b, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(b);
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)),
               "r"(bytes)
               : "memory");
}

// bytes (a multiple of 16, both addresses 16-byte aligned) into shared memory,
// completing on the mbarrier.
__device__ __forceinline__ void bulk_load(void* dst, const uint8_t* src, unsigned bytes,
                                          uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ uint64_t sw64_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;               // LBO, unused for swizzled K-major
  d |= (uint64_t)(512 >> 4) << 32;      // SBO: 8 rows x 64 B
  d |= (uint64_t)1 << 46;               // descriptor version for tcgen05
  d |= (uint64_t)4 << 61;               // 64-byte swizzle
  return d;
}

// The MMA warp runs as a whole and elects the thread that issues (always the
// same one): its operands are then known to be uniform.  One thread on its own
// took 3200 clocks to issue a K block's MMAs beside busy converting warps,
// which take 2650.
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t ad, uint64_t bd, uint32_t idesc,
                                         uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n elect.sync _|q, 0xffffffff;\n"
      " @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* b) {
  asm volatile(
      "{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n"
      " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(
          smem_u32(b))
      : "memory");
}

// (hi, lo) += x in FP32 pairs (TwoSum, then renormalise).
__device__ __forceinline__ void ff_add(float& hi, float& lo, float x) {
  const float s = __fadd_rn(hi, x);
  const float bb = __fsub_rn(s, hi);
  const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(x, bb));
  const float l = __fadd_rn(lo, e);
  const float h = __fadd_rn(s, l);
  lo = __fsub_rn(l, __fsub_rn(h, s));
  hi = h;
}

// An FP32 value times 2^ek (negated when neg) as an FP64, assembled from the
// bits on the integer pipe -- the FP64 pipe is this GPU's scarce resource and
// the epilogue of a short-K product would otherwise be bound by it.  Exact for
// FP32 normals; zero and FP32 subnormals give 0, and so do results below the
// FP64 normal range (negligible next to the rest of the sum).
__device__ __forceinline__ double f32_scaled(float f, int ek, unsigned neg) {
  const unsigned b = __float_as_uint(f);
  const int ex = (int)((b >> 23) & 0xFF);
  const int e64 = ex - 127 + 1023 + ek;
  const unsigned long long bits = ((unsigned long long)((b >> 31) ^ neg) << 63) |
                                  ((unsigned long long)(e64 & 0x7FF) << 52) |
                                  ((unsigned long long)(b & 0x7FFFFF) << 29);
  return (ex == 0 || e64 <= 0) ? 0.0 : __longlong_as_double(bits);
}

// 16 consecutive TMEM columns of this warp's 32 lanes (one load, one wait).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15}, [%16];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

// The accumulators change hands in groups of ACC_GROUP, the first levels'
// first: the MMAs finish them in that order (issue_block), each with a commit
// on full[g], and the epilogue warps give each back on empty[g] as soon as it
// is read.  So the first groups are drained while the last one is still being
// added to, and the next MMAs start on the first ones while the last is
// drained; handed over in one piece the tensor core idled through every drain.
// A group is what one MMA can cover: three levels.  Over a 16384^2 mixed
// factorization the products took 218 ms with one level an MMA, 188 with two
// and 180 with three.
constexpr int ACC_GROUP = 3;
constexpr int MAX_GROUPS = MAX_ACC / ACC_GROUP;
static_assert(MAX_ACC % ACC_GROUP == 0 && ACC_GROUP * TN <= 256, "one MMA covers a group");
struct Handover {
  uint64_t* full;   // [MAX_GROUPS]
  uint64_t* empty;  // [MAX_GROUPS]
};

// Drains the nacc accumulators of this warp's 16 columns, take(q, values), as
// the round'th use of the barriers; false (in every lane) if a wait gave up.
template <typename Take>
__device__ __forceinline__ bool drain_levels(uint32_t tacc, int nacc, Handover h, int round,
                                             unsigned lim, volatile int* abort_flag, int lane,
                                             Take take) {
  static_assert(EPI_COLS == 16, "one 16-column load per accumulator");
#pragma unroll
  for (int q = 0; q < MAX_ACC; ++q) {
    if (q >= nacc) continue;
    const int g = q / ACC_GROUP;
    if (q % ACC_GROUP == 0) {
      // One outcome per warp: TMEM loads are warp-wide.
      if (!warp_wait(&h.full[g], round & 1, lim, abort_flag)) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    float v[16];
    tmem_ld16(tacc + (uint32_t)(q * TN), v);
    if (q % ACC_GROUP == ACC_GROUP - 1 || q == nacc - 1) {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      warp_arrive(&h.empty[g], lane);
    }
    take(q, v);
  }
  return true;
}

// The running sums of a thread's 16 outputs.  Over any K: float-float pairs
// (FloatSums).  Over K <= 256 (ExactSums): integers in units of 2^-48, level
// 6's -- the accumulators of levels 0 to 4 are integers in their own units, the
// one that levels 5 and 6 share is a multiple of level 6's, and all of them
// together stay below 2^71.  A 64-bit integer holds the sum down to 2^-40,
// level 5's unit, and a byte the 8 bits below it, so nothing that the tensor
// core hands over is dropped, however small the product is beside its row's and
// column's scales; one rounding to FP64 is left.  That takes fewer instructions
// an accumulator than a float-float addition, makes the FP64 value on the
// integer pipe, which leaves one FP64 addition an output instead of two, and
// errs no more: 1.8e-16 to 2.1e-16 of the product's norm against 6.0e-16 for
// Gaussian operands of K = 64 to 256, and the same where the operands are graded
// in opposite directions along K (K = 4 to 256), whose results are far below
// their scales.  (Without the byte those erred up to 1.5 times as much; it takes
// the 8192 x 8192 x 128 update from 0.398 to 0.420 ms -- 0.600 with
// float-float sums and an MMA a level.)
struct FloatSums {
  float hi[EPI_COLS], lo[EPI_COLS];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int c = 0; c < EPI_COLS; ++c) hi[c] = lo[c] = 0.f;
  }
  __device__ __forceinline__ void add(int, const float* v) {
#pragma unroll
    for (int c = 0; c < EPI_COLS; ++c) ff_add(hi[c], lo[c], v[c]);
  }
  // sign * sum * 2^ek: the two exact conversions take no FP64 instruction,
  // their sum one (exact: hi + lo fits in FP64).
  __device__ __forceinline__ double value(int c, int ek, unsigned neg) const {
    return f32_scaled(hi[c], ek, neg) + f32_scaled(lo[c], ek, neg);
  }
};

struct ExactSums {
  long long sum[EPI_COLS];
  uint32_t rest[EPI_COLS / 4];  // a byte an output
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int c = 0; c < EPI_COLS; ++c) sum[c] = 0;
#pragma unroll
    for (int c = 0; c < EPI_COLS / 4; ++c) rest[c] = 0u;
  }
  // q: a constant once unrolled.  Levels 0 and 1 only touch the upper word;
  // the others are wide multiply-adds, off the integer pipe.
  __device__ __forceinline__ void add(int q, const float* v) {
    const float unit = __uint_as_float((uint32_t)(127 + 8 * q) << 23);
#pragma unroll
    for (int c = 0; c < EPI_COLS; ++c) {
      float t = v[c] * unit;
      if (q == MAX_ACC - 1) {
        // Rounded down; 256 times the rest is an integer below 256, and the
        // lowest byte of that plus 2^23.
        const float f = floorf(t);
        const uint32_t r = __float_as_uint(fmaf(t - f, 256.f, 8388608.f));
        rest[c / 4] = __byte_perm(rest[c / 4], r, c % 4 == 0   ? 0x3214
                                                  : c % 4 == 1 ? 0x3240
                                                  : c % 4 == 2 ? 0x3410
                                                               : 0x4210);
        t = f;
      }
      const int i = __float2int_rn(t);
      if (q < 2)
        sum[c] += (long long)((unsigned long long)(unsigned)(q == 0 ? i * 256 : i) << 32);
      else
        asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(sum[c]) : "r"(i), "r"(1 << (40 - 8 * q)));
    }
  }
  // sign * sum * 2^(ek - 40), rounded to FP64 (half away from zero); results
  // below the FP64 normal range give 0.
  __device__ __forceinline__ double value(int c, int ek, unsigned neg) const {
    // The byte below is appended where the result is one word long with it, and
    // rounded off where it is below a quarter of the result's last place.
    const unsigned below = rest[c / 4] >> (8 * (c % 4)) & 0xFFu;
    const bool fits = (unsigned)((int)(sum[c] >> 32) + 0x400000) < 0x800000u;  // |sum| < 2^54
    const long long v = fits ? (long long)((unsigned long long)sum[c] << 8 | below)
                             : sum[c] + (long long)(below >> 7);
    const unsigned long long u = (unsigned long long)(v < 0 ? -v : v);
    unsigned h = (unsigned)(u >> 32), l = (unsigned)u;
    int e = ek + (fits ? 1037 : 1045);  // biased exponent - 1 of a leading bit 63
    const bool low = h == 0u;
    h = low ? l : h;
    l = low ? 0u : l;
    e -= low ? 32 : 0;
    const int z = __clz((int)h);
    h = __funnelshift_l(l, h, z);
    l <<= z & 31;
    e -= z;
    const unsigned sign = ((unsigned)((unsigned long long)v >> 32) ^ (neg << 31)) & 0x80000000u;
    const unsigned ml = __funnelshift_r(l, h, 11);
    // The mantissa's leading bit (bit 20 of h >> 11) adds the 1 to e.
    const unsigned long long bits =
        (((unsigned long long)((h >> 11) + (unsigned)e * 0x100000u + sign) << 32) | ml) +
        ((l >> 10) & 1u);
    // No bit set, or below or above FP64's normal range.
    const bool none = (int)h >= 0 || e < 0, inf = e >= 2046;
    const unsigned bh = none ? 0u : (inf ? sign | 0x7FF00000u : (unsigned)(bits >> 32));
    return __hiloint2double((int)bh, none || inf ? 0 : (int)(unsigned)bits);
  }
};

// Raises colexp[n0 + c], c < EPI_COLS, to the largest exponent field over the
// warp's rows: w[i] holds columns 2i and 2i+1, each exponent field at bits
// 4..14 of its half.  Halving the columns with each exchange takes 9 shuffles
// and one atomic instruction where a reduction a column took 16 of each.
__device__ __forceinline__ void raise_exponents(uint32_t (&w)[EPI_COLS / 2], int* colexp, int n0,
                                                int N, int lane) {
#pragma unroll
  for (int h = EPI_COLS / 4; h >= 1; h >>= 1) {
    const int o = 4 * h;
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? w[i] : w[i + h], o);
      w[i] = __vmaxu2(up ? w[i + h] : w[i], got);
    }
  }
  w[0] = __vmaxu2(w[0], __shfl_xor_sync(0xffffffffu, w[0], 2));
  w[0] = __vmaxu2(w[0], __shfl_xor_sync(0xffffffffu, w[0], 1));
  const int n = n0 + 2 * (lane >> 2) + (lane & 1);
  const int m = (int)(((lane & 1) ? w[0] >> 16 : w[0] & 0xFFFFu) >> 4);
  if ((lane & 2) == 0 && n < N && m != 0) atomicMax(colexp + n, m);
}

// Output of one row's EPI_COLS columns: out = sign * sum * 2^(ea + eb - 14)
// (mode 0) or C += that (mode 1), C's entries loaded LOAD_BATCH ahead.  FULL: all of the columns are there.
template <bool FULL, typename Sums>
__device__ __forceinline__ void write_cols(const OzkArgs& a, int r, int n0, double* crow,
                                           const Sums& sums, bool live) {
  static_assert(EPI_COLS == 16, "two columns a word, eight words for 32 lanes");
  const unsigned neg = a.sign < 0.0 ? 1u : 0u;
  const int er = live ? a.ea[r] - 14 : 0;
  double* p = crow + (long long)n0 * a.ccs;
  constexpr int LOAD_BATCH = 8;
  double cv[LOAD_BATCH];
  const uint32_t counted = live && r >= a.row_lo ? 0x7FF07FF0u : 0u;
  uint32_t ex[EPI_COLS / 2];
#pragma unroll
  for (int j = 0; j < EPI_COLS; ++j) {
    if (j % LOAD_BATCH == 0) {
#pragma unroll
      for (int i = 0; i < LOAD_BATCH; ++i)
        cv[i] = (a.mode == 1 && live && (FULL || n0 + j + i < a.N)) ? p[(long long)(j + i) * a.ccs]
                                                                    : 0.0;
    }
    const int n = n0 + j;
    double out = 0.0;
    if (FULL || n < a.N) {
      const int ek = er + (a.eb_raw ? scale_of_raw(a.eb_raw[n]) : a.eb[n]);
      const double v = sums.value(j, ek, neg);
      out = a.mode == 0 ? v : cv[j % LOAD_BATCH] + v;
      if (live) p[(long long)j * a.ccs] = out;
    }
    if (j & 1)
      ex[j / 2] = __byte_perm(ex[j / 2], (uint32_t)__double2hiint(out), 0x7632) & counted;
    else
      ex[j / 2] = (uint32_t)__double2hiint(out);
  }
  if (a.colexp != nullptr)  // kernel-uniform; every lane of the warp is here
    raise_exponents(ex, a.colexp, n0, a.N, threadIdx.x & 31);
}

template <typename Sums>
__device__ __forceinline__ void write_row(const OzkArgs& a, int r, int n0, double* crow,
                                          const Sums& sums, bool live) {
  if (n0 + EPI_COLS <= a.N)
    write_cols<true>(a, r, n0, crow, sums, live);
  else
    write_cols<false>(a, r, n0, crow, sums, live);
}

// Digit-pair MMAs of one K block into the accumulators at tb: pair (s, t) into
// acc_of_level(s + t).  The B digits of a stage follow one another in shared
// memory and so do the accumulators in TMEM, so one MMA of N = n x TN columns
// multiplies digit s of A with n consecutive digits of B into n consecutive
// levels: an MMA costs at least 62 clocks, whatever its N up to 128, and 1/2
// clock a column beyond, and reads its A tile from shared memory once.
// FIRST: the accumulators restart -- each group is waited for (its round'th
// hand-back) and overwritten; last: each group is committed once complete.
// False if a wait gave up.
template <int S, bool FIRST>
__device__ __forceinline__ bool issue_pairs(uint32_t tb, uint64_t da0, uint64_t db0, int s_rt,
                                            uint32_t idesc, bool last, Handover h, int round,
                                            unsigned lim, volatile int* abort_flag) {
  // S > 0: fully unrolled (every descriptor offset, TMEM column and accumulate
  // flag a constant, so the single issuing thread spends its time on
  // tcgen05.mma instead of loop and index arithmetic); S = 0: s_rt digits.
  const int ns = S > 0 ? S : s_rt;
  const int nacc = S > 0 ? n_acc(S) : n_acc(s_rt);
#pragma unroll
  for (int g = 0; g < MAX_GROUPS; ++g) {
    const int lo = g * ACC_GROUP;
    const int hi = lo + ACC_GROUP < nacc ? lo + ACC_GROUP : nacc;
    if (lo >= nacc) continue;
    if (FIRST) {
      if (!warp_wait(&h.empty[g], (round & 1) ^ 1, lim, abort_flag)) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
#pragma unroll
    for (int s = 0; s < 7; ++s) {
#pragma unroll
      for (int kk = 0; kk < TK / 16; ++kk) {
        const uint64_t da = da0 + (uint64_t)((s * A_TILE) >> 4) + 2 * kk;
        if (s < hi) {
          const int q0 = s > lo ? s : lo, n = hi - q0;
          mma_bf16(tb + (uint32_t)(q0 * TN), da,
                   db0 + (uint64_t)(((q0 - s) * B_TILE) >> 4) + 2 * kk,
                   idesc + ((uint32_t)(n * TN >> 3) << 17), FIRST && s == 0 && kk == 0 ? 0u : 1u);
        }
        if (ns > nacc && hi == nacc && s < ns)  // level 6 shares the last accumulator
          mma_bf16(tb + (uint32_t)((nacc - 1) * TN), da,
                   db0 + (uint64_t)(((ns - 1 - s) * B_TILE) >> 4) + 2 * kk,
                   idesc + ((uint32_t)(TN >> 3) << 17), 1u);
      }
    }
    if (last) mma_commit(&h.full[g]);
  }
  return true;
}

__device__ __forceinline__ bool issue_block(uint32_t tb, uint64_t da0, uint64_t db0, int S,
                                            uint32_t idesc, bool first, bool last, Handover h,
                                            int round, unsigned lim, volatile int* abort_flag) {
  if (S == 7)
    return first ? issue_pairs<7, true>(tb, da0, db0, S, idesc, last, h, round, lim, abort_flag)
                 : issue_pairs<7, false>(tb, da0, db0, S, idesc, last, h, round, lim, abort_flag);
  return first ? issue_pairs<0, true>(tb, da0, db0, S, idesc, last, h, round, lim, abort_flag)
               : issue_pairs<0, false>(tb, da0, db0, S, idesc, last, h, round, lim, abort_flag);
}

__global__ void __launch_bounds__(NT, 1) ozk_gemm_kernel(OzkArgs a) {
  HQ_PDL_WAIT();
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[MAX_STAGES], empty_bar[MAX_STAGES];
  __shared__ __align__(8) uint64_t acc_full[MAX_GROUPS], acc_empty[MAX_GROUPS], done_bar;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int s_abort;
  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
  const int S = a.S;
  const int a_stage = S * A_TILE, b_stage = S * B_TILE;
  const int nacc = n_acc(S);
  const uint32_t tmem_cols = tmem_pow2((uint32_t)(nacc * TN));
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  uint8_t* sA = smem;
  const int STAGES = a.stages;
  uint8_t* sB = smem + STAGES * a_stage;
  const int mt = blockIdx.x, nt = blockIdx.y, z = blockIdx.z;
  const int kb0 = z * a.kb_per_z;
  const int nkb = min(a.KB - kb0, a.kb_per_z);
  const int ndrain = (nkb + KB_PER_DRAIN - 1) / KB_PER_DRAIN;

  if (tid == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    for (int g = 0; g < MAX_GROUPS; ++g) {
      mbar_init(&acc_full[g], 1);
      mbar_init(&acc_empty[g], NEPI / 32);
    }
    mbar_init(&done_bar, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base)),
                 "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tbase = tmem_base;
  const unsigned lim = a.spin_limit;
  const Handover hand = {acc_full, acc_empty};
  int copies_issued = 0;

  if (warp == PRODUCER_WARP) {
    // Producer: one elected lane streams the digit tiles through the ring.
    if (lane == 0) {
      for (int i = 0; i < nkb; ++i) {
        const int st = i % STAGES;
        if (!mbar_wait(&empty_bar[st], ((i / STAGES) & 1) ^ 1, lim, &s_abort)) {
          s_abort = 1;
          break;
        }
        mbar_expect_tx(&full_bar[st], (unsigned)(a_stage + b_stage));
        bulk_load(sA + st * a_stage, a.A + ((long long)mt * a.KB + kb0 + i) * a_stage, a_stage,
                  &full_bar[st]);
        bulk_load(sB + st * b_stage, a.B + ((long long)nt * a.KB + kb0 + i) * b_stage, b_stage,
                  &full_bar[st]);
        ++copies_issued;
      }
    }
  } else if (warp == MMA_WARP) {
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TM >> 4) << 24);
    for (int i = 0; i < nkb; ++i) {
      const int st = i % STAGES;
      if (!warp_wait(&full_bar[st], (i / STAGES) & 1, lim, &s_abort)) {
        s_abort = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // Every accumulator restarts after a drain, every KB_PER_DRAIN blocks.
      if (!issue_block(tbase, sw64_desc(smem_u32(sA + st * a_stage)),
                       sw64_desc(smem_u32(sB + st * b_stage)), S, idesc, i % KB_PER_DRAIN == 0,
                       (i + 1) % KB_PER_DRAIN == 0 || i + 1 == nkb, hand, i / KB_PER_DRAIN, lim,
                       &s_abort)) {
        s_abort = 1;
        break;
      }
      mma_commit(&empty_bar[st]);
    }
    // Nothing of the tensor core's may arrive in shared memory after exit.
    mma_commit(&done_bar);
    if (!warp_wait(&done_bar, 0, lim, nullptr)) s_abort = 1;
  } else {
    // Epilogue warps 0-19: TMEM lanes 32*(warp&3).. = tile rows, columns
    // (warp>>2)*EPI_COLS.. of the tile.
    FloatSums sums;
    sums.clear();
    const int col0 = (warp >> 2) * EPI_COLS;
    const uint32_t tacc = tbase + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)col0;
    bool ok = true;
    for (int d = 0; d < ndrain && ok; ++d)
      ok = drain_levels(tacc, nacc, hand, d, lim, &s_abort, lane,
                        [&](int q, const float* v) { sums.add(q, v); });
    if (!ok) {
      s_abort = 1;
    } else {
      const int r = mt * TM + (warp & 3) * 32 + lane;
      if (r < a.M)
        write_row(a, r, nt * TN + col0, a.C + (long long)r * a.crs + (long long)z * a.zstride,
                  sums, true);
    }
  }

  // Teardown: on abort, wait (bounded) for in-flight copies first.
  __syncthreads();
  if (s_abort) {
    if (tid == 0) atomicCAS(a.err, 0, HQ_ERR_BARRIER_TIMEOUT);
    if (warp == PRODUCER_WARP && lane == 0) {
      // The last copy issued into each stage is the only one that can still
      // be in flight.
      for (int i = copies_issued > STAGES ? copies_issued - STAGES : 0; i < copies_issued; ++i)
        mbar_wait(&full_bar[i % STAGES], (i / STAGES) & 1, lim, nullptr);
    }
    __syncthreads();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase),
                 "r"(tmem_cols)
                 : "memory");
}

// Long-K product whose N-side operand is read as FP64 (C in the block update
// W1 = U'^T C): the producer brings each K block of C (80 columns x 32 rows,
// 20 KB) with a 2-D tensor-map load next to the M side's digit tiles, and the
// epilogue warps -- idle between drains -- cut it into the seven digit planes
// in shared memory, in the 64-byte-swizzled layout the MMA descriptors read
// (16-byte chunk c of row r of a 64-byte row at chunk c ^ ((r >> 1) & 3)).
// The column scales come from eb_raw (each column's largest exponent field,
// recorded by the epilogue of the update that wrote C), so nothing is read
// twice: the trailing matrix is read once as FP64 instead of being split to
// 14 bytes of digits per entry and read back.  The digits are those
// ozk_split_chunk_kernel writes.  The writes (generic proxy) are
// fenced to the async proxy before the MMAs.
// K <= 256 takes the sums that the short-K kernel takes (the last blocks of a
// factorization), so both routes give the same bits there too.
constexpr int C64_TILE = TN * TK * 8;  // 20 KB of FP64 per stage
// The FP64 tiles have a producer warp of their own: two lanes of one warp that
// wait for different barriers hold each other up.
constexpr int C64_PRODUCER_WARP = 22;
constexpr int NT_C64 = NT + 32;

// One thread's share of a block's conversion: 4 consecutive K entries (h-th
// quarter of the 32) of tile column c, read as two 16-byte loads, written as
// 8 bytes of each digit plane.
template <int S>
__device__ __forceinline__ void convert_quarter(const double* __restrict__ sC, uint8_t* sBst, int c,
                                                int h, int shift_base) {
  const double2* x2 = reinterpret_cast<const double2*>(sC + c * TK + h * 4);
  const double2 p0 = x2[0], p1 = x2[1];
  const unsigned long long w0 = digit_word<S>(p0.x, shift_base);
  const unsigned long long w1 = digit_word<S>(p0.y, shift_base);
  const unsigned long long w2 = digit_word<S>(p1.x, shift_base);
  const unsigned long long w3 = digit_word<S>(p1.y, shift_base);
  const int phys = (h >> 1) ^ ((c >> 1) & 3);  // 64-byte swizzle of the 16-byte chunk
  uint8_t* dst = sBst + c * (TK * 2) + phys * 16 + (h & 1) * 8;
#pragma unroll
  for (int s = 0; s < S; ++s)
    *reinterpret_cast<uint2*>(dst + s * B_TILE) =
        make_uint2(digit_pair<S>(w0, w1, s), digit_pair<S>(w2, w3, s));
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

template <typename Sums>
__global__ void __launch_bounds__(NT_C64, 1) ozk_gemm_c64_kernel(
    OzkArgs a, const __grid_constant__ CUtensorMap tmC) {
  HQ_PDL_WAIT();
  constexpr int S = 7;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // full_bar: the M side's digits of a block landed and those of the N side
  // are cut; c_full: its FP64 N-side tile landed; c_empty: the converters are
  // done with that FP64 tile; empty_bar: the MMAs are done with the A and B
  // stages.  The FP64 tile of block i is fetched as soon as block i - 2's was
  // converted, so its load never waits for the MMAs.
  __shared__ __align__(8) uint64_t full_bar[MAX_STAGES], c_full[MAX_STAGES], c_empty[MAX_STAGES],
      empty_bar[MAX_STAGES];
  __shared__ __align__(8) uint64_t acc_full[MAX_GROUPS], acc_empty[MAX_GROUPS], done_bar;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int s_abort;
  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
  const int a_stage = S * A_TILE, b_stage = S * B_TILE;
  const int nacc = n_acc(S);
  const uint32_t tmem_cols = tmem_pow2((uint32_t)(nacc * TN));
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  const int STAGES = a.stages;
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * a_stage;
  uint8_t* sC = sB + STAGES * b_stage;  // FP64 staging, C64_TILE per stage
  const int mt = blockIdx.x, nt = blockIdx.y, z = blockIdx.z;
  const int kb0 = z * a.kb_per_z;
  const int nkb = min(a.KB - kb0, a.kb_per_z);

  if (tid == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full_bar[i], 1 + NEPI / 32);
      mbar_init(&c_full[i], 1);
      mbar_init(&c_empty[i], NEPI / 32);
      mbar_init(&empty_bar[i], 1);
    }
    for (int g = 0; g < MAX_GROUPS; ++g) {
      mbar_init(&acc_full[g], 1);
      mbar_init(&acc_empty[g], NEPI / 32);
    }
    mbar_init(&done_bar, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base)),
                 "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tbase = tmem_base;
  const unsigned lim = a.spin_limit;
  const Handover hand = {acc_full, acc_empty};
  int a_issued = 0, c_issued = 0;  // the two producers

  if (warp == PRODUCER_WARP) {
    if (lane == 0) {  // the M side's digit tiles, as the MMAs free the stages
      for (int i = 0; i < nkb; ++i) {
        const int st = i % STAGES;
        if (!mbar_wait(&empty_bar[st], ((i / STAGES) & 1) ^ 1, lim, &s_abort)) {
          s_abort = 1;
          break;
        }
        mbar_expect_tx(&full_bar[st], (unsigned)a_stage);
        bulk_load(sA + st * a_stage, a.A + ((long long)mt * a.KB + kb0 + i) * a_stage, a_stage,
                  &full_bar[st]);
        ++a_issued;
      }
    }
  } else if (warp == C64_PRODUCER_WARP) {
    if (lane == 0) {  // the FP64 tiles, as the converters free them
      for (int i = 0; i < nkb; ++i) {
        const int st = i % STAGES;
        if (!mbar_wait(&c_empty[st], ((i / STAGES) & 1) ^ 1, lim, &s_abort)) {
          s_abort = 1;
          break;
        }
        mbar_expect_tx(&c_full[st], (unsigned)C64_TILE);
        tma_load_2d(sC + st * C64_TILE, &tmC, (kb0 + i) * TK, nt * TN, &c_full[st]);
        ++c_issued;
      }
    }
  } else if (warp == MMA_WARP) {
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TM >> 4) << 24);
    for (int i = 0; i < nkb; ++i) {
      const int st = i % STAGES;
      if (!warp_wait(&full_bar[st], (i / STAGES) & 1, lim, &s_abort)) {
        s_abort = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (!issue_block(tbase, sw64_desc(smem_u32(sA + st * a_stage)),
                       sw64_desc(smem_u32(sB + st * b_stage)), S, idesc, i % KB_PER_DRAIN == 0,
                       (i + 1) % KB_PER_DRAIN == 0 || i + 1 == nkb, hand, i / KB_PER_DRAIN, lim,
                       &s_abort)) {
        s_abort = 1;
        break;
      }
      mma_commit(&empty_bar[st]);
    }
    // Nothing of the tensor core's may arrive in shared memory after exit.
    mma_commit(&done_bar);
    if (!warp_wait(&done_bar, 0, lim, nullptr)) s_abort = 1;
  } else {
    // Epilogue warps 0-19: convert every K block, drain every 256 K, write.
    Sums sums;
    sums.clear();
    const int col0 = (warp >> 2) * EPI_COLS;
    const uint32_t tacc = tbase + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)col0;
    // Conversion task of this thread: column cc of the tile, quarter cq
    // (4 K entries) of the block's 32 -- 80 x 8 tasks, one per epilogue thread.
    static_assert(TN * (TK / 4) == NEPI, "one conversion task per epilogue thread");
    const int cc = tid >> 3, cq = tid & 7;
    int shift_base = 0;
    {
      const int n = nt * TN + cc;
      shift_base = 8 * S - 1076 - (n < a.N ? scale_of_raw(a.eb_raw[n]) : 0);
    }
    bool ok = true;
    auto drain = [&](int d) {
      return drain_levels(tacc, nacc, hand, d, lim, &s_abort, lane,
                          [&](int q, const float* v) { sums.add(q, v); });
    };
    for (int i = 0; i < nkb && ok; ++i) {
      const int st = i % STAGES;
      // The FP64 tile is here, and the MMAs of block i - STAGES are done with
      // the B stage the digits go to.
      ok = __all_sync(0xffffffffu,
                      mbar_wait(&c_full[st], (i / STAGES) & 1, lim, &s_abort) &&
                          mbar_wait(&empty_bar[st], ((i / STAGES) & 1) ^ 1, lim, &s_abort));
      if (!ok) break;
      convert_quarter<S>(reinterpret_cast<const double*>(sC + st * C64_TILE), sB + st * b_stage,
                         cc, cq, shift_base);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&full_bar[st]);
        mbar_arrive(&c_empty[st]);
      }
      // The drain of the K blocks before this one, after this one's digits are
      // out: the MMAs that follow the drain find their operands ready.
      if (i % KB_PER_DRAIN == 0 && i > 0) ok = drain(i / KB_PER_DRAIN - 1);
    }
    if (ok && nkb > 0) ok = drain((nkb - 1) / KB_PER_DRAIN);
    if (!ok) {
      s_abort = 1;
    } else {
      const int r = mt * TM + (warp & 3) * 32 + lane;
      if (r < a.M)
        write_row(a, r, nt * TN + col0, a.C + (long long)r * a.crs + (long long)z * a.zstride,
                  sums, true);
    }
  }

  // Teardown: on abort, wait (bounded) for in-flight copies first.
  __syncthreads();
  if (s_abort) {
    if (tid == 0) atomicCAS(a.err, 0, HQ_ERR_BARRIER_TIMEOUT);
    if (warp == PRODUCER_WARP && lane == 0) {
      for (int i = a_issued > STAGES ? a_issued - STAGES : 0; i < a_issued; ++i)
        mbar_wait(&full_bar[i % STAGES], (i / STAGES) & 1, lim, nullptr);
    }
    if (warp == C64_PRODUCER_WARP && lane == 0) {
      for (int i = c_issued > STAGES ? c_issued - STAGES : 0; i < c_issued; ++i)
        mbar_wait(&c_full[i % STAGES], (i / STAGES) & 1, lim, nullptr);
    }
    __syncthreads();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase),
                 "r"(tmem_cols)
                 : "memory");
}

// Persistent variant for short products (K <= 256, so no intermediate drain
// of the exact levels): one CTA per SM walks the output tiles (TM x TN), down
// the columns (what the CTAs update at one time is then contiguous), and
// the producer streams operand stages ahead across tile boundaries.  The
// epilogue warps first drain a tile's accumulators into registers and hand
// the TMEM back, then do the FP64 output (the part bound by the FP64 pipe and
// by C's memory traffic) while the MMAs of the next tile run.  Mode 1
// (C += sign * A B^T) or 0 (C = sign * A B^T), no grid.z split.
__global__ void __launch_bounds__(NT, 1) ozk_gemm_short_kernel(OzkArgs a) {
  HQ_PDL_WAIT();
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[MAX_STAGES], empty_bar[MAX_STAGES];
  __shared__ __align__(8) uint64_t acc_full[MAX_GROUPS], acc_empty[MAX_GROUPS], done_bar;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int s_abort;
  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
  const int S = a.S;
  const int a_stage = S * A_TILE, b_stage = S * B_TILE;
  const int nacc = n_acc(S);
  const uint32_t tmem_cols = tmem_pow2((uint32_t)(nacc * TN));
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  const int STAGES = a.stages;
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * a_stage;
  const int MT = (a.M + TM - 1) / TM, NTL = (a.N + TN - 1) / TN;
  const int ntiles = MT * NTL, nkb = a.KB;

  if (tid == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    for (int g = 0; g < MAX_GROUPS; ++g) {
      mbar_init(&acc_full[g], 1);
      mbar_init(&acc_empty[g], NEPI / 32);
    }
    mbar_init(&done_bar, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base)),
                 "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tbase = tmem_base;
  const unsigned lim = a.spin_limit;
  const Handover hand = {acc_full, acc_empty};
  int copies_issued = 0;

  if (warp == PRODUCER_WARP) {
    if (lane == 0) {
      int i = 0;  // stage counter across tiles
      for (int t = blockIdx.x; t < ntiles && !s_abort; t += gridDim.x) {
        const int mt = t % MT, nt = t / MT;
        for (int kb = 0; kb < nkb; ++kb, ++i) {
          const int st = i % STAGES;
          if (!mbar_wait(&empty_bar[st], ((i / STAGES) & 1) ^ 1, lim, &s_abort)) {
            s_abort = 1;
            break;
          }
          mbar_expect_tx(&full_bar[st], (unsigned)(a_stage + b_stage));
          bulk_load(sA + st * a_stage, a.A + ((long long)mt * nkb + kb) * a_stage, a_stage,
                    &full_bar[st]);
          bulk_load(sB + st * b_stage, a.B + ((long long)nt * nkb + kb) * b_stage, b_stage,
                    &full_bar[st]);
          ++copies_issued;
        }
      }
    }
  } else if (warp == MMA_WARP) {
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TM >> 4) << 24);
    int i = 0, lt = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++lt) {
      bool ok = true;
      for (int kb = 0; kb < nkb && ok; ++kb, ++i) {
        const int st = i % STAGES;
        ok = warp_wait(&full_bar[st], (i / STAGES) & 1, lim, &s_abort);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        ok = issue_block(tbase, sw64_desc(smem_u32(sA + st * a_stage)),
                         sw64_desc(smem_u32(sB + st * b_stage)), S, idesc, kb == 0,
                         kb + 1 == nkb, hand, lt, lim, &s_abort);
        if (ok) mma_commit(&empty_bar[st]);
      }
      if (!ok) {
        s_abort = 1;
        break;
      }
    }
    // Nothing of the tensor core's may arrive in shared memory after exit.
    mma_commit(&done_bar);
    if (!warp_wait(&done_bar, 0, lim, nullptr)) s_abort = 1;
  } else {
    const int col0 = (warp >> 2) * EPI_COLS;
    const uint32_t tacc = tbase + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)col0;
    int lt = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++lt) {
      ExactSums sums;
      sums.clear();
      // One outcome per warp: the TMEM loads and the exponent reduction are
      // warp-wide, so no lane may leave the loop alone.
      if (!drain_levels(tacc, nacc, hand, lt, lim, &s_abort, lane,
                        [&](int q, const float* v) { sums.add(q, v); })) {
        s_abort = 1;
        break;
      }
      const int mt = t % MT, nt = t / MT;
      const int r = mt * TM + (warp & 3) * 32 + lane;
      // Every lane takes part (the column-exponent reduction is warp-wide);
      // rows past M only skip their loads and stores.
      write_row(a, r, nt * TN + col0, a.C + (long long)(r < a.M ? r : 0) * a.crs, sums, r < a.M);
    }
  }

  // Teardown: on abort, wait (bounded) for in-flight copies first.
  __syncthreads();
  if (s_abort) {
    if (tid == 0) atomicCAS(a.err, 0, HQ_ERR_BARRIER_TIMEOUT);
    if (warp == PRODUCER_WARP && lane == 0) {
      for (int i = copies_issued > STAGES ? copies_issued - STAGES : 0; i < copies_issued; ++i)
        mbar_wait(&full_bar[i % STAGES], (i / STAGES) & 1, lim, nullptr);
    }
    __syncthreads();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase),
                 "r"(tmem_cols)
                 : "memory");
}

__global__ void ozk_sum_slices(int M, int N, int Z, const double* __restrict__ ws,
                               double* __restrict__ C, long long crs, long long ccs, int accumulate) {
  HQ_PDL_WAIT();
  const long long total = (long long)M * N;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(e % M), c = (int)(e / M);
    double s = 0.0;
    for (int zz = 0; zz < Z; ++zz) s += ws[e + (long long)zz * total];
    double* p = C + (long long)r * crs + (long long)c * ccs;
    *p = accumulate ? *p + s : s;
  }
}

}  // namespace

// side 0: M-side tiles (TM rows); 1: N-side tiles (TN rows) for the general
// kernel; 2: N-side tiles of TN_SHORT rows for the short-K kernel.
extern "C" size_t hq_ozk_tile_bytes(int rows, int K, int S, int side) {
  const int TR = side == 0 ? TM : (side == 2 ? TN_SHORT : TN);
  const long long RT = (rows + TR - 1) / TR, KB = (K + TK - 1) / TK;
  return (size_t)(RT * KB * S) * (size_t)(TR * TK * 2);
}

extern "C" int hq_ozk_rowmax_raw(cudaStream_t stream, const double* X, long long rs,
                                 long long ks, int R, int K, int rows_total, int* raw) {
  if (R <= 0 || K <= 0) return 0;
  const int e = hq_zero_words(stream, raw, (size_t)rows_total, nullptr, 0);
  if (e) return e;
  if (rs == 1 && ks != 1)
    hq_launch(ozk_rowmax_cm_kernel,
              dim3((R + 31) / 32, (K + ROWMAX_CM_SPAN - 1) / ROWMAX_CM_SPAN), 256, 0, stream, X, ks,
              R, K, raw);
  else
    hq_launch(ozk_rowmax_atomic_kernel, dim3(R, (K + ROWMAX_SPAN - 1) / ROWMAX_SPAN), 256, 0,
              stream, X, rs, ks, K, raw);
  hq_count_launches(1);
  return (int)cudaGetLastError();
}

extern "C" int hq_ozk_split_rows(int R, int side) {
  const int TR = side == 0 ? TM : (side == 2 ? TN_SHORT : TN);
  return (R + TR - 1) / TR * TR;
}

extern "C" int hq_ozk_split(cudaStream_t stream, const double* X, long long rs, long long ks,
                            int R, int K, int S, int side, void* tiles, int* exps, int* raw) {
  if (R <= 0 || K <= 0) return 0;
  if (S < 1 || S > 7) return (int)cudaErrorInvalidValue;
  const int TR = side == 0 ? TM : (side == 2 ? TN_SHORT : TN);
  const int RT = (R + TR - 1) / TR, KB = (K + TK - 1) / TK;
  const int rows_total = RT * TR;
  int blocks = (rows_total + 7) / 8;
  if (blocks > 4096) blocks = 4096;
  uint8_t* t = static_cast<uint8_t*>(tiles);
  // Rows of 512 or more take two passes, spread over CTAs (4000 x 4000: the
  // exponents in 34 us, then the digits in 54; one CTA a row that held the row in
  // registers took 133, its one pass bound by latency).
  if (S == 7 && K >= 512) {
    if (raw == nullptr) return (int)cudaErrorInvalidValue;
    const int e = hq_ozk_rowmax_raw(stream, X, rs, ks, R, K, rows_total, raw);
    return e ? e : hq_ozk_split_raw(stream, X, rs, ks, R, K, S, side, tiles, exps, raw);
  }
  if (rs == 1 && ks != 1 && K <= CM_KMAX) {  // column-major rows of a short operand
    const int cb = (rows_total + 31) / 32;
    switch (S) {
#define HQ_SPLIT_CM_CASE(SS)                                                            \
  case SS:                                                                              \
    hq_launch(ozk_split_cm_kernel<SS>, cb, 256, 0, stream, X, ks, R, K, TR, KB, rows_total, t, exps); \
    break;
      HQ_SPLIT_CM_CASE(1) HQ_SPLIT_CM_CASE(2) HQ_SPLIT_CM_CASE(3) HQ_SPLIT_CM_CASE(4)
      HQ_SPLIT_CM_CASE(5) HQ_SPLIT_CM_CASE(6) HQ_SPLIT_CM_CASE(7)
#undef HQ_SPLIT_CM_CASE
    }
    hq_count_launches(1);
    return (int)cudaGetLastError();
  }
  switch (S) {
#define HQ_SPLIT_CASE(SS)                                                                  \
  case SS:                                                                                 \
    hq_launch(ozk_split_kernel<SS>, blocks, 256, 0, stream, X, rs, ks, R, K, TR, KB, rows_total, t, \
                                                     exps);                                \
    break;
    HQ_SPLIT_CASE(1) HQ_SPLIT_CASE(2) HQ_SPLIT_CASE(3) HQ_SPLIT_CASE(4) HQ_SPLIT_CASE(5)
    HQ_SPLIT_CASE(6) HQ_SPLIT_CASE(7)
#undef HQ_SPLIT_CASE
  }
  hq_count_launches(1);
  return (int)cudaGetLastError();
}

// The split with each row's largest exponent field already known (raw[r],
// e.g. produced by the epilogue of the update that wrote X): one streaming
// pass, no row maximum.  exps receives the scale exponents as hq_ozk_split
// writes them.
extern "C" int hq_ozk_split_raw(cudaStream_t stream, const double* X, long long rs, long long ks,
                                int R, int K, int S, int side, void* tiles, int* exps,
                                const int* raw) {
  if (R <= 0 || K <= 0) return 0;
  if (S != 7) return (int)cudaErrorInvalidValue;
  const int TR = side == 0 ? TM : (side == 2 ? TN_SHORT : TN);
  const int RT = (R + TR - 1) / TR, KB = (K + TK - 1) / TK;
  const int rows_total = RT * TR;
  const long long chunks = (long long)rows_total * KB * (TK / 8);
  long long cblocks = (chunks + 255) / 256;
  if (cblocks > 65536) cblocks = 65536;
  hq_launch(ozk_split_chunk_kernel<7>, (unsigned)cblocks, 256, 0, stream,
      X, rs, ks, R, K, TR, KB, rows_total, static_cast<uint8_t*>(tiles), exps, raw);
  hq_count_launches(1);
  return (int)cudaGetLastError();
}

// Split K of the long products (one CTA per SM): the time is about (waves)
// x (K blocks per CTA + a fixed cost of ~2 per tile) plus the slices' sum.
// Taking the split that minimizes it, instead of the first one past two
// waves, keeps the last wave from running mostly empty (modelled 16 % less
// W1 time over a 16384^2 factorization's blocks).  Both long kernels use it,
// so they sum the same slices in the same order.
static int choose_split(long long tiles, int KB, int M, int N, size_t ws_elems, int num_sms) {
  const int max_z = (KB + KB_PER_DRAIN - 1) / KB_PER_DRAIN;
  int Z = 1;
  double best = 1e300;
  for (int z = 1; z <= max_z; ++z) {
    if (z > 1 && (size_t)(z + 1) * M * N > ws_elems) break;
    int kz = (KB + z - 1) / z;
    kz = (kz + KB_PER_DRAIN - 1) / KB_PER_DRAIN * KB_PER_DRAIN;
    const int zz = (KB + kz - 1) / kz;
    const long long waves = (tiles * zz + num_sms - 1) / num_sms;
    const double sum = zz > 1 ? (double)zz * M * N / (6000.0 * num_sms) : 0.0;
    const double cost = (double)waves * (kz + 2.0) + sum;
    if (cost < best) {
      best = cost;
      Z = zz;
    }
  }
  return Z;
}

extern "C" int hq_ozk_gemm(cudaStream_t stream, const hq_device_info* dev, int M, int N, int K,
                           int S, const void* Atiles, const int* ea, const void* Btiles,
                           const int* eb, int mode, double sign, double* C, long long crs,
                           long long ccs, double* ws, size_t ws_elems, int* err,
                           unsigned spin_limit) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (S < 1 || S > 7) return (int)cudaErrorInvalidValue;
  const int MT = (M + TM - 1) / TM, NTL = (N + TN - 1) / TN, KB = (K + TK - 1) / TK;
  // Split K across grid.z (mode 0 only).
  int Z = 1;
  if (mode == 0 && ws != nullptr)
    Z = choose_split((long long)MT * NTL, KB, M, N, ws_elems, dev->num_sms);
  int kb_per_z = (KB + Z - 1) / Z;
  kb_per_z = (kb_per_z + KB_PER_DRAIN - 1) / KB_PER_DRAIN * KB_PER_DRAIN;
  Z = (KB + kb_per_z - 1) / kb_per_z;
  OzkArgs a;
  a.A = static_cast<const uint8_t*>(Atiles);
  a.B = static_cast<const uint8_t*>(Btiles);
  a.ea = ea;
  a.eb = eb;
  a.M = M;
  a.N = N;
  a.S = S;
  a.KB = KB;
  a.kb_per_z = kb_per_z;
  a.mode = mode;
  a.sign = sign;
  a.err = err;
  a.spin_limit = spin_limit;
  a.colexp = nullptr;
  a.row_lo = 0;
  a.eb_raw = nullptr;
  if (Z > 1) {
    a.C = ws;
    a.crs = 1;
    a.ccs = M;
    a.zstride = (long long)M * N;
  } else {
    a.C = C;
    a.crs = crs;
    a.ccs = ccs;
    a.zstride = 0;
  }
  int stages = MAX_STAGES;
  size_t smem = (size_t)stages * S * (A_TILE + B_TILE) + 1024;
  if (smem > dev->smem_optin) {
    stages = 2;
    smem = (size_t)stages * S * (A_TILE + B_TILE) + 1024;
  }
  if (smem > dev->smem_optin) return (int)cudaErrorInvalidValue;
  a.stages = stages;
  cudaError_t e =
      cudaFuncSetAttribute(ozk_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  hq_launch(ozk_gemm_kernel, dim3(MT, NTL, Z), NT, smem, stream, a);
  hq_count_launches(1);
  if (Z > 1) {
    long long total = (long long)M * N;
    int blocks = (int)((total + 255) / 256);
    if (blocks > dev->num_sms * 8) blocks = dev->num_sms * 8;
    hq_launch(ozk_sum_slices, blocks, 256, 0, stream, M, N, Z, ws, C, crs, ccs, 0);
    hq_count_launches(1);
  }
  return (int)cudaGetLastError();
}

// W1-style product with an FP64 N-side operand: Y element (n, k) at
// Y[n * yld + k] (k contiguous), n < N, k < K; raw[n] = row n's largest
// exponent field.  Mode 0 only (C = sign * A Y^T, split K through ws as in
// hq_ozk_gemm).  Returns cudaErrorNotSupported when Y's layout does not meet
// the tensor-map rules (16-byte aligned base and stride), so the caller can
// split Y instead.
extern "C" int hq_ozk_gemm_c64(cudaStream_t stream, const hq_device_info* dev, int M, int N,
                               int K, const void* Atiles, const int* ea, const double* Y,
                               long long yld, const int* raw, double sign, double* C,
                               long long crs, long long ccs, double* ws, size_t ws_elems,
                               int* err, unsigned spin_limit) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  constexpr int S = 7;
  if ((reinterpret_cast<uintptr_t>(Y) & 15) != 0 || ((yld * 8) & 15) != 0 || yld < K)
    return (int)cudaErrorNotSupported;
  const size_t smem = (size_t)2 * (S * (A_TILE + B_TILE) + C64_TILE) + 1024;
  if (smem > dev->smem_optin) return (int)cudaErrorNotSupported;
  const int MT = (M + TM - 1) / TM, NTL = (N + TN - 1) / TN, KB = (K + TK - 1) / TK;
  int Z = 1;
  if (ws != nullptr) Z = choose_split((long long)MT * NTL, KB, M, N, ws_elems, dev->num_sms);
  int kb_per_z = (KB + Z - 1) / Z;
  kb_per_z = (kb_per_z + KB_PER_DRAIN - 1) / KB_PER_DRAIN * KB_PER_DRAIN;
  Z = (KB + kb_per_z - 1) / kb_per_z;
  OzkArgs a;
  a.A = static_cast<const uint8_t*>(Atiles);
  a.B = nullptr;
  a.ea = ea;
  a.eb = nullptr;
  a.eb_raw = raw;
  a.M = M;
  a.N = N;
  a.S = S;
  a.KB = KB;
  a.kb_per_z = kb_per_z;
  a.mode = 0;
  a.sign = sign;
  a.err = err;
  a.spin_limit = spin_limit;
  a.colexp = nullptr;
  a.row_lo = 0;
  a.stages = 2;
  if (Z > 1) {
    a.C = ws;
    a.crs = 1;
    a.ccs = M;
    a.zstride = (long long)M * N;
  } else {
    a.C = C;
    a.crs = crs;
    a.ccs = ccs;
    a.zstride = 0;
  }
  CUtensorMap tmC;
  {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if (encode == nullptr) {
      void* fn = nullptr;
      cudaDriverEntryPointQueryResult q;
      cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000,
                                                       cudaEnableDefault, &q);
      if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || fn == nullptr)
        return (int)cudaErrorNotSupported;
      encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N};
    const cuuint64_t strides[1] = {(cuuint64_t)yld * 8};
    const cuuint32_t box[2] = {(cuuint32_t)TK, (cuuint32_t)TN};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = encode(&tmC, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<double*>(Y), dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return (int)cudaErrorNotSupported;
  }
  const auto kernel =
      KB <= KB_PER_DRAIN ? ozk_gemm_c64_kernel<ExactSums> : ozk_gemm_c64_kernel<FloatSums>;
  cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  hq_launch(kernel, dim3(MT, NTL, Z), NT_C64, smem, stream, a, tmC);
  hq_count_launches(1);
  if (Z > 1) {
    long long total = (long long)M * N;
    int blocks = (int)((total + 255) / 256);
    if (blocks > dev->num_sms * 8) blocks = dev->num_sms * 8;
    hq_launch(ozk_sum_slices, blocks, 256, 0, stream, M, N, Z, ws, C, crs, ccs, 0);
    hq_count_launches(1);
  }
  return (int)cudaGetLastError();
}

// Short products (K <= 256): the persistent kernel; B must be split with side
// 2 (TN_SHORT-row tiles).
extern "C" int hq_ozk_short_ok(int K) { return K > 0 && K <= KB_PER_DRAIN * TK; }

extern "C" int hq_ozk_gemm_short(cudaStream_t stream, const hq_device_info* dev, int M, int N,
                                 int K, int S, const void* Atiles, const int* ea,
                                 const void* Btiles, const int* eb, int mode, double sign,
                                 double* C, long long crs, long long ccs, int* colexp, int row_lo,
                                 int* err, unsigned spin_limit) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (S < 1 || S > 7 || !hq_ozk_short_ok(K)) return (int)cudaErrorInvalidValue;
  constexpr int TNV = TN_SHORT;
  OzkArgs a;
  a.A = static_cast<const uint8_t*>(Atiles);
  a.B = static_cast<const uint8_t*>(Btiles);
  a.ea = ea;
  a.eb = eb;
  a.M = M;
  a.N = N;
  a.S = S;
  a.KB = (K + TK - 1) / TK;
  a.kb_per_z = a.KB;
  a.mode = mode;
  a.sign = sign;
  a.err = err;
  a.spin_limit = spin_limit;
  a.C = C;
  a.crs = crs;
  a.ccs = ccs;
  a.zstride = 0;
  a.colexp = mode == 1 ? colexp : nullptr;
  a.row_lo = row_lo;
  a.eb_raw = nullptr;
  const size_t per_stage = (size_t)S * (A_TILE + B_TILE);
  int stages = MAX_STAGES;
  while (stages > 2 && (size_t)stages * per_stage + 1024 > dev->smem_optin) --stages;
  const size_t smem = (size_t)stages * per_stage + 1024;
  if (smem > dev->smem_optin) return (int)cudaErrorInvalidValue;
  a.stages = stages;
  cudaError_t e = cudaFuncSetAttribute(ozk_gemm_short_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const long long tiles = (long long)((M + TM - 1) / TM) * ((N + TNV - 1) / TNV);
  const int grid = (int)(tiles < dev->num_sms ? tiles : dev->num_sms);
  hq_launch(ozk_gemm_short_kernel, grid, NT, smem, stream, a);
  hq_count_launches(1);
  return (int)cudaGetLastError();
}
