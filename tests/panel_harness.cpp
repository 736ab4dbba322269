// The panel kernel's own source on the CPU, one CTA: the threads are coroutines,
// and a schedule runs the warps one after the other, each as far as it gets
// before it waits for the others.  A word that one warp writes and another
// reads without a barrier between them then holds another value under another
// order of the warps.  panel_kernel.inc is cut out of qrp_panel.cu by the test
// (up to the launch code, the dynamic shared memory's declaration replaced).
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>
#include <ucontext.h>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
using std::isnan;
using std::max;
using std::min;

#undef __global__
#undef __device__
#undef __host__
#undef __shared__
#undef __launch_bounds__
#undef __forceinline__
#undef __align__
#define __global__
#define __device__
#define __host__
#define __shared__ static
#define __launch_bounds__(...)
#define __forceinline__ inline
#define __align__(n) __attribute__((aligned(n)))

struct Idx { int x, y, z; };
static Idx threadIdx, blockIdx{0, 0, 0}, gridDim{1, 1, 1}, blockDim;

namespace emu {

enum Wait { RUN, WARP, BLOCK, POLL, DONE };
struct Fiber {
  ucontext_t ctx;
  std::vector<char> stack;
  Wait wait = RUN;
  unsigned gen = 0, polls = 0;
};
std::vector<Fiber> fibers;
ucontext_t home;
int cur = 0, nthreads = 0;
unsigned warp_gen[32], block_gen;
int warp_in[32], block_in;
unsigned long long slot[32][2][32];
int block_or, block_or_out;
int barriers;  // grid barriers

void yield(Wait w, unsigned gen) {
  Fiber& f = fibers[cur];
  f.wait = w;
  f.gen = gen;
  swapcontext(&f.ctx, &home);
}
bool ready(const Fiber& f, int t) {
  switch (f.wait) {
    case RUN: return true;
    case WARP: return warp_gen[t >> 5] != f.gen;
    case BLOCK: return block_gen != f.gen;
    default: return false;
  }
}
// All lanes hand in v; the 32 values.
const unsigned long long* warp_all(unsigned long long v) {
  const int w = cur >> 5, l = cur & 31;
  const unsigned g = warp_gen[w];
  slot[w][g & 1][l] = v;
  if (++warp_in[w] == 32) {
    warp_in[w] = 0;
    ++warp_gen[w];
  } else {
    yield(WARP, g);
  }
  return slot[w][g & 1];
}
int block_sync(int v) {
  const unsigned g = block_gen;
  block_or |= v;
  if (++block_in == nthreads) {
    block_in = 0;
    block_or_out = block_or;
    block_or = 0;
    ++block_gen;
  } else {
    yield(BLOCK, g);
  }
  return block_or_out;
}

void (*body)();
void entry() {
  body();
  fibers[cur].wait = DONE;
  swapcontext(&fibers[cur].ctx, &home);
}
// Runs nt threads; order 0: the lowest warp first, 1: the highest.  False when
// they no longer get on.
bool run(int nt, int order, void (*fn)()) {
  nthreads = nt;
  body = fn;
  blockDim.x = nt;
  memset(warp_gen, 0, sizeof warp_gen);
  memset(warp_in, 0, sizeof warp_in);
  block_gen = 0;
  block_in = block_or = barriers = 0;
  fibers.assign(nt, Fiber());
  for (int t = 0; t < nt; ++t) {
    Fiber& f = fibers[t];
    f.stack.resize(1 << 16);
    getcontext(&f.ctx);
    f.ctx.uc_stack.ss_sp = f.stack.data();
    f.ctx.uc_stack.ss_size = f.stack.size();
    f.ctx.uc_link = nullptr;
    makecontext(&f.ctx, entry, 0);
  }
  for (int idle = 0; idle < 64;) {
    bool any = false, all_done = true;
    for (int i = 0; i < nt / 32; ++i) {
      const int w = order ? nt / 32 - 1 - i : i;
      for (bool progress = true; progress;) {
        progress = false;
        for (int t = 32 * w; t < 32 * w + 32; ++t)
          if (ready(fibers[t], t)) {
            cur = t;
            threadIdx = {t, 0, 0};
            fibers[t].wait = RUN;
            swapcontext(&home, &fibers[t].ctx);
            progress = any = true;
          }
      }
    }
    for (Fiber& f : fibers) {
      all_done = all_done && f.wait == DONE;
      if (f.wait == POLL) f.wait = RUN;
    }
    if (all_done) return true;
    idle = any ? 0 : idle + 1;
  }
  return false;
}

}  // namespace emu

static inline long long __double_as_longlong(double x) { long long b; memcpy(&b, &x, 8); return b; }
static inline double __longlong_as_double(long long b) { double x; memcpy(&x, &b, 8); return x; }
static inline unsigned __float_as_uint(float x) { unsigned b; memcpy(&b, &x, 4); return b; }
static inline float __uint_as_float(unsigned b) { float x; memcpy(&x, &b, 4); return x; }
static inline float emu_rsqrtf(float x) { return 1.0f / sqrtf(x); }
static inline float __frcp_rn(float x) { return 1.0f / x; }
#define rsqrtf emu_rsqrtf
template <typename T> static inline T __ldcg(const T* p) { return *p; }
template <typename T> static inline T __ldg(const T* p) { return *p; }
static inline int atomicCAS(int* p, int c, int v) { const int o = *p; if (o == c) *p = v; return o; }
static inline void __nanosleep(unsigned) {}
static inline void __syncthreads() { emu::block_sync(0); }
static inline int __syncthreads_or(int v) { return emu::block_sync(v != 0); }
template <typename T> static inline T __shfl_xor_sync(unsigned, T v, int o) {
  unsigned long long b = 0;
  memcpy(&b, &v, sizeof v);
  const int l = emu::cur & 31;
  const unsigned long long r = emu::warp_all(b)[l ^ o];
  memcpy(&v, &r, sizeof v);
  return v;
}
template <typename T> static inline T __shfl_sync(unsigned, T v, int from) {
  unsigned long long b = 0;
  memcpy(&b, &v, sizeof v);
  const unsigned long long r = emu::warp_all(b)[from & 31];
  memcpy(&v, &r, sizeof v);
  return v;
}
static inline unsigned __reduce_max_sync(unsigned, unsigned v) {
  const unsigned long long* a = emu::warp_all(v);
  unsigned r = 0;
  for (int i = 0; i < 32; ++i) r = max(r, (unsigned)a[i]);
  return r;
}
static inline int __reduce_min_sync(unsigned, int v) {
  const unsigned long long* a = emu::warp_all((unsigned)v);
  int r = 0x7fffffff;
  for (int i = 0; i < 32; ++i) r = min(r, (int)(unsigned)a[i]);
  return r;
}

// What hq_common.cuh writes in PTX has its meaning here.
#define hq_st_word ptx_st_word
#define hq_ld_word ptx_ld_word
#define hq_red_word ptx_red_word
#define hq_grid_barrier ptx_grid_barrier
#include "hq_common.cuh"
#undef hq_st_word
#undef hq_ld_word
#undef hq_red_word
#undef hq_grid_barrier
#undef HQ_PDL_WAIT
#define HQ_PDL_WAIT()
static void hq_st_word(void* p, unsigned long long lo, unsigned long long hi) {
  ((unsigned long long*)p)[0] = lo;
  ((unsigned long long*)p)[1] = hi;
}
// A polling thread goes on for a while before the others have their turn.
static void emu_poll() {
  if ((++emu::fibers[emu::cur].polls & 63) == 0) emu::yield(emu::POLL, 0);
}
static void hq_ld_word(const void* p, unsigned long long& lo, unsigned long long& hi) {
  emu_poll();
  lo = ((const unsigned long long*)p)[0];
  hi = ((const unsigned long long*)p)[1];
}
static void hq_ld_word(const void* p, unsigned long long& v) {
  emu_poll();
  v = *(const unsigned long long*)p;
}
static void hq_red_word(void* p, unsigned long long v) { *(unsigned long long*)p += v; }
static bool hq_grid_barrier(unsigned*, int*, unsigned, unsigned, int*) {
  if (emu::cur == 0) ++emu::barriers;
  __syncthreads();
  return true;
}
static double* emu_smem;
#include "panel_kernel.inc"

namespace {
PnArgs g_args;
void small_panel() { panel_qrp_kernel<256, 1, 4>(g_args); }
void wide_panel() { panel_qrp_kernel<512, 1, 2>(g_args); }
}  // namespace

// The pivoted panel of A (m x n, lda = m) by one CTA, the warps in the given
// order.  Returns 0, the kernel's error word, or -1 when no thread gets on.
extern "C" int hq_test_panel(int m, int n, int pivoting, int smem_mode, int order, double* A,
                             double* tau, int* perm, int* barriers) {
  const int R = HQ_PANEL_R(n), ps = (n + 2) & ~1;
  std::vector<double> part(HQ_PANEL_PART_ELEMS(1, n) + 2);
  std::vector<double> smem((size_t)4 * n + n + 2 + (smem_mode ? (size_t)(m | 1) * n : 0));
  unsigned bar = 0;
  int err = 0;
  PnArgs a = {};
  a.mp = m;
  a.nc = n;
  a.ns = m < n ? m : n;
  a.pivoting = pivoting;
  a.P = A;
  a.ldp = m;
  a.tau = tau;
  a.perm = perm;
  a.part = part.data();
  a.pstride = ps;
  a.acc = (unsigned long long*)(part.data() + 2 * ps);
  a.rows = a.acc + (size_t)2 * R * ps * FX_CS;
  a.bar = &bar;
  a.err = &err;
  a.spin_limit = 1000;
  a.smem_mode = smem_mode;
  a.rloc_max = m;
  a.ldxs = m | 1;
  g_args = a;
  emu_smem = smem.data();
  const bool ok = R == 4 ? emu::run(256, order, small_panel) : emu::run(512, order, wide_panel);
  *barriers = emu::barriers;
  return ok ? err : -1;
}

extern "C" int hq_test_norm_cancelled(double nd, double thr) { return hq_norm_cancelled(nd, thr); }
