// vebi_solver.cuh -- building blocks of the persistent cooperative PPE solvers: the bounded
// grid barrier, the deterministic block-partial reductions, the solver arguments and the
// FP64 ELL row product (sparse_atime, linear_solver.F90:254-273).
#pragma once
#include "vebi_ctx.cuh"

namespace vebi {

// polls of a grid barrier before it gives up: 1.9 to 2.1 s with 64 to 2 blocks on an idle GPU (a poll takes
// 0.22 to 0.25 us, measured), longer beside other traffic to L2
constexpr unsigned long long SPIN_LIMIT = 1ull << 23;

#ifdef VEBI_BARRIER_TIMESTAMPS
// Diagnostic build only (vebisph_gb300/barrier_profile.py): block 0 records the global timer
// when it arrives at and leaves every grid barrier, so the time of each solver phase and of the
// wait for the slowest block can be read back.  Each translation unit has its own copy; the
// solvers of vebi_mg.cu export theirs.
constexpr int BAR_TS_MAX = 16384;
static __device__ unsigned long long g_bar_ts[2][BAR_TS_MAX];
static __device__ unsigned int g_bar_n;
// every block's arrival time at the barriers BAR_ALL_FIRST .. BAR_ALL_FIRST + BAR_ALL_N - 1 of
// the solve (one iteration and more), and the SM each block runs on
constexpr int BAR_ALL_FIRST = 200, BAR_ALL_N = 64, BAR_ALL_BLOCKS = 2048;
static __device__ unsigned int g_bar_blk_n[BAR_ALL_BLOCKS];
static __device__ unsigned long long g_bar_all[BAR_ALL_N][BAR_ALL_BLOCKS];
static __device__ unsigned int g_bar_smid[BAR_ALL_BLOCKS];
__device__ __forceinline__ unsigned long long bar_clock() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
#endif

#ifdef VEBI_BARRIER_TIMESTAMPS
__device__ __forceinline__ void bar_mark(unsigned long long ts_arrive) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const unsigned int q = g_bar_n++;
    if (q < BAR_TS_MAX) {
      g_bar_ts[0][q] = ts_arrive;
      g_bar_ts[1][q] = bar_clock();
    }
  }
  if (threadIdx.x == 0 && blockIdx.x < BAR_ALL_BLOCKS) {
    const unsigned int q = g_bar_blk_n[blockIdx.x]++;
    if (q >= BAR_ALL_FIRST && q < BAR_ALL_FIRST + BAR_ALL_N) g_bar_all[q - BAR_ALL_FIRST][blockIdx.x] = ts_arrive;
    if (q == 0) {
      unsigned int sm;
      asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
      g_bar_smid[blockIdx.x] = sm;
    }
  }
}
#define BAR_ARRIVE const unsigned long long ts_arrive_ = bar_clock()
#define BAR_LEAVE bar_mark(ts_arrive_)
#else
#define BAR_ARRIVE (void)0
#define BAR_LEAVE (void)0
#endif

// ---- words that blocks of the grid signal each other through (gpu scope)
#ifdef __CUDACC__
__device__ __forceinline__ unsigned int atom_add_release(unsigned int* a, unsigned int v) {
  unsigned int old;
  asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(a), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* a) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a) : "memory");
  return v;
}
#else  // the emulation's that runs these kernels on the CPU
unsigned int atom_add_release(unsigned int* a, unsigned int v);
unsigned int ld_acquire(const unsigned int* a);
#endif

// Poll *word until done(value); false when more than `limit` polls go by (VEBI_ERR_TIMEOUT is
// recorded) or another block has recorded an error, looked at every 64th poll.  A poll is one
// round trip to L2 (0.22-0.25 us), so sleeping between polls only adds to the wait.
template <class Done>
__device__ __forceinline__ bool poll_bounded(const unsigned int* word, int* error, unsigned long long limit, Done done) {
  for (unsigned long long spins = 0;; ++spins) {
    if (done(ld_acquire(word))) return true;
    if ((spins & 63) == 63 && *((volatile int*)error) != 0) return false;
    if (spins >= limit) {
      atomicCAS(error, 0, VEBI_ERR_TIMEOUT);
      return false;
    }
  }
}

// Arrival and wait of one thread per block at the grid barrier.  Block 0 adds 2^31 less the
// other blocks' number and every other block adds one, so the counter's top bit flips when all
// have arrived and its low bits return to zero: one atomic per block and no reset, which a
// waiter would otherwise see one round trip later.
__device__ __forceinline__ bool barrier_arrive_wait(unsigned int* count, int* error, unsigned long long limit) {
  const unsigned int old = atom_add_release(count, blockIdx.x == 0 ? 0x80000000u - (gridDim.x - 1u) : 1u);
  return poll_bounded(count, error, limit, [=](unsigned int cur) { return ((cur ^ old) & 0x80000000u) != 0u; });
}

// bounded grid-wide barrier for a co-resident (cooperative) grid; false on error/timeout.
// A block that polls more than `limit` times records VEBI_ERR_TIMEOUT and returns false, and so
// does every block that is waiting, or comes to wait, after an error is recorded.  The writes of
// every thread before it are visible to every thread after it: the block barriers order them
// with thread 0's release and acquire.
// Measured with 7 / 152 / 760 blocks of 256 threads: 0.68 / 1.17 / 2.6 us; with a reset counter,
// a generation word and fences around volatile polls it was 1.6 / 2.9 / 7.4 us.
__device__ __forceinline__ bool grid_sync_bounded(Scal* s, unsigned long long limit) {
  BAR_ARRIVE;
  __syncthreads();
  int bad = 0;
  if (threadIdx.x == 0) bad = barrier_arrive_wait(&s->bar_count, &s->error, limit) ? 0 : 1;
  bad = __syncthreads_or(bad);
  BAR_LEAVE;
  return bad == 0;
}

__device__ __forceinline__ bool grid_sync(Scal* s) { return grid_sync_bounded(s, SPIN_LIMIT); }

// a solve starts only on a state without a recorded failure (of this step or an earlier one)
__device__ __forceinline__ bool state_failed(const Scal* s) {
  return *((const volatile int*)&s->first_error) != 0 || *((const volatile int*)&s->error) != 0;
}

// ---- grid-wide sums
// Shared memory of a solver block: the reductions' work space, the last reduction's results (up
// to four values derived from the sums and a flag, the same in every block) and the iteration's
// scalars, which thread 0 updates and every thread reads where a pass needs one.
struct SolverSh {
  double x[2][TPB];       // one value per thread
  double y[TPB];          // after the first tree level of two values
  double w[2][TPB / 32];  // warp sums
  double v[4];
  double rho, alpha, omega, beta, n2r0, n2s0, n2;
  int flag;
};

__device__ __forceinline__ double plus_zero(double x) {  // 0.0 + x without the FP64 pipe
  const long long b = __double_as_longlong(x);
  return __longlong_as_double(b == (long long)0x8000000000000000ull ? 0ll : b);
}

// Block partial of one or two values into part[q*nb + blockIdx.x], by thread q.  The sums are
// those of a shuffle tree over each warp (lane l + lane l+16, then 8, 4, 2, 1) and of the warps
// in order.  An FP64 instruction holds a warp scheduler for 64-76 cycles on this GPU however few
// of its lanes are active, so the tree is packed: the 16 sums of a warp's first level take half a
// warp, and only as many warps run it as it fills (20 instructions a value in place of 40).
template <int NV>
__device__ __forceinline__ void block_partial(double a, double b, double* part, SolverSh& sh) {
  constexpr int W = TPB / 32;
  const int t = threadIdx.x;
  sh.x[0][t] = a;
  if (NV > 1) sh.x[1][t] = b;
  __syncthreads();
  if (NV == 1) {
    if (t < TPB / 2) {
      const double* q = sh.x[0] + (t >> 4) * 32 + (t & 15);
      double y = q[0] + q[16];
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) y += __shfl_down_sync(0xffffffffu, y, o, 16);
      if ((t & 15) == 0) sh.w[0][t >> 4] = y;
    }
  } else {
    const double* q = sh.x[t / (TPB / 2)] + ((t % (TPB / 2)) >> 4) * 32 + (t & 15);
    sh.y[t] = q[0] + q[16];
    __syncthreads();
    if (t < TPB / 2) {
      const double* r = sh.y + (t >> 3) * 16 + (t & 7);
      double y = r[0] + r[8];
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) y += __shfl_down_sync(0xffffffffu, y, o, 8);
      if ((t & 7) == 0) sh.w[(t >> 3) / W][(t >> 3) % W] = y;
    }
  }
  __syncthreads();
  if (t < NV) {
    double v = plus_zero(sh.w[t][0]);
#pragma unroll
    for (int q = 1; q < W; ++q) v += sh.w[t][q];
    part[(size_t)t * gridDim.x + blockIdx.x] = v;
  }
  if (t < 32) __syncwarp();
}

// Sum of n terms that other blocks of this launch wrote, by one warp in a fixed order: lane l takes
// terms l, l+32, ... in order, then the lanes by a shuffle tree (levels that would only add the
// zeros of lanes without a term are skipped).  The sum is lane 0's.  Up to 512 terms are loaded at
// once, so the warp waits for L2 once or twice, not once per 32 terms.  The adds leave their chain
// by a branch: predicated off, an FP64 add still takes its 64 cycles of the scheduler.  Measured
// with 8 / 12 / 16 / 24 loads ahead: the 100k-particle solve 46.3 / 46.1 / 45.3 / 49.9 ms (24
// spill), 51.4 with one at a time.
constexpr int SUM_AHEAD = 16;
static __device__ __noinline__ double warp_sum_in_order(const double* p, int n) {
  const int lane = threadIdx.x & 31;
  double v = 0.0;
  int b = 0;
  do {
    double u[SUM_AHEAD];
#pragma unroll
    for (int e = 0; e < SUM_AHEAD; ++e) {
      const int k = b + 32 * e + lane;
      u[e] = k < n ? __ldcg(p + k) : 0.0;
    }
    v = b == 0 ? plus_zero(u[0]) : v + u[0];
#pragma unroll
    for (int e = 1; e < SUM_AHEAD; ++e) {
      if (b + 32 * e >= n) break;
      v += u[e];
    }
    b += 32 * SUM_AHEAD;
  } while (b < n);
#pragma unroll 1
  for (int o = n > 16 ? 16 : n > 8 ? 8 : n > 4 ? 4 : n > 2 ? 2 : n > 1 ? 1 : 0; o > 0; o >>= 1)
    v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// sum of the block partials of value q into sh.v[q], by warp q
template <int NV>
__device__ __forceinline__ void sum_partials(const double* part, int nb, SolverSh& sh) {
  const int q = threadIdx.x >> 5;
  if (q < NV) {
    const double v = warp_sum_in_order(part + (size_t)q * nb, nb);
    if ((threadIdx.x & 31) == 0) sh.v[q] = v;
  }
  if (NV > 1) __syncthreads();
}

// every solver's first statement; the caller's first barrier orders it before any use
__device__ __forceinline__ void solver_begin(SolverSh& sh) {
  if (threadIdx.x == 0) {
    sh.alpha = sh.omega = sh.n2r0 = sh.n2s0 = 1.0;
    sh.beta = sh.n2 = 0.0;
  }
}

// The part of grid_reduce that does not depend on the caller's post, one copy per kernel: the
// sums in sh.v[0..NV-1] for thread 0.
template <int NV>
static __device__ __noinline__ bool grid_sums(Scal* s, double a, double b, double* part, SolverSh& sh) {
  block_partial<NV>(a, b, part, sh);
  int bad = 0;
  if (threadIdx.x == 0) bad = barrier_arrive_wait(&s->bar_count, &s->error, SPIN_LIMIT) ? 0 : 1;
  if (__syncthreads_or(bad)) return false;
  sum_partials<NV>(part, gridDim.x, sh);
  return true;
}

// Grid-wide sums of one or two values, which are also a grid barrier; false on error/timeout.
// post(v, flag), run by thread 0 on the sums v[0..NV-1], derives the iteration's scalars in
// v[0..3], in sh and in a flag (its divisions, square roots and comparisons), so uniform FP64
// work is done once per block and not by every warp.  Every block sums the partials itself: a
// form in which the last block to arrive did it for all, at one more round trip, was slower from
// 7 to 760 blocks (the 100k-particle FP64 solve 55.5 ms against 51.7).
// `part` takes NV * gridDim.x block partials.
template <int NV, class Post>
__device__ __forceinline__ bool grid_reduce(Scal* s, double a, double b, double* part, SolverSh& sh, Post post) {
  BAR_ARRIVE;
  if (!grid_sums<NV>(s, a, b, part, sh)) return false;
  if (threadIdx.x == 0) {
    sh.flag = 0;
    post(sh.v, sh.flag);
  }
  __syncthreads();
  BAR_LEAVE;
  return true;
}

// A vector pass over the rows tid, tid + stride, ... with each row's operands loaded one row
// ahead: load(i) returns row i's operands, body(i, ops) does the arithmetic and the stores.
// The next row's loads are issued before the current row's arithmetic, so a warp waiting for
// the FP64 pipe (2 lanes per clock per SM on this GPU) already has its next loads in flight.
// Rows are visited in the same order as a plain loop, so sums come out bit for bit the same.
template <class Load, class Body>
__device__ __forceinline__ void rows_ahead(int tid, int stride, int n, Load load, Body body) {
  if (tid >= n) return;
  auto cur = load(tid);
  for (int i = tid; i < n; i += stride) {
    auto nxt = cur;
    if (i + stride < n) nxt = load(i + stride);
    body(i, cur);
    cur = nxt;
  }
}

// Solver arguments: only what the loop touches (keeps the kernel's register footprint small).
struct BiArgs {
  double *x, *r, *rb, *v, *p, *pinv, *s, *sinv, *t, *rinvM, *part, *P;
  const double *B, *diag, *val;
  const int *col, *cnt;
  Scal* sc;
  long long stride;
  int n, itermax;
  double tol;
  int warm;
};

// y_i = A_ii x_i + sum_k A_ik x_col(ik)  (sparse_atime, linear_solver.F90:254-273).  Four
// interleaved accumulators keep four independent load chains (column -> x) in flight per thread.
// x was written inside this kernel by other blocks: the grid barrier's release/acquire fences
// (gpu scope, followed by a CTA barrier) make those writes visible to the L1-cached loads
// (ld.global.ca) that follow, as in a cooperative-groups grid sync; neighbouring rows share most
// of their columns, so the gathers mostly hit L1.
__device__ __forceinline__ double spmv_row(const BiArgs& a, const double* xv, int i) {
  const int cnt = __ldg(a.cnt + i);
  const double* vp = a.val + i;
  const int* cp = a.col + i;
  const long long st = a.stride;
  double b0 = __ldg(a.diag + i) * __ldca(xv + i), b1 = 0.0, b2 = 0.0, b3 = 0.0;
  int k = 0;
  for (; k + 3 < cnt; k += 4) {
    const int c0 = __ldg(cp), c1 = __ldg(cp + st), c2 = __ldg(cp + 2 * st), c3 = __ldg(cp + 3 * st);
    const double v0 = __ldg(vp), v1 = __ldg(vp + st), v2 = __ldg(vp + 2 * st), v3 = __ldg(vp + 3 * st);
    b0 = fma(v0, __ldca(xv + c0), b0);
    b1 = fma(v1, __ldca(xv + c1), b1);
    b2 = fma(v2, __ldca(xv + c2), b2);
    b3 = fma(v3, __ldca(xv + c3), b3);
    cp += 4 * st;
    vp += 4 * st;
  }
  for (; k < cnt; ++k) {
    b0 = fma(__ldg(vp), __ldca(xv + __ldg(cp)), b0);
    cp += st;
    vp += st;
  }
  return (b0 + b1) + (b2 + b3);
}

// ---- mixed precision: FP64 recurrences, FP32 difference-form SpMV (see vebi_ppe.cu)
struct MxArgs {
  double *x, *r, *rb, *v, *p, *s, *t, *rinvM, *part, *P;
  float2 *pi, *si;                     // p_inv, s_inv as (hi, lo)
  const double *B, *rs;                // right-hand side, FP64 row sums
  const float* val32;
  const int *col, *cnt;
  Scal* sc;
  long long stride;
  int n, itermax;
  double tol;
  int warm;
};

// (hi, lo) FP32 pair of a double and back; conversions on the integer pipe (widen, narrow)
__device__ __forceinline__ float2 split2(double v) {
  const float h = narrow(v);
  return make_float2(h, narrow(v - widen(h)));
}
__device__ __forceinline__ double join2(float2 q) { return widen(q.x) + widen(q.y); }

__device__ __forceinline__ double spmv_diff32(const MxArgs& a, const float2* xv, int i) {
  const int cnt = __ldg(a.cnt + i);
  const float* vp = a.val32 + i;
  const int* cp = a.col + i;
  const long long st = a.stride;
  const float2 xi = __ldca(xv + i);
  float b0 = 0.0f, b1 = 0.0f, b2 = 0.0f, b3 = 0.0f;
  int k = 0;
  for (; k + 3 < cnt; k += 4) {
    const int c0 = __ldg(cp), c1 = __ldg(cp + st), c2 = __ldg(cp + 2 * st), c3 = __ldg(cp + 3 * st);
    const float v0 = __ldg(vp), v1 = __ldg(vp + st), v2 = __ldg(vp + 2 * st), v3 = __ldg(vp + 3 * st);
    const float2 x0 = __ldca(xv + c0), x1 = __ldca(xv + c1), x2 = __ldca(xv + c2), x3 = __ldca(xv + c3);
    b0 = fmaf(v0, (x0.x - xi.x) + (x0.y - xi.y), b0);
    b1 = fmaf(v1, (x1.x - xi.x) + (x1.y - xi.y), b1);
    b2 = fmaf(v2, (x2.x - xi.x) + (x2.y - xi.y), b2);
    b3 = fmaf(v3, (x3.x - xi.x) + (x3.y - xi.y), b3);
    cp += 4 * st;
    vp += 4 * st;
  }
  for (; k < cnt; ++k) {
    const float2 x0 = __ldca(xv + __ldg(cp));
    b0 = fmaf(__ldg(vp), (x0.x - xi.x) + (x0.y - xi.y), b0);
    cp += st;
    vp += st;
  }
  return fma(__ldg(a.rs + i), join2(xi), widen((b0 + b1) + (b2 + b3)));
}

}  // namespace vebi
