// vebi_resident.cu -- the FP64 BiCGSTAB of a small or medium PPE, spread over the whole GPU with
// its vectors in registers.
//
//  SPARSE_PBICGSTAB_nonull (closed)       linear_solver.F90:275-425
//  SPARSE_PBICGSTAB (open, Jacobi)        linear_solver.F90:82-227
//
// k_bicgstab (vebi_ppe.cu) gives each block 256 rows and each row one thread.  On a small system
// that leaves SMs idle -- a 10k-row solve occupies 40 of 152 -- and each row walks its 44 slots
// through two dependent trips to L2 per four slots, after every barrier.  Here the rows are dealt
// in groups of 32 to one block per SM, up to 256 rows a block:
//  * a product takes four lanes a row, one for each of the four interleaved accumulators of
//    spmv_row, so a row waits for its slots' operands once; up to 56 slots of a row stay in its
//    lanes' registers for the whole solve when a block has at most 128 rows;
//  * each row's r, r_bar, v, p, s, t, x stay in its thread's registers: only the gathered vectors
//    p_inv and s_inv and the reductions' partial sums pass through L2.
// Every sum runs in k_bicgstab's order -- a shuffle tree over 32 rows, the eight groups of a
// virtual block of 256 rows in sequence, the virtual blocks in lane order -- so the solution is
// the same bit for bit, whatever the number of SMs.
//
// What bounds it.  FP64 issues one warp instruction per 64-76 cycles and scheduler on this GPU:
// ~107 operations a row and iteration are 64 cycles per row of an SM (2 us at 66 rows).  The
// dependent chain of an iteration is the rest: five to seven barriers of ~1.1 us, five sums of some 20
// dependent adds (0.6-1 us with their load), six quotients of ~0.2 us, two products' gathers.
// Measured, ms per solve, k_bicgstab / this kernel: 1.7k rows x 60 iterations 2.39 / 1.16, 2.9k x
// 75 (open) 2.48 / 1.25, 10k x 139 5.37 / 3.36, 20k x 363 14.9 / 12.0, 29k x 247 10.2 / 9.7.
#include <atomic>

#include "vebi_resident.cuh"

namespace vebi {

namespace {

constexpr int RES_MAX_ROWS = 256;   // rows of a block: four lanes a row fill it

// One of a row's four lanes: lane q has spmv_row's accumulator q, which takes slots q, q+4, ... of
// the whole quads of slots; lane 0 also takes the diagonal before them and the up to three slots
// after them.
struct LaneRow {
  int row, q, nq, cnt;  // row (or -1), lane, whole quads, slots
  __device__ __forceinline__ LaneRow(const BiArgs& a, int row_, bool in)
      : row(in ? row_ : -1), q((int)threadIdx.x & 3), nq(0), cnt(0) {
    if (in) {
      cnt = __ldg(a.cnt + row);
      nq = cnt >> 2;
    }
  }
  // N slots k(u), u = 0.. N-1, of which those with in(u): columns and values, then operands, then FMAs
  template <int N, class Slot, class In, class Value>
  __device__ __forceinline__ void slots(const BiArgs& a, const double* xv, double& b, Slot k, In in, Value value) const {
    int c[N];
    double v[N], x[N];
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const long long o = (long long)k(u) * a.stride + row;
      c[u] = in(u) ? __ldg(a.col + o) : 0;
      v[u] = in(u) ? __ldg(a.val + o) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < N; ++u) x[u] = in(u) ? __ldca(xv + c[u]) : 0.0;
#pragma unroll
    for (int u = 0; u < N; ++u)
      if (in(u)) b = fma(v[u], value(x[u]), b);
  }
};

// KEEP: this many quads of a row stay in registers for the whole solve (0: all come from L2).
// RAW (closed domains): the products gather p and s and take off the mean and scale as they do, twice the
// FP64 operations a slot for two barriers less.
template <bool NONULL, int T_MAX, int KEEP, bool RAW = false>
__global__ void __launch_bounds__(T_MAX, 1) k_bicgstab_resident(BiArgs a, int gpb, int nvb) {
  __shared__ ResSh sh;
  __shared__ double vec[RES_MAX_ROWS];  // a product's results, by row of the block
  // the vector a product gathers goes out before the reduction that precedes the product, whose barrier
  // then is the only one: s_inv of an open domain as it is; with RAW, p and s before their mean is known
  constexpr bool EARLY = RAW || !NONULL;
  const int n = a.n, t = threadIdx.x;
  const int R = gpb * RES_GROUP, row0 = blockIdx.x * R;
  Scal* s = a.sc;
  if (state_failed(s)) return;
  const GridBar bar{&s->bar_count, &s->error};
  const double rinv1 = 1.0 / (1.0 + 1.0e-15);
  const double small = NONULL ? 1.0e-6 : 4.0;  // open solver: the integer expression 10-6
  const double dn = (double)n, rdn = fp::reciprocal(dn), tol2 = a.tol * a.tol;
  res_begin(sh);
  // this thread's row in the vector passes
  const int i = row0 + t;
  const bool mine = t < R && i < n;
  const int l = t >> 2;  // this lane's row of the block in the products
  const LaneRow L(a, row0 + l, l < R && row0 + l < n);
  int ck[KEEP ? KEEP : 1];
  double vk[KEEP ? KEEP : 1];
  double dk = 0.0;
  if (L.row >= 0 && L.q == 0) dk = __ldg(a.diag + L.row);
  if (KEEP && L.row >= 0) {
#pragma unroll
    for (int e = 0; e < KEEP; ++e) {
      const long long o = (4ll * e + L.q) * a.stride + L.row;
      ck[e] = e < L.nq ? __ldg(a.col + o) : 0;
      vk[e] = e < L.nq ? __ldg(a.val + o) : 0.0;
    }
  }
  // y = A x for the block's rows, to their threads (x complete and visible in every block)
  auto product = [&](const double* xv, double shift) {
    auto value = [&](double x) { return RAW ? fp::mul_int(x - shift, rinv1) : x; };
    double b = 0.0;
    if (L.row >= 0) {
      if (KEEP) {
        double x[KEEP ? KEEP : 1];
#pragma unroll
        for (int e = 0; e < KEEP; ++e) x[e] = e < L.nq ? __ldca(xv + ck[e]) : 0.0;
        if (L.q == 0) b = dk * value(__ldca(xv + L.row));
#pragma unroll
        for (int e = 0; e < KEEP; ++e)
          if (e < L.nq) b = fma(vk[e], value(x[e]), b);
      } else if (L.q == 0) {
        b = dk * value(__ldca(xv + L.row));
      }
      constexpr int Q = KEEP ? 4 : 6;
#pragma unroll 1
      for (int m = KEEP; m < L.nq; m += Q)
        L.slots<Q>(a, xv, b, [&](int u) { return 4 * (m + u) + L.q; }, [&](int u) { return m + u < L.nq; }, value);
      if (L.q == 0)
        L.slots<3>(a, xv, b, [&](int u) { return 4 * L.nq + u; }, [&](int u) { return 4 * L.nq + u < L.cnt; }, value);
    }
    b += __shfl_xor_sync(0xffffffffu, b, 1);  // (b0 + b1) + (b2 + b3)
    b += __shfl_xor_sync(0xffffffffu, b, 2);
    if (L.q == 0 && L.row >= 0) vec[l] = b;
    __syncthreads();
    return mine ? vec[t] : 0.0;
  };
  double r = 0.0, rb = 0.0, v = 0.0, p = 0.0, x = 0.0, rinvM = rinv1;
  if (a.warm) {  // x0 = P of the previous step: r0 = B - A x0
    if (mine) {
      x = a.P[i];
      a.pinv[i] = x;
    }
    if (!grid_sync(s)) return;
    const double y = product(a.pinv, 0.0);
    if (mine) r = a.B[i] - y;
    if (!grid_sync(s)) return;  // every product has read x0 before p_inv is written
  } else if (mine) {
    r = a.B[i];
  }
  rb = r;
  if (!NONULL && mine) rinvM = 1.0 / (__ldg(a.diag + i) + 1.0e-15);
  if (!res_reduce<1>(bar, mine ? fma(r, r, 0.0) : 0.0, 0.0, a.part, gpb, nvb, sh, [&]() { sh.rho = sh.v[0]; })) return;
  int iter = 1, warn = 0;
  bool done = false, at_s = false;
  while (iter <= a.itermax) {
    if (is_zero(sh.rho)) { warn |= VEBI_WARN_BICGSTAB_BREAKDOWN; done = true; break; }
    if (mine) p = iter == 1 ? r : fma(sh.beta, fma(-sh.omega, v, p), r);
    if (RAW && mine) a.pinv[i] = p;
    if (NONULL) {
      if (!res_reduce<1>(bar, mine ? plus_zero(p) : 0.0, 0.0, a.part, gpb, nvb, sh, [&]() { sh.mean = fp::quotient(sh.v[0], dn, rdn); }))
        return;
      p = p - sh.mean;
    }
    const double pinv = p * rinvM;
    if (!RAW) {
      if (mine) a.pinv[i] = pinv;
      if (!grid_sync(s)) return;
    }
    v = product(a.pinv, sh.mean);
    if (!res_reduce<1>(bar, mine ? fma(rb, v, 0.0) : 0.0, 0.0, a.part, gpb, nvb, sh,
                       [&]() { sh.alpha = fp::quotient(sh.rho, sh.v[0] + 1.0e-15); }))
      return;
    const double alpha = sh.alpha;
    double sv = mine ? fma(-alpha, v, r) : 0.0;
    if (EARLY && mine) a.sinv[i] = NONULL ? sv : sv * rinvM;
    if (!res_reduce<2>(bar, mine ? fma(sv, sv, 0.0) : 0.0, mine ? plus_zero(sv) : 0.0, a.part, gpb, nvb, sh, [&]() {
          sh.n2 = sh.v[0];
          if (iter == 1) sh.n2s0 = (sh.v[0] <= small) ? 1.0 : sh.v[0];
          sh.flag = sh.v[0] <= tol2 * sh.n2s0;
          if (NONULL) sh.mean = fp::quotient(sh.v[1], dn, rdn);
        }))
      return;
    if (sh.flag) {
      x = fma(alpha, pinv, x);
      done = at_s = true;
      break;
    }
    if (NONULL) sv = sv - sh.mean;
    const double sinv = sv * rinvM;
    if (!EARLY) {
      if (mine) a.sinv[i] = sinv;
      if (!grid_sync(s)) return;
    }
    const double tv = product(a.sinv, sh.mean);
    if (!res_reduce<2>(bar, mine ? fma(tv, sv, 0.0) : 0.0, mine ? fma(tv, tv, 0.0) : 0.0, a.part, gpb, nvb, sh,
                       [&]() { sh.omega = fp::quotient(sh.v[0], sh.v[1] + 1.0e-15); }))
      return;
    const double omega = sh.omega;
    x = fma(omega, sinv, fma(alpha, pinv, x));
    r = fma(-omega, tv, sv);
    if (!res_reduce<2>(bar, mine ? fma(r, r, 0.0) : 0.0, mine ? fma(rb, r, 0.0) : 0.0, a.part, gpb, nvb, sh, [&]() {
          sh.n2 = sh.v[0];
          if (iter == 1) sh.n2r0 = (sh.v[0] <= small) ? 1.0 : sh.v[0];
          sh.flag = sh.v[0] <= tol2 * sh.n2r0;
          sh.beta = fp::quotient(fp::quotient(sh.v[1], sh.rho + 1.0e-15) * alpha, omega + 1.0e-15);
          sh.rho = sh.v[1];
        }))
      return;
    if (sh.flag) { done = true; break; }
    iter = iter + 1;
  }
  if (!done) warn |= VEBI_WARN_MAXITER;
  if (mine) a.P[i] = x;
  if (blockIdx.x == 0 && t == 0) {
    s->ls_iters = iter;
    s->ls_iters_total += iter;
    s->ls_residual = sqrt(sh.n2 / (at_s ? sh.n2s0 : sh.n2r0));
    atomicOr(&s->warnings, warn);
  }
}

}  // namespace

// doubles of partial sums the resident solver needs for n rows: two areas of two sums a group
size_t resident_partials(int n) { return 4 * (size_t)RES_VB * ((n + 255) / 256); }

namespace {

// groups of rows per SM, or 0 when the solve does not fit: at most 256 rows (eight groups, four lanes a
// row) per SM, and a caller whose k_bicgstab grid has one row per thread (ceil(n / 256) blocks, whose
// summation order this kernel keeps).  Above 256 rows an SM the FP64 pipe is busy either way: 60k /
// 100k rows with two rows or one lane a row took 33 / 47 ms against k_bicgstab's 32 / 48.
int resident_groups(const Ctx& x, int n) {
  const int nvb = (n + TPB - 1) / TPB;
  if (nvb > x.coop_blocks || nvb > RES_MAX_VB) return 0;
  const int gpb = (nvb * RES_VB + x.nsm - 1) / x.nsm;
  return gpb * RES_GROUP <= RES_MAX_ROWS ? gpb : 0;
}

// From two groups per SM on, one spread solve fills the register files, so those of several contexts
// that host threads step at the same time follow one another; k_bicgstab takes few SMs and overlaps.
// So a spread solve of that size is for a call that has the GPU to itself.  Steps per second of 1 / 2 /
// 4 / 8 / 16 contexts with a thread each, spread / k_bicgstab: 10k rows 255 / 295 / 289 / 293 / 294 and
// 193 / 381 / 653 / 1037 / 1363, 20k 149 / 156 / 156 / 156 / 155 and 135 / 243 / 371 / 475 / 503; one
// group per SM, 1.7k rows, 718 / 1360 / 2459 / 4104 / 5108 and 465 / 893 / 1752 / 3377 / 6259.  The bits
// are the same either way.
bool by_company(int gpb) { return gpb > 1; }

std::atomic<int> g_stepping[64];  // calls in progress by device
std::atomic<int>& stepping(int device) { return g_stepping[device < 64 ? device : 63]; }

}  // namespace

Stepping::Stepping(int device_) : device(device_) { ++stepping(device); }
Stepping::~Stepping() { --stepping(device); }
bool stepping_alone(int device) { return stepping(device) <= 1; }

// whether the kernel of x's solve depends on x.alone, and so the captured step does
bool resident_by_company(const Ctx& x) {
  return x.precision == VEBI_PREC_FP64 && x.c.precond == 0 && !x.in_batch && x.solver_rows_per_thread <= 1 &&
         by_company(resident_groups(x, x.c.npfb));
}

// Runs the solve when it fits and the GPU is free for it.  false: not launched.
bool launch_bicgstab_resident(Ctx& x, const BiArgs& a, bool nonull) {
  const int gpb = resident_groups(x, a.n), nvb = (a.n + TPB - 1) / TPB;
  if (!gpb || (by_company(gpb) && !x.alone)) return false;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((nvb * RES_VB + gpb - 1) / gpb);
  cfg.blockDim = dim3(4 * gpb * RES_GROUP);
  cfg.stream = x.st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  auto go = [&](auto closed, auto open) { return cudaLaunchKernelEx(&cfg, nonull ? closed : open, a, gpb, nvb); };
  // RAW while an SM has one group of rows: 40^2 / 60^2 / 80^2 particles (one, one, two groups) without and
  // with it 1.21 / 2.79 / 2.60 and 1.16 / 2.72 / 2.65 ms
  const cudaError_t e =
      nonull && !a.warm && gpb == 1 ? cudaLaunchKernelEx(&cfg, k_bicgstab_resident<true, 512, 14, true>, a, gpb, nvb)
      : cfg.blockDim.x <= 512       ? go(k_bicgstab_resident<true, 512, 14>, k_bicgstab_resident<false, 512, 14>)
                                    : go(k_bicgstab_resident<true, 1024, 0>, k_bicgstab_resident<false, 1024, 0>);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  x.launches++;
  return true;
}

}  // namespace vebi
