// vebi_noalloc.cu -- a pressure-Poisson solve that allocates nothing.
//
// Some callers cannot call cudaMalloc: a host framework whose own allocator owns all device
// memory (raw allocations are forbidden or invisible to its accounting), or a real-time time
// loop that must not allocate once it runs.  For them vebi_ppe_solve_noalloc runs the same
// BiCGSTAB as the time step on an ELL matrix and right-hand side the caller already holds in
// device memory, and keeps its Krylov vectors, block partial sums and barrier state in registers
// and in the file-scope array below instead of in allocated buffers.
//
// Limits and rules of the shared array:
//  * at most VEBI_NOALLOC_MAX_ROWS rows (65536); larger systems are rejected with VEBI_ERR_ARG;
//  * the array is ~4.3 MB and every GPU that loads this library holds it until the process exits;
//  * all calls on a device share it and it keeps the last call's contents: each call clears the
//    part that must start at zero (barrier counters, error word) before its kernel runs, and
//    calls that overlap on the GPU (two streams, or two host threads) race on it;
//  * the first call on a device looks up the array's device address (cudaGetSymbolAddress) with
//    that device current; make that first call before any stream capture begins.
//
// Errors: with iters_out or residual_out given, the call waits for the solve and returns its
// device-side status (VEBI_ERR_TIMEOUT if a grid barrier gave up).  With both NULL the call only
// enqueues the work and returns launch errors; a device-side failure then shows in the output,
// which the kernel fills with NaN.
#include <mutex>
#include <string>

#include "vebi_fp64.cuh"
#include "vebi_resident.cuh"

namespace vebi {

namespace {

constexpr int NA_VECS = 8;              // r, r_bar, v, p, p_inv, s, s_inv, t
constexpr int NA_MAX_BLOCKS = 2048;     // co-resident blocks the solver may use
constexpr int NA_SLOTS = 12;            // partial-sum slots (as in the step's solver)
constexpr size_t NA_CTRL = 32;          // doubles reserved for control words (256 B)
constexpr size_t NA_DOUBLES =
    NA_CTRL + (size_t)NA_VECS * VEBI_NOALLOC_MAX_ROWS + (size_t)NA_SLOTS * NA_MAX_BLOCKS;

// The scratch.  Host code must not take its address directly: in host code this name is a
// host-side stand-in, not a device address.  Host code uses the address from
// cudaGetSymbolAddress (g_dev_addr below); device code may name it directly.
static __device__ __align__(256) double g_noalloc_scratch[NA_DOUBLES];

struct NaCtrl {  // lives in the first NA_CTRL doubles of the scratch
  unsigned int bar_count;
  unsigned int bar_gen;
  int error;
  int iters;
  int warnings;
  int pad;
  double residual;
};

struct NaArgs {
  const int* cnt;
  const int* col;
  const double* val;
  const double* diag;
  const double* rhs;
  double* x;
  long long stride;
  int n;
  int closed;
  int itermax;
  double tol;
  double* scratch;  // device address of g_noalloc_scratch
};

constexpr unsigned long long NA_SPIN_LIMIT = 1ull << 25;

__device__ __forceinline__ bool na_sync(NaCtrl* c) {
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned int* vgen = &c->bar_gen;
    volatile int* verr = &c->error;
    unsigned int g = *vgen;
    __threadfence();
    unsigned int arrived = atomicAdd(&c->bar_count, 1u) + 1u;
    if (arrived == gridDim.x) {
      atomicExch(&c->bar_count, 0u);
      __threadfence();
      atomicAdd(&c->bar_gen, 1u);
    } else {
      unsigned long long spins = 0;
      while (*vgen == g) {
        if (*verr != 0) break;
        if (++spins > NA_SPIN_LIMIT) {
          atomicCAS(&c->error, 0, VEBI_ERR_TIMEOUT);
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
  }
  __syncthreads();
  return *((volatile int*)&c->error) == 0;
}

// A block that leaves the solve on an error (a barrier that timed out, or saw another block's
// timeout) fills its rows of x with NaN, so a failed solve cannot pass for a result even when
// the caller reads nothing back.  Every block reaches the barrier that failed or returns from
// it with the error, and the blocks' rows (i = tid, tid + stride, ...) cover 0..n-1.
__device__ __forceinline__ void na_fail_rows(double* x, int n, int tid, int stride) {
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  for (int i = tid; i < n; i += stride) x[i] = nan;
}

__device__ __forceinline__ void na_partials(double a, double b, int nval, double* part, double* sh) {
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
  }
  int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { sh[w] = a; sh[32 + w] = b; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double sa = 0.0, sb = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) { sa += sh[q]; sb += sh[32 + q]; }
    part[blockIdx.x] = sa;
    if (nval > 1) part[gridDim.x + blockIdx.x] = sb;
  }
  __syncthreads();
}

__device__ __forceinline__ void na_reduce(const double* part, int nb, int nval, double* out, double* shv) {
  if (threadIdx.x < 32) {
    for (int q = 0; q < nval; ++q) {
      double v = 0.0;
      for (int b = threadIdx.x; b < nb; b += 32) v += __ldcg(part + (size_t)q * nb + b);
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (threadIdx.x == 0) shv[q] = v;
    }
  }
  __syncthreads();
  for (int q = 0; q < nval; ++q) out[q] = shv[q];
  __syncthreads();
}

__device__ __forceinline__ double na_spmv(const NaArgs& a, const double* xv, int i) {
  double bb = a.diag[i] * __ldcg(xv + i);
  const int cnt = a.cnt[i];
  for (int k = 0; k < cnt; ++k) {
    size_t e = (size_t)k * a.stride + i;
    bb = fma(a.val[e], __ldcg(xv + a.col[e]), bb);
  }
  return bb;
}

constexpr int NA_T_MAX = 512;  // rows of a block, one thread a row
constexpr int NA_AHEAD = 16;   // a row's operands loaded at a time
constexpr int NA_KEEP = 64;    // slots of a row held in shared memory, if it takes as many

// SPARSE_PBICGSTAB_nonull / SPARSE_PBICGSTAB (linear_solver.F90:275-425 / 82-227) with x0 = 0
template <bool NONULL>
__global__ void __launch_bounds__(TPB) k_na_bicgstab(NaArgs a) {
  __shared__ double sh[64];
  __shared__ double shv[4];
  NaCtrl* ctl = reinterpret_cast<NaCtrl*>(a.scratch);
  const size_t N = VEBI_NOALLOC_MAX_ROWS;
  double* base = a.scratch + NA_CTRL;
  double *r = base, *rb = base + N, *v = base + 2 * N, *p = base + 3 * N, *pinv = base + 4 * N;
  double *sv = base + 5 * N, *sinv = base + 6 * N, *t = base + 7 * N;
  double* part = base + (size_t)NA_VECS * N;
  const int n = a.n, nb = gridDim.x;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  double* x = a.x;
  const double small = NONULL ? 1.0e-6 : 4.0;
  auto den = [&](int i) -> double { return NONULL ? (1.0 + 1.0e-15) : (a.diag[i] + 1.0e-15); };
  double red[4];
  double acc = 0.0;
  for (int i = tid; i < n; i += stride) {
    double bi = a.rhs[i];
    x[i] = 0.0;
    r[i] = bi;
    rb[i] = bi;
    v[i] = 0.0;
    p[i] = 0.0;
    acc += bi * bi;
  }
  na_partials(acc, 0.0, 1, part + 10 * (size_t)nb, sh);
  if (!na_sync(ctl)) { na_fail_rows(x, n, tid, stride); return; }
  na_reduce(part + 10 * (size_t)nb, nb, 1, red, shv);
  double rho = red[0], rho0 = 1.0, alpha = 1.0, omega = 1.0, n2r0 = 1.0, n2s0 = 1.0, resid = 0.0;
  int iter = 1, warn = 0;
  bool done = false;
  while (iter <= a.itermax) {
    if (rho == 0.0) { warn |= VEBI_WARN_BICGSTAB_BREAKDOWN; done = true; break; }
    double beta = rho / (rho0 + 1.0e-15) * alpha / (omega + 1.0e-15);
    acc = 0.0;
    for (int i = tid; i < n; i += stride) {
      double pi = (iter == 1) ? r[i] : r[i] + beta * (p[i] - omega * v[i]);
      p[i] = pi;
      acc += pi;
    }
    if (NONULL) {
      na_partials(acc, 0.0, 1, part, sh);
      if (!na_sync(ctl)) { na_fail_rows(x, n, tid, stride); return; }
      na_reduce(part, nb, 1, red, shv);
      const double mean = red[0] / (double)n;
      for (int i = tid; i < n; i += stride) {
        double pi = p[i] - mean;
        p[i] = pi;
        pinv[i] = pi / den(i);
      }
    } else {
      for (int i = tid; i < n; i += stride) pinv[i] = p[i] / den(i);
    }
    if (!na_sync(ctl)) { na_fail_rows(x, n, tid, stride); return; }
    acc = 0.0;
    for (int i = tid; i < n; i += stride) {
      double vi = na_spmv(a, pinv, i);
      v[i] = vi;
      acc += rb[i] * vi;
    }
    na_partials(acc, 0.0, 1, part + 2 * (size_t)nb, sh);
    if (!na_sync(ctl)) { na_fail_rows(x, n, tid, stride); return; }
    na_reduce(part + 2 * (size_t)nb, nb, 1, red, shv);
    alpha = rho / (red[0] + 1.0e-15);
    double a2 = 0.0;
    acc = 0.0;
    for (int i = tid; i < n; i += stride) {
      double si = r[i] - alpha * v[i];
      sv[i] = si;
      acc += si * si;
      a2 += si;
    }
    na_partials(acc, a2, 2, part + 4 * (size_t)nb, sh);
    if (!na_sync(ctl)) { na_fail_rows(x, n, tid, stride); return; }
    na_reduce(part + 4 * (size_t)nb, nb, 2, red, shv);
    const double n2s = red[0], mean_s = red[1] / (double)n;
    if (iter == 1) n2s0 = (n2s <= small) ? 1.0 : n2s;
    if (n2s <= a.tol * a.tol * n2s0) {
      for (int i = tid; i < n; i += stride) x[i] = x[i] + alpha * pinv[i];
      resid = sqrt(n2s / n2s0);
      done = true;
      break;
    }
    for (int i = tid; i < n; i += stride) {
      double si = sv[i];
      if (NONULL) { si = si - mean_s; sv[i] = si; }
      sinv[i] = si / den(i);
    }
    if (!na_sync(ctl)) { na_fail_rows(x, n, tid, stride); return; }
    acc = 0.0;
    a2 = 0.0;
    for (int i = tid; i < n; i += stride) {
      double ti = na_spmv(a, sinv, i);
      t[i] = ti;
      acc += ti * sv[i];
      a2 += ti * ti;
    }
    na_partials(acc, a2, 2, part + 6 * (size_t)nb, sh);
    if (!na_sync(ctl)) { na_fail_rows(x, n, tid, stride); return; }
    na_reduce(part + 6 * (size_t)nb, nb, 2, red, shv);
    omega = red[0] / (red[1] + 1.0e-15);
    acc = 0.0;
    a2 = 0.0;
    for (int i = tid; i < n; i += stride) {
      x[i] = x[i] + alpha * pinv[i] + omega * sinv[i];
      double ri = sv[i] - omega * t[i];
      r[i] = ri;
      acc += ri * ri;
      a2 += rb[i] * ri;
    }
    na_partials(acc, a2, 2, part + 8 * (size_t)nb, sh);
    if (!na_sync(ctl)) { na_fail_rows(x, n, tid, stride); return; }
    na_reduce(part + 8 * (size_t)nb, nb, 2, red, shv);
    const double n2r = red[0];
    if (iter == 1) n2r0 = (n2r <= small) ? 1.0 : n2r;
    resid = sqrt(n2r / n2r0);
    if (n2r <= a.tol * a.tol * n2r0) { done = true; break; }
    iter = iter + 1;
    rho0 = rho;
    rho = red[1];
  }
  if (!done) warn |= VEBI_WARN_MAXITER;
  if (tid == 0) {
    ctl->iters = iter;
    ctl->residual = resid;
    ctl->warnings = warn;
  }
}

// The same solve for up to NA_T_MAX rows per SM: the rows dealt in groups of 32 to one block per SM
// (vebi_resident.cuh), a row a thread.  The row's vectors stay in registers and its first slots in
// shared memory for the whole solve, so a product waits for L2 once per NA_AHEAD operands, all of
// them in flight, and not twice per slot; only p_inv, s_inv and the partial sums pass through L2.
// A row's product is one chain in slot order and every sum keeps k_na_bicgstab's order, so the
// solution is that kernel's bit for bit (compared on the CPU, where the number of SMs is a test's).
// What bounds it: up to two warps a scheduler, the chain of an iteration (seven barriers, five
// sums, two products of 45 dependent FMAs), ~24 us; above that the FP64 pipe, at ~150 operations a row.
// Measured against k_na_bicgstab, ms per solve: 576 rows x 24 iterations 0.57 / 1.45, 16k x 98
// 2.70 / 6.29 (open, x 164, 3.84 / 9.57), 36k x 142 4.90 / 9.61, 65k x 196 8.4 / 15.7.
template <bool NONULL>
__global__ void __launch_bounds__(NA_T_MAX, 1) k_na_resident(NaArgs a, int gpb, int nvb, int keep) {
  extern __shared__ double na_mat[];  // the first `keep` slots of the block's rows: values, then columns
  __shared__ ResSh sh;
  NaCtrl* ctl = reinterpret_cast<NaCtrl*>(a.scratch);
  const GridBar bar{&ctl->bar_count, &ctl->error};
  const int n = a.n, t = threadIdx.x, R = blockDim.x;
  const int i = blockIdx.x * R + t;
  const bool mine = i < n;
  double* const pinv_all = a.scratch + NA_CTRL;
  double* const sinv_all = pinv_all + VEBI_NOALLOC_MAX_ROWS;
  double* const parts = sinv_all + VEBI_NOALLOC_MAX_ROWS;
  const double small = NONULL ? 1.0e-6 : 4.0, dn = (double)n;
  double* const vals = na_mat + t;
  int* const cols = reinterpret_cast<int*>(na_mat + (size_t)keep * R) + t;
  const int cnt = mine ? a.cnt[i] : 0;
  for (int k = 0; k < keep && k < cnt; ++k) {
    vals[k * R] = a.val[(size_t)k * a.stride + i];
    cols[k * R] = a.col[(size_t)k * a.stride + i];
  }
  res_begin(sh);
  const double di = mine ? a.diag[i] : 0.0;
  const double den = NONULL ? (1.0 + 1.0e-15) : (di + 1.0e-15), rden = fp::reciprocal(fp::magnitude(den));
  const double rdn = fp::reciprocal(dn);
  // A's row times xv, slot after slot; NA_AHEAD operands are loaded at a time, before the chain
  // that adds those before them.  The chain is left by a branch for the whole warp: predicated off,
  // an FMA still takes its 64 cycles.
  const int shared_slots = min(cnt, keep), warp_slots = __reduce_max_sync(0xffffffffu, shared_slots);
  auto product = [&](const double* xv) {
    double u[2][NA_AHEAD];
    auto fetch = [&](int k0, double* o) {
#pragma unroll
      for (int e = 0; e < NA_AHEAD; ++e) o[e] = k0 + e < shared_slots ? __ldca(xv + cols[(k0 + e) * R]) : 0.0;
    };
    auto chain = [&](int k0, const double* o, double& b) {
#pragma unroll
      for (int e = 0; e < NA_AHEAD; ++e) {
        if (e % 2 == 0 && k0 + e >= warp_slots) return;
        if (k0 + e < shared_slots) b = fma(vals[(k0 + e) * R], o[e], b);
      }
    };
    fetch(0, u[0]);
    double b = mine ? di * __ldca(xv + i) : 0.0;
#pragma unroll 1
    for (int k = 0; k < warp_slots; k += 2 * NA_AHEAD) {
      fetch(k + NA_AHEAD, u[1]);
      chain(k, u[0], b);
      fetch(k + 2 * NA_AHEAD, u[0]);
      chain(k + NA_AHEAD, u[1], b);
    }
    for (int k = keep; k < cnt; ++k) {
      const size_t e = (size_t)k * a.stride + i;
      b = fma(a.val[e], __ldcg(xv + a.col[e]), b);
    }
    return b;
  };
  double r = mine ? a.rhs[i] : 0.0, rb = r, v = 0.0, p = 0.0, x = 0.0;
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  auto failed = [&]() {
    if (mine) a.x[i] = nan;
  };
  if (!res_reduce<1>(bar, mine ? plus_zero(r * r) : 0.0, 0.0, parts, gpb, nvb, sh, [&]() { sh.rho = sh.v[0]; }))
    return failed();
  int iter = 1, warn = 0;
  bool done = false, at_s = false;
  while (iter <= a.itermax) {
    if (is_zero(sh.rho)) { warn |= VEBI_WARN_BICGSTAB_BREAKDOWN; done = true; break; }
    p = iter == 1 ? r : r + sh.beta * (p - sh.omega * v);
    if (NONULL) {
      if (!res_reduce<1>(bar, mine ? plus_zero(p) : 0.0, 0.0, parts, gpb, nvb, sh, [&]() { sh.mean = fp::quotient(sh.v[0], dn, rdn); }))
        return failed();
      p = p - sh.mean;
    }
    const double pinv = fp::quotient(p, den, rden);
    if (mine) pinv_all[i] = pinv;
    if (!res_sync(bar)) return failed();
    v = product(pinv_all);
    if (!res_reduce<1>(bar, mine ? plus_zero(rb * v) : 0.0, 0.0, parts, gpb, nvb, sh,
                       [&]() { sh.alpha = fp::quotient(sh.rho, sh.v[0] + 1.0e-15); }))
      return failed();
    const double alpha = sh.alpha;
    double s = r - alpha * v, sinv = 0.0;
    if (!NONULL) {  // before the reduction, whose barrier the product needs anyway
      sinv = fp::quotient(s, den, rden);
      if (mine) sinv_all[i] = sinv;
    }
    if (!res_reduce<2>(bar, mine ? plus_zero(s * s) : 0.0, mine ? plus_zero(s) : 0.0, parts, gpb, nvb, sh, [&]() {
          sh.n2 = sh.v[0];
          if (iter == 1) sh.n2s0 = (sh.v[0] <= small) ? 1.0 : sh.v[0];
          sh.flag = sh.v[0] <= a.tol * a.tol * sh.n2s0;
          if (NONULL) sh.mean = fp::quotient(sh.v[1], dn, rdn);
        }))
      return failed();
    if (sh.flag) {
      x = x + alpha * pinv;
      done = at_s = true;
      break;
    }
    if (NONULL) {
      s = s - sh.mean;
      sinv = fp::quotient(s, den, rden);
      if (mine) sinv_all[i] = sinv;
      if (!res_sync(bar)) return failed();
    }
    const double tv = product(sinv_all);
    if (!res_reduce<2>(bar, mine ? plus_zero(tv * s) : 0.0, mine ? plus_zero(tv * tv) : 0.0, parts, gpb, nvb, sh,
                       [&]() { sh.omega = fp::quotient(sh.v[0], sh.v[1] + 1.0e-15); }))
      return failed();
    const double omega = sh.omega;
    x = x + alpha * pinv + omega * sinv;
    r = s - omega * tv;
    if (!res_reduce<2>(bar, mine ? plus_zero(r * r) : 0.0, mine ? plus_zero(rb * r) : 0.0, parts, gpb, nvb, sh, [&]() {
          sh.n2 = sh.v[0];
          if (iter == 1) sh.n2r0 = (sh.v[0] <= small) ? 1.0 : sh.v[0];
          sh.flag = sh.v[0] <= a.tol * a.tol * sh.n2r0;
          sh.beta = fp::quotient(fp::quotient(sh.v[1], sh.rho + 1.0e-15) * alpha, omega + 1.0e-15);
          sh.rho = sh.v[1];
        }))
      return failed();
    if (sh.flag) { done = true; break; }
    iter = iter + 1;
  }
  if (!done) warn |= VEBI_WARN_MAXITER;
  if (mine) a.x[i] = x;
  if (blockIdx.x == 0 && t == 0) {
    ctl->iters = iter;
    ctl->residual = sqrt(sh.n2 / (at_s ? sh.n2s0 : sh.n2r0));
    ctl->warnings = warn;
  }
}

// per-device set-up: the scratch's device address, looked up with that device current
constexpr int NA_MAX_DEVICES = 64;
std::mutex g_mu;
struct NaDevice {
  double* addr;
  int blocks;  // co-resident blocks of k_na_bicgstab
  int nsm;
  int shared;  // bytes of dynamic shared memory a block of k_na_resident may have
};
NaDevice g_dev[NA_MAX_DEVICES] = {};

}  // namespace
}  // namespace vebi

extern "C" void vebi_set_last_error_internal(const char* msg);

namespace vebi {
namespace {

int na_fail(int code, const std::string& m) {
  vebi_set_last_error_internal(m.c_str());
  return code;
}

}  // namespace
}  // namespace vebi

using namespace vebi;

extern "C" int vebi_ppe_solve_noalloc(const int32_t* ij_count, const int32_t* ppe_col, const double* ppe_val,
                                      const double* ppe_diag, const double* rhs, double* x, int32_t n,
                                      int64_t ell_stride, int32_t closed_domain, double tol, int32_t itermax,
                                      void* stream, int32_t* iters_out, double* residual_out) {
  if (!ij_count || !ppe_col || !ppe_val || !ppe_diag || !rhs || !x)
    return na_fail(VEBI_ERR_ARG, "vebi_ppe_solve_noalloc: null array");
  if (n < 1 || n > VEBI_NOALLOC_MAX_ROWS)
    return na_fail(VEBI_ERR_ARG, "vebi_ppe_solve_noalloc: n must be in 1..VEBI_NOALLOC_MAX_ROWS (65536)");
  if (ell_stride < n) return na_fail(VEBI_ERR_ARG, "vebi_ppe_solve_noalloc: ell_stride < n");
  if (!(tol > 0.0) || itermax < 1) return na_fail(VEBI_ERR_ARG, "vebi_ppe_solve_noalloc: bad tol/itermax");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NA_MAX_DEVICES)
    return na_fail(VEBI_ERR_NO_DEVICE, "vebi_ppe_solve_noalloc: no current CUDA device");
  NaDevice g;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    NaDevice& q = g_dev[dev];
    if (!q.addr) {
      void* p = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (e != cudaSuccess || !p)
        return na_fail(VEBI_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
      int nsm = 0, per = 0, per2 = 0, shared = 0;
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_na_bicgstab<true>, TPB, 0);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per2, k_na_bicgstab<false>, TPB, 0);
      per = per < per2 ? per : per2;
      q.nsm = nsm < 1 ? 1 : nsm;
      const long long b = (long long)(per < 1 ? 1 : per) * q.nsm;
      q.blocks = (int)(b > NA_MAX_BLOCKS ? NA_MAX_BLOCKS : b);
      cudaDeviceGetAttribute(&shared, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
      shared -= (int)sizeof(ResSh) + 1024;
      if (shared > 0 &&
          cudaFuncSetAttribute(k_na_resident<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, shared) == cudaSuccess &&
          cudaFuncSetAttribute(k_na_resident<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, shared) == cudaSuccess)
        q.shared = shared;
      else
        cudaGetLastError();  // k_na_bicgstab then
      q.addr = static_cast<double*>(p);
    }
    g = q;
  }
  double* const addr = g.addr;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (iters_out || residual_out) {
    // the read-back waits for the stream, which a stream being captured cannot do
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaError_t ce = cudaStreamIsCapturing(st, &cs);
    if (ce != cudaSuccess) return na_fail(VEBI_ERR_CUDA, std::string("cudaStreamIsCapturing: ") + cudaGetErrorString(ce));
    if (cs != cudaStreamCaptureStatusNone)
      return na_fail(VEBI_ERR_ARG, "vebi_ppe_solve_noalloc: iters_out and residual_out must be NULL while the "
                                   "stream is being captured (the read-back waits for the stream)");
  }
  // clear the control words; the vectors are initialised by the kernel itself
  cudaError_t e = cudaMemsetAsync(addr, 0, NA_CTRL * sizeof(double), st);
  if (e != cudaSuccess) return na_fail(VEBI_ERR_CUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
  NaArgs a{ij_count, ppe_col, ppe_val, ppe_diag, rhs, x, (long long)ell_stride, n, closed_domain ? 1 : 0,
           itermax, tol, addr};
  // k_na_resident wherever its rows fit, as it is the faster one up to the 65,536 rows of the array;
  // k_na_bicgstab is for a GPU (or a slice of one) of fewer than n / NA_T_MAX SMs
  cudaLaunchConfig_t cfg = {};
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const int nvb = (n + TPB - 1) / TPB, groups = nvb * RES_VB;
  int gpb = (groups + g.nsm - 1) / g.nsm;
  if (gpb < 2) gpb = 2;  // two warps: one for each of two sums
  const int rows = gpb * RES_GROUP;
  const int fit = rows <= NA_T_MAX ? g.shared / (12 * rows) : 0, keep = fit < NA_KEEP ? fit : NA_KEEP;
  if (keep > 0) {
    cfg.gridDim = dim3((groups + gpb - 1) / gpb);
    cfg.blockDim = dim3(rows);
    cfg.dynamicSmemBytes = (size_t)12 * rows * keep;
    e = closed_domain ? cudaLaunchKernelEx(&cfg, k_na_resident<true>, a, gpb, nvb, keep)
                      : cudaLaunchKernelEx(&cfg, k_na_resident<false>, a, gpb, nvb, keep);
  } else {
    cfg.gridDim = dim3(nvb < g.blocks ? nvb : g.blocks);
    cfg.blockDim = dim3(TPB);
    e = closed_domain ? cudaLaunchKernelEx(&cfg, k_na_bicgstab<true>, a) : cudaLaunchKernelEx(&cfg, k_na_bicgstab<false>, a);
  }
  if (e != cudaSuccess) return na_fail(VEBI_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(e));
  if (iters_out || residual_out) {
    NaCtrl ctl;
    e = cudaMemcpyAsync(&ctl, addr, sizeof(NaCtrl), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return na_fail(VEBI_ERR_CUDA, std::string("read-back: ") + cudaGetErrorString(e));
    if (iters_out) *iters_out = ctl.iters;
    if (residual_out) *residual_out = ctl.residual;
    if (ctl.error) return na_fail(ctl.error, "vebi_ppe_solve_noalloc: device-side error");
  }
  return VEBI_OK;
}
