// vebi_resident.cuh -- grid-wide sums for solvers that keep a row's vectors in a thread's registers
// and deal the rows in groups of 32 to one block per SM, in the order of a grid of 256-row blocks.
#pragma once
#include "vebi_solver.cuh"

namespace vebi {

struct GridBar {  // the barrier's counter and the word that errors are recorded in
  unsigned int* count;
  int* error;
};

constexpr int RES_GROUP = 32;       // rows of a group (a warp's rows in the vector passes)
constexpr int RES_VB = 8;           // groups of a virtual block (256 rows)
constexpr int RES_MAX_VB = 256;     // virtual blocks the shared table holds

struct ResSh {
  double vb[2 * RES_MAX_VB]; // virtual-block sums
  double v[2];
  double rho, alpha, omega, beta, n2r0, n2s0, n2, mean;
  int flag, turn;
};

// every resident solver's first statement
__device__ __forceinline__ void res_begin(ResSh& sh) {
  if (threadIdx.x == 0) {
    sh.alpha = sh.omega = sh.n2r0 = sh.n2s0 = 1.0;
    sh.beta = sh.n2 = 0.0;
    sh.turn = 0;
  }
  __syncthreads();
}

// the grid-wide sums of a and (NV = 2) b over all rows, a barrier among them: for thread 0 the
// totals are in sh.v when this returns true.
// The partial sums go to one of two areas of `parts`, each reduction to the one that the last did not
// take.  A reduction writes its area before its barrier and reads it after, and a block that has read
// goes on to the next reduction's writes while a slower one still reads: those two must not share an
// area.  Two are enough, as a block writes an area again only past the barrier of the reduction between,
// at which every block arrives after its reads.  The turn is kept here and not written into the solvers:
// a closed domain's iteration has five reductions, so areas fixed per reduction would give its last and
// the next iteration's first the same one.
template <int NV>
static __device__ __noinline__ bool res_sums(GridBar bar, double a, double b, double* parts, int gpb, int nvb, ResSh& sh) {
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  const int G = nvb * RES_VB, g0 = blockIdx.x * gpb;
  const int turn = sh.turn;
  double* const part = parts + turn * 2 * G;
  if (w < gpb) {
    double z;
    if (NV == 1) {
      z = a;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) z += __shfl_down_sync(0xffffffffu, z, o);
    } else {  // both trees at once: lanes 0..15 carry a's, lanes 16..31 b's
      const bool lo = lane < 16;
      z = (lo ? a : b) + __shfl_xor_sync(0xffffffffu, lo ? b : a, 16);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) z += __shfl_down_sync(0xffffffffu, z, o, 16);
    }
    if ((lane == 0 || (NV > 1 && lane == 16)) && g0 + w < G) part[(size_t)(lane >> 4) * G + g0 + w] = z;
  }
  __syncthreads();
  int bad = 0;
  if (t == 0) {
    sh.turn = turn ^ 1;
    bad = barrier_arrive_wait(bar.count, bar.error, SPIN_LIMIT) ? 0 : 1;
  }
  if (__syncthreads_or(bad)) return false;
  auto vb_sum = [&](int q, int vb) {  // a virtual block's eight group sums in sequence
    const double2* p = reinterpret_cast<const double2*>(part + (size_t)q * G + (size_t)vb * RES_VB);
    double2 u[RES_VB / 2];
#pragma unroll
    for (int k = 0; k < RES_VB / 2; ++k) u[k] = __ldcg(p + k);
    double z = plus_zero(u[0].x) + u[0].y;
#pragma unroll
    for (int k = 1; k < RES_VB / 2; ++k) {
      z += u[k].x;
      z += u[k].y;
    }
    return z;
  };
  const bool spread = nvb > 32;  // over all threads, else each summing lane does its own
  if (spread) {
    for (int e = t; e < NV * nvb; e += blockDim.x) sh.vb[e] = vb_sum(e / nvb, e % nvb);
    __syncthreads();
  }
  if (w < NV) {  // warp q: lane l adds virtual blocks l, l+32, ... in order, then the lanes' tree
    double z = 0.0;
    if (lane < nvb) z = plus_zero(spread ? sh.vb[w * nvb + lane] : vb_sum(w, lane));
#pragma unroll 1
    for (int e = lane + 32; e < nvb; e += 32) z += sh.vb[w * nvb + e];
    for (int o = 16; o > 0; o >>= 1)
      if (o < nvb) z += __shfl_down_sync(0xffffffffu, z, o);
    if (lane == 0) sh.v[w] = z;
  }
  if (NV > 1) __syncthreads();
  return true;
}

__device__ __forceinline__ bool res_sync(GridBar bar) {
  __syncthreads();
  int bad = 0;
  if (threadIdx.x == 0) bad = barrier_arrive_wait(bar.count, bar.error, SPIN_LIMIT) ? 0 : 1;
  return __syncthreads_or(bad) == 0;
}

// grid_reduce over the resident layout: post() runs on thread 0 with the sums in sh.v
template <int NV, class Post>
__device__ __forceinline__ bool res_reduce(GridBar bar, double a, double b, double* parts, int gpb, int nvb, ResSh& sh,
                                           Post post) {
  if (!res_sums<NV>(bar, a, b, parts, gpb, nvb, sh)) return false;
  if (threadIdx.x == 0) post();
  __syncthreads();
  return true;
}

}  // namespace vebi
