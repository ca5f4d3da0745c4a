// vebi_lanes.cuh -- pair sums of a row by one thread or by eight lanes, in the same order.
//
// A thread per row leaves most of the GPU idle on a small domain: 20k rows are 664 warps on 608
// schedulers, and each walks its 44 pairs through two dependent trips to memory a pair.  With eight
// lanes a row, a lane loads and evaluates every eighth pair, so eight pairs' trips are in flight; the
// terms are then added in pair order, so the sums are the same bit for bit.
#pragma once
#include "vebi_ctx.cuh"

namespace vebi {

constexpr int LANES = 8;       // lanes a row
constexpr int LANES_TPB = 64;  // threads a block: small blocks spread a small domain over the SMs
// Rows up to which eight lanes take a row: one line for all kernels, between 20k, where every
// one gains, and 60k, where the heaviest (the FP64 predictor) loses.  Measured, us, a thread / eight lanes
// a row, with 1.7k, 20k and 60k rows: FP64 predictor 154 / 33, 176 / 86, 207 / 227; FP64 gradients
// 76 / 25, 84 / 47, 108 / 98; FP32 weights (20k, 60k) 48 / 16, 46 / 33; shifting 41 / 21, 41 / 43;
// predictor 72 / 37, 84 / 76: lines of their own would win the FP64 gradients and the FP32 weights and
// predictor some 10 us each about 60k rows.
// The pressure gradient, whose pairs are cheap, has its own, measured on the FP64 kernel: 34 / 18 at 1.7k,
// 31 / 29 at 10k, 53 / 63 at 20k.  The FP32 one takes the same line; it is not measured by eight lanes.
constexpr int LANE_ROWS = 30000;
constexpr int LANE_ROWS_PGRAD = 10000;

// this thread's row (a valid one also past the end), and whether it is one
template <int P>
__device__ __forceinline__ int lane_row(int n, bool& in) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) / P;
  in = i < n;
  return in ? i : n - 1;
}

// FP32: add(load(k)) for the pairs k = 0 .. cnt-1 in order, in every lane of the row.  load's result
// is a struct of floats.
template <int P, int U = 1, class Load, class Add>
__device__ __forceinline__ void pair_sums32(int cnt, Load load, Add add) {
  if constexpr (P == 1) {
#pragma unroll U
    for (int k = 0; k < cnt; ++k) add(load(k));
  } else {
    using T = decltype(load(0));
    constexpr int W = sizeof(T) / sizeof(float);
    const int q = threadIdx.x & (P - 1);
    const int most = __reduce_max_sync(0xffffffffu, cnt);
    for (int k0 = 0; k0 < most; k0 += P) {
      union {
        T t;
        float f[W];
      } v, w;
      for (int e = 0; e < W; ++e) v.f[e] = 0.f;
      if (k0 + q < cnt) v.t = load(k0 + q);
#pragma unroll
      for (int u = 0; u < P; ++u) {
#pragma unroll
        for (int e = 0; e < W; ++e) w.f[e] = __shfl_sync(0xffffffffu, v.f[e], u, P);
        if (k0 + u < cnt) add(w.t);
      }
    }
  }
}

// FP64: S sums of the pairs' terms in order, each of D terms a pair: load(k, t) gives t[S * D], sum s
// adds t[s * D], t[s * D + 1].  Lane s adds sum s (an FP64 add takes as long for one lane as for 32);
// the sums come back in every lane.
template <int S, int D, class Load>
__device__ __forceinline__ void pair_sums64(int cnt, Load load, double (&out)[S]) {
  static_assert(S <= LANES, "a lane a sum");
  __shared__ double sh[LANES_TPB / LANES][S * D][LANES + 1];
  const int q = threadIdx.x & (LANES - 1), r = threadIdx.x / LANES;
  const int most = __reduce_max_sync(0xffffffffu, cnt);
  double acc = 0.0;
  for (int k0 = 0; k0 < most; k0 += LANES) {
    if (k0 + q < cnt) {
      double t[S * D];
      load(k0 + q, t);
#pragma unroll
      for (int e = 0; e < S * D; ++e) sh[r][e][q] = t[e];
    }
    __syncwarp();
    if (q < S)
#pragma unroll
      for (int u = 0; u < LANES; ++u) {
        if (k0 + u >= cnt) break;
#pragma unroll
        for (int e = 0; e < D; ++e) acc += sh[r][q * D + e][u];
      }
    __syncwarp();
  }
#pragma unroll
  for (int s = 0; s < S; ++s) out[s] = __shfl_sync(0xffffffffu, acc, s, LANES);
}

// launch kern<LANES> up to `line` rows, else kern<1>, over the rows
#define LAUNCH_ROWS(x, kern, line)                                                                            \
  do {                                                                                                        \
    if ((x).c.npfb <= (line))                                                                                 \
      VEBI_LAUNCH(x, kern<LANES>, grid_for((long long)LANES * (x).c.npfb, LANES_TPB), LANES_TPB, (x).c, (x).d); \
    else                                                                                                      \
      VEBI_LAUNCH(x, kern<1>, grid_for((x).c.npfb), TPB, (x).c, (x).d);                                       \
  } while (0)

}  // namespace vebi
