// vebi_fp64.cuh on the GPU, with the GPU's own FP32 starts: products, quotients and roots against the FP64
// instructions, bit for bit, over seeded operands of every class (as check.cpp draws them).
// Prints the operands tried and the wrong ones; exits 0 when there are none.
#include <cstdio>
#include <cstdlib>

#include "vebi_fp64.cuh"

using namespace vebi::fp;

__device__ uint64_t mix(uint64_t z) {  // SplitMix64
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
__device__ double operand(uint64_t seed, int mode) {
  const uint64_t r = mix(seed), s = mix(r), e = mode == 0 ? 993 + s % 60 : mode == 1 ? s % 2048 : mode == 2 ? 1023 : 823 + s % 400;
  uint64_t b = (r & 0x800fffffffffffffull) | e << 52;
  switch ((s >> 32) % 16) {
    case 0: b &= 0xfffffffffffff000ull; break;
    case 1: b &= ~0xffffffffffffull; break;
    case 2: b |= 0xffffffffff000ull; break;
    case 3: b &= 0xfff0000000000000ull; break;
    case 4: b &= 0xfffffffff8000000ull; break;
    case 5: b |= 0xfffffffffffffull; break;
    default: break;
  }
  return __longlong_as_double((long long)b);
}
__device__ bool same(double a, double b) {
  return (a != a && b != b) || __double_as_longlong(a) == __double_as_longlong(b);
}

__global__ void check(long long n, unsigned long long* bad) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    double a = operand(2 * t, t & 3), b = operand(2 * t + 1, t & 3), y;
    if (t % 97 == 0) a = t % 2 ? 0.0 : -0.0;
    if (t % 101 == 0) b = 0.0;
    const double p = magnitude(b);
    if (!same(mul_int(a, b), a * b)) atomicAdd(bad, 1ull);
    if (!same(quotient(a, b), a / b)) atomicAdd(bad + 1, 1ull);
    if (!same(quotient(a, b, reciprocal(p)), a / b)) atomicAdd(bad + 1, 1ull);
    if (!same(root(p, y), sqrt(p))) atomicAdd(bad + 2, 1ull);
    // 1 / sqrt(x) as the pair kernels use it: the root's y as a start for a quotient by the root
    const double r = root(p, y), q = a * y;
    if (!is_zero(a) && !same(quotient_near(a, r, y, q), a / r)) atomicAdd(bad + 1, 1ull);
  }
}

int main(int argc, char** argv) {
  const long long n = argc > 1 ? atoll(argv[1]) : 1ll << 26;
  unsigned long long *d = nullptr, h[3] = {1, 1, 1};
  cudaError_t e = cudaMalloc(&d, sizeof(h));
  if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof(h));
  if (e == cudaSuccess) {
    check<<<1216, 256>>>(n, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    std::printf("%s\n", cudaGetErrorString(e));
    return 2;
  }
  std::printf("%lld operands: %llu products, %llu quotients, %llu roots wrong\n", n, h[0], h[1], h[2]);
  return h[0] + h[1] + h[2] != 0;
}
