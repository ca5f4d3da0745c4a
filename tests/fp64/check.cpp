// vebi_fp64.cuh on the host: products, quotients and roots against the processor's, bit for bit,
// over seeded operands of every class -- random significands near one and over the whole range of
// exponents, short and nearly full significands, powers of two, zeros, subnormals, infinities and
// NaN -- with the FP32 starts off by up to two units as the GPU's approximations may be.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "vebi_fp64.cuh"

static uint64_t state = 0x2545f4914f6cdd1dull;
static uint64_t next() {  // SplitMix64
  uint64_t z = (state += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

namespace vebi {
namespace fp {
static inline float off(float y) { return y < 1.0f && y > 0.5001f ? bits_f(f_bits(y) + (uint32_t)((int)(next() % 5) - 2)) : y; }
static inline float rcp_start(float m) { return off(1.0f / m); }
static inline float rsqrt_start(float m) { return off(1.0f / std::sqrt(m)); }
}  // namespace fp
}  // namespace vebi
using namespace vebi::fp;

static double operand(int mode) {
  const uint64_t e = mode == 0 ? 993 + next() % 60 : mode == 1 ? next() % 2048 : mode == 2 ? 1023 : 823 + next() % 400;
  uint64_t b = (next() & 0x800fffffffffffffull) | e << 52;
  switch (next() % 16) {
    case 0: b &= 0xfffffffffffff000ull; break;
    case 1: b &= ~0xffffffffffffull; break;
    case 2: b |= 0xffffffffff000ull; break;
    case 3: b &= 0xfff0000000000000ull; break;
    case 4: b &= 0xfffffffff8000000ull; break;
    case 5: b |= 0xfffffffffffffull; break;
    default: break;
  }
  double x;
  std::memcpy(&x, &b, 8);
  return x;
}
static bool same(double a, double b) {
  uint64_t x, y;
  std::memcpy(&x, &a, 8);
  std::memcpy(&y, &b, 8);
  return (a != a && b != b) || x == y;
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 4000000;
  long bad = 0, unsure = 0, plain = 0;
  for (long i = 0; i < n; ++i) {
    double a = operand(i & 3), b = operand(i & 3);
    if (i % 97 == 0) a = i % 2 ? 0.0 : -0.0;
    if (i % 101 == 0) b = 0.0;
    const double p = std::fabs(b);
    bad += !same(mul_int(a, b), a * b);
    if (!is_zero(a)) {  // callers keep a zero numerator as it is
      const double y = reciprocal(p);
      bad += !same(quotient_near(a, p, y, a * y), a / p);
    }
    double y;
    bad += !same(root(p, y), std::sqrt(p));
    if ((i & 3) == 2) {  // the share of random operands that take the operation itself
      const uint64_t m = (next() & 0xfffffffffffffull) | 0x3ff0000000000000ull;
      double u;
      std::memcpy(&u, &m, 8);
      double q = a * reciprocal(u);
      const double r = std::fma(-u, q, a);
      ++plain;
      if (((hi(a) & 0xfffff) | lo(a)) && !is_zero(a)) unsure += !settle(q, r, reciprocal(u), 0);
    }
  }
  std::printf("%ld operands: %ld wrong; %.2g of %ld quotients unsettled\n", n, bad, (double)unsure / plain, plain);
  return bad != 0 || unsure > plain / 500;
}
