// vebi_fp64.cuh -- binary64 products, quotients and square roots on the integer and FP32 pipes,
// rounded to nearest even bit for bit as the FP64 instructions round them.
//
// This GPU issues an FP64 instruction per 64-76 cycles and scheduler, whatever it is and however
// few lanes it has; a / b costs 8.8 of them and sqrt 10.8 (measured).  The same cycles hold 64-76
// integer or FP32 instructions, which the pair kernels leave unused.  So
//  * mul_int multiplies the 53-bit significands with four 32 x 32 -> 64 products and rounds
//    (IEEE 754's definition; ~40 instructions): beside the FP64 pipe, a kernel's products are free;
//  * quotient and root take two FP64 instructions, an approximation and its residual a - b q or
//    x - g^2 by fused multiply-add (Markstein, "IA-64 and Elementary Functions", 2000).  The
//    residual says how many units in the last place the result is off, to a fraction of a unit, so the
//    nearest number is found by an integer addition -- or, next to a rounding boundary (2e-4 of
//    the results), for zeros, subnormals, infinities, NaN and next to powers of two, by the
//    operation itself in a call.  (A call: inlined, the compiler computes it ahead of the test.)
//  * the approximations are 1/b and 1/sqrt(x) in two FP32 parts, Newton's iteration from the FP32
//    approximation instructions.
// Everything but those two instructions compiles for the host too, where a test compares the
// results with the processor's.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define VF_FN __device__ __forceinline__
#define VF_CALL static __device__ __noinline__
#else
#include <cmath>
#include <cstring>
#define VF_FN static inline
#define VF_CALL static __attribute__((noinline))
#endif

namespace vebi {
namespace fp {

#ifdef __CUDACC__
VF_FN int hi(double x) { return __double2hiint(x); }
VF_FN uint32_t lo(double x) { return (uint32_t)__double2loint(x); }
VF_FN double pack(int h, uint32_t l) { return __hiloint2double(h, (int)l); }
VF_FN float bits_f(uint32_t u) { return __uint_as_float(u); }
VF_FN uint32_t f_bits(float f) { return __float_as_uint(f); }
VF_FN uint32_t funnel(uint32_t l, uint32_t h, uint32_t s) { return __funnelshift_l(l, h, s); }
VF_FN float rcp_start(float m) { return __fdividef(1.0f, m); }
VF_FN float rsqrt_start(float m) { return rsqrtf(m); }
VF_FN int to_int(float f) { return __float2int_rn(f); }
#else
VF_FN int hi(double x) { uint64_t b; std::memcpy(&b, &x, 8); return (int)(b >> 32); }
VF_FN uint32_t lo(double x) { uint64_t b; std::memcpy(&b, &x, 8); return (uint32_t)b; }
VF_FN double pack(int h, uint32_t l) { uint64_t b = (uint64_t)(uint32_t)h << 32 | l; double x; std::memcpy(&x, &b, 8); return x; }
VF_FN float bits_f(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
VF_FN uint32_t f_bits(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
VF_FN uint32_t funnel(uint32_t l, uint32_t h, uint32_t s) { return (uint32_t)((((uint64_t)h << 32 | l) << s) >> 32); }
VF_FN float rcp_start(float m);    // the test's: 1/m and 1/sqrt(m) to within a few units
VF_FN float rsqrt_start(float m);
VF_FN int to_int(float f) { return (int)std::lrintf(f); }
using std::fma;
using std::sqrt;
#endif

VF_FN bool is_zero(double v) { return ((uint32_t)hi(v) << 1 | lo(v)) == 0u; }
VF_FN int exponent(int h) { return (h >> 20) & 0x7ff; }
// top 24 bits of the significand as a float in [1, 2)
VF_FN float significand(int h, uint32_t l) { return bits_f(0x3f800000u | ((uint32_t)h & 0xfffffu) << 3 | l >> 29); }

VF_CALL double multiplied(double a, double b) { return a * b; }
VF_CALL double divided(double a, double b) { return a / b; }
VF_CALL double rooted(double x) { return sqrt(x); }

// a * b
VF_FN double mul_int(double a, double b) {
  const int ha = hi(a), hb = hi(b);
  const uint32_t la = lo(a), lb = lo(b);
  const uint32_t ma = ((uint32_t)ha & 0xfffffu) | 0x100000u, mb = ((uint32_t)hb & 0xfffffu) | 0x100000u;
  const int ea = exponent(ha), eb = exponent(hb);
  // the 106-bit product as top (42 bits), t, and the low word
  const uint64_t low = (uint64_t)la * lb;
  uint64_t mid = (uint64_t)ma * lb + (low >> 32);
  mid += (uint64_t)la * mb;
  const uint64_t top = (uint64_t)ma * mb + (mid >> 32);
  const uint32_t t = (uint32_t)mid, tl = (uint32_t)top, th = (uint32_t)(top >> 32);
  const uint32_t sh = (th & 0x200u) ? 11u : 12u;  // leading bit 105 or 104
  const uint32_t mh = funnel(tl, th, sh), ml = funnel(t, tl, sh);
  const uint32_t rest = t << sh | ((uint32_t)low != 0u ? 1u : 0u);  // below the last place, with a sticky bit
  const uint32_t up = (rest | (ml & 1u)) > 0x80000000u ? 1u : 0u;
  const int e = ea + eb - 1011 - (int)sh;
  const uint32_t sign = (uint32_t)(ha ^ hb) & 0x80000000u;
  const uint64_t m = ((uint64_t)mh << 32 | ml) + up;  // a carry past the significand raises the exponent
  if ((uint32_t)(ea - 1) < 2046u && (uint32_t)(eb - 1) < 2046u && (uint32_t)(e - 1) < 2045u)
    return pack((int)(((uint32_t)(m >> 32) + ((uint32_t)(e - 1) << 20)) | sign), (uint32_t)m);
  if (ea < 2047 && eb < 2047 && (is_zero(a) || is_zero(b))) return pack((int)sign, 0u);
  return multiplied(a, b);
}

// y0 + y1 with y0 in [0.5, 1], |y1| < 2^-20, times 2^-e: 45 bits or so, the exponent field unchecked
VF_FN double joined(float y0, float y1, int e) {
  const uint32_t u = f_bits(y0);
  const uint64_t b = ((uint64_t)((u >> 3) + (896u << 20)) << 32 | (uint64_t)(u << 29)) +
                     (uint64_t)((int64_t)to_int(y1 * 70368744177664.0f) * 128);  // y1 2^46, units of 2^-53
  return pack((int)((uint32_t)(b >> 32) - ((uint32_t)e << 20)), (uint32_t)b);
}
// lower part of the significand: what significand() leaves out, 23 bits of it
VF_FN float significand_low(uint32_t l) {
  return (bits_f(0x3f800000u | (l & 0x1fffffffu) >> 6) - 1.0f) * 1.1920928955078125e-7f;
}

// 1 / b to some 45 bits (b > 0)
VF_FN double reciprocal(double b) {
  const int h = hi(b);
  const uint32_t l = lo(b);
  const float mh = significand(h, l), ml = significand_low(l);
  const float y0 = rcp_start(mh);
  float e = fmaf(-mh, y0, 1.0f);
  e = fmaf(-ml, y0, e);
  return joined(y0, fmaf(e, e, e) * y0, exponent(h) - 1023);
}
// 1 / sqrt(x) to some 45 bits (x > 0)
VF_FN double reciprocal_root(double x) {
  const int h = hi(x);
  const uint32_t l = lo(x);
  const int ex = exponent(h) - 1023, odd = ex & 1;
  const float s = odd ? 2.0f : 1.0f;
  const float mh = significand(h, l) * s, ml = significand_low(l) * s;
  const float y0 = rsqrt_start(mh);
  const float p = y0 * y0, pl = fmaf(y0, y0, -p);
  float e = fmaf(-mh, p, 1.0f);
  e = fmaf(-mh, pl, e);
  e = fmaf(-ml, p, e);
  return joined(y0, y0 * e * fmaf(0.375f, e, 0.5f), (ex - odd) >> 1);
}

// q moved by the residual r: q + r y 2^-halve is the exact result.  Its distance from q in units of
// q's last place, below 2^(s+2), is found to a part in 2^21; false when the nearest number is not
// certain (s > 9, next to a boundary between two numbers, or q's neighbours differ in exponent).
VF_FN bool settle(double& q, double r, double y, int halve) {
  const int hq = hi(q), hr = hi(r), hy = hi(y);
  const int er = exponent(hr);
  if (er == 0) return is_zero(r) && exponent(hq) > 0;
  const int s = er + exponent(hy) - exponent(hq) - 971 - halve;
  const int sc = s < -30 ? -30 : s;
  const float f = significand(hr, lo(r)) * significand(hy, lo(y)) * bits_f((uint32_t)(sc + 127) << 23);
  const float g = f + 12582912.0f;  // f rounded to an integer, in the low bits
  const int k = (int)(f_bits(g) - 0x4b400000u);
  const float off = f - (g - 12582912.0f);
  const bool sure = s <= 9 && fabsf(off) < 0.5f - bits_f((uint32_t)(sc + 108) << 23) &&
                    ((uint32_t)hq & 0xfffffu) - 1u < 0xffffeu && (uint32_t)(exponent(hq) - 1) < 2045u;
  const int64_t d = (hq ^ hr ^ hy) < 0 ? -(int64_t)k : (int64_t)k;
  const uint64_t b = ((uint64_t)(uint32_t)hq << 32 | lo(q)) + (uint64_t)d;
  q = pack((int)(b >> 32), (uint32_t)b);
  return sure;
}

// the residual of a number this large does not reach down to the subnormals
VF_FN bool exact_residual(double a) { return exponent(hi(a)) > 110; }
// a / b from q near it and y near 1 / b
VF_FN double quotient_near(double a, double b, double y, double q) {
  return settle(q, fma(-b, q, a), y, 0) && exact_residual(a) ? q : divided(a, b);
}
VF_FN double magnitude(double x) { return pack(hi(x) & 0x7fffffff, lo(x)); }
// a / b for any b, from y = 1 / |b| to some 45 bits
VF_FN double quotient(double a, double b, double y) {
  if (is_zero(a)) return divided(a, b);
  const double ys = pack((int)((uint32_t)hi(y) | ((uint32_t)hi(b) & 0x80000000u)), lo(y));
  return quotient_near(a, b, ys, a * ys);
}
// a / b; where 1 / b is not a normal number (as of 0, NaN or an infinity), as divided
VF_FN double quotient(double a, double b) {
  return (uint32_t)(exponent(hi(b)) - 1) < 2044u ? quotient(a, b, reciprocal(magnitude(b))) : divided(a, b);
}
// sqrt(x); y = reciprocal_root(x)
VF_FN double root(double x, double& y) {
  y = reciprocal_root(x);
  double g = x * y;
  return settle(g, fma(-g, g, x), y, 1) && exact_residual(x) ? g : rooted(x);
}

}  // namespace fp
}  // namespace vebi
