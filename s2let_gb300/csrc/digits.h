// Integer conversions of the digit slices (mixed.h has the number format; mixed.cu
// uses them on the device, the tests on the host).
#pragma once

#include <cmath>

#include "fxarith.h"

namespace s2g {
namespace {

constexpr int kS = 7;     // digit slices per operand (split precision)
constexpr int kSmax = 8;  // and of the 64-bit form (FP64 results)

#ifdef __CUDACC__
#define S2G_UNROLL _Pragma("unroll")
#else
#define S2G_UNROLL
#endif

S2G_DI uint64_t mul_high(uint64_t a, uint64_t b) {
#ifdef __CUDACC__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// Balanced digits of q = round(v 2^(48-e)), |v| < 2^e: q = sum_j d_j 2^(42-7j)
// with d_1..d_6 in [-64, 63] (base-128 digits taken from the low end) and
// d_0 in [-64, 64].  Integer arithmetic only, so the split costs no FP64 work.
S2G_DI void int_digits(long long q, int *d) {
S2G_UNROLL
  for (int j = kS - 1; j >= 1; --j) {
    int r = (int)(q & 127);
    if (r >= 64) r -= 128;
    d[j] = r;
    q = (q - r) >> 7;
  }
  d[0] = (int)q;
}
// round(v 2^(48-e)) for |v| < 2^e, from the significand bits (no FP64 work)
S2G_DI long long fixed48(double v, int e) {
  const uint64_t u = bits_of(v);
  const int E = (int)((u >> 52) & 0x7FF);
  if (E == 0) return 0;
  const long long M = (long long)((u & 0xFFFFFFFFFFFFFull) | (1ull << 52));
  const int sh = E - 1075 + 48 - e;  // v 2^(48-e) = M 2^sh
  long long q;
  if (sh >= 0)
    q = M << sh;  // |v| < 2^e keeps this below 2^48
  else if (sh > -64)
    q = (M + (1ll << (-sh - 1))) >> (-sh);
  else
    q = 0;
  return (u >> 63) ? -q : q;
}

// round(v 2^(55-e)) for |v| < 2^e (subnormals included)
S2G_DI long long fixed55(double v, int e) {
  const uint64_t u = bits_of(v);
  const int E = (int)((u >> 52) & 0x7FF);
  const long long M = (long long)((u & 0xFFFFFFFFFFFFFull) | (E ? 1ull << 52 : 0ull));
  const int sh = (E ? E : 1) - 1075 + 55 - e;  // v 2^(55-e) = M 2^sh, sh <= 2
  long long q;
  if (sh >= 0)
    q = M << sh;
  else if (sh > -64)
    q = (M + (1ll << (-sh - 1))) >> (-sh);
  else
    q = 0;
  return (u >> 63) ? -q : q;
}
// The eighth digit of a table value: what the seven leave of v 2^-e, in units
// of 2^-55 (|digit| <= 64; with it the value is represented to 2^-56).
S2G_DI int eighth_digit(double v, int e) { return (int)(fixed55(v, e) - fixed48(v, e) * 128); }
// Balanced base-128 digits d_0 .. d_(S-1) of q, |q| <= 2^(7S-1), plus 64, one
// per byte: digit S-1-b in byte b of lo for b < 4, digit S-5-b in byte b of hi.
// Adding 64 in every digit position makes the balanced digits the 7-bit fields
// of the sum (the first is 8 bits wide: d_0 + 64 may be 128); each word's
// fields move apart by a step of 14 bits to 16 and one of 7 to 8.
template <int S>
S2G_DI void digit_bytes(long long q, uint32_t &lo, uint32_t &hi) {
  constexpr long long kBias = S == kS ? 0x0001020408102040ll : 0x0081020408102040ll;
  const unsigned long long u = (unsigned long long)(q + kBias);
  const auto bytes = [](uint32_t x, uint32_t sel, uint32_t mask) {
    const uint32_t t = (x & 0x3FFFu) | ((x << 2) & ~0x3FFFu);
    return ((t & sel) | ((t << 1) & ~sel)) & mask;
  };
  lo = bytes((uint32_t)u & 0xFFFFFFFu, 0x007F007Fu, 0x7F7F7F7Fu);
  hi = S == kS ? bytes((uint32_t)(u >> 28), 0x00FF007Fu, 0x00FF7F7Fu)
               : bytes((uint32_t)(u >> 28), 0x007F007Fu, 0xFF7F7F7Fu);
}

// v, negated when n is odd
S2G_DI double flip_sign(double v, int n) { return double_of(bits_of(v) ^ ((uint64_t)n << 63)); }
// FP64 paths that are rarely taken stay out of line: inlined, they were executed
// speculatively and kept the FP64 unit busy (k_slice_x from coefficients 189 us
// instead of 137 at L = 512, 32 maps).
#ifdef __CUDACC__
__device__ __noinline__ double mul_fp64(double x, double y) { return __dmul_rn(x, y); }
#else
inline double mul_fp64(double x, double y) { return x * y; }
#endif
// x y rounded to nearest, by a 64 x 64-bit integer product (the 64 bits below the
// kept high half only move results within 2^-11 units in the last place of a
// rounding boundary); zeros, subnormals, infinities, NaN and results near the
// ends of the range go to the FP64 unit.
S2G_DI double mul_int(double x, double y) {
  const uint64_t ux = bits_of(x), uy = bits_of(y);
  const int ex = (int)(ux >> 52) & 0x7FF, ey = (int)(uy >> 52) & 0x7FF, e = ex + ey - 1023;
  if ((unsigned)(ex - 1) >= 2046u || (unsigned)(ey - 1) >= 2046u || (unsigned)(e - 1) >= 2044u) return mul_fp64(x, y);
  // significands with the leading bit at the top: product in [2^62, 2^64)
  uint64_t p = mul_high((ux << 11) | (1ull << 63), (uy << 11) | (1ull << 63));
  const int n = p >> 63 ? 0 : 1;
  p <<= n;
  // the leading bit and a rounding carry run into the exponent field
  return double_of(((ux ^ uy) & (1ull << 63)) | (((uint64_t)(e - n) << 52) + (p >> 11) + ((p >> 10) & 1)));
}

// (hi 2^28 + lo) 2^k of two 64-bit words as a double, rounded once, in integers
S2G_DI double join71(long long hi, long long lo, int k) {
  hi += lo >> 28;
  uint32_t l = (uint32_t)lo & 0xFFFFFFFu;
  const unsigned long long s = (unsigned long long)hi & (1ull << 63);
  if (s) {  // magnitude of hi 2^28 + l
    hi = -hi - (l != 0);
    l = (0u - l) & 0xFFFFFFFu;
  }
  unsigned long long a = (unsigned long long)hi;
  int n, top;  // a normalised by n, exponent of its leading bit
  if (a >> 28) {
    n = clz64((long long)a);
    top = 63 - n + 28;
    a = (a << n) | (n >= 28 ? (unsigned long long)l << (n - 28) : (unsigned long long)(l >> (28 - n)));
  } else {
    a = (a << 28) | l;
    if (a == 0) return 0.0;
    n = clz64((long long)a);
    top = 63 - n;
    a <<= n;
  }
  const int E = 1023 + top + k;
  if (E <= 0 || E >= 2046) {
    const double d = ldexp((double)(a >> 11), top + k - 52);
    return s ? -d : d;
  }
  return double_of(s | ((((unsigned long long)(E - 1)) << 52) + (a >> 11) + ((a >> 10) & 1)));
}
}  // namespace
}  // namespace s2g
