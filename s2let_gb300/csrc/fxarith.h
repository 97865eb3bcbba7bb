// Complex block fixed-point arithmetic on 64-bit integers (device code), used
// by the ring DFTs.
//
// A block of values shares one power-of-two scale; a complex value is a
// longlong2 (re, im).  GB300 issues an integer add on every FP32 lane and a
// 32 x 32 + 64 multiply-add (mad.wide.s32) at half that rate, against 1/64 for
// FP64 instructions (measured, SMSP cycles per warp instruction: add.u32 1.03,
// add.u64 2.07, mad.wide.s32 2.13, fma.f32 1.05, one FP64 FMA 64).  A complex
// addition is two 64-bit adds (against 16 FP32 instructions in double-float)
// and a complex product by a 62-bit constant 12 multiply-adds (32 in
// double-float), with an absolute rounding error of about one unit of the
// 64-bit word per operation.
//
// Constants (twiddles, chirps, kernel spectra) are w = (h 2^32 + l) 2^-62 with |w|
// <= 1 (the spectra: < 2) and a balanced low word |l| < 2^31, as int4 (re.h, re.l, im.h,
// im.l).  Data words are split the same way (h signed, l balanced), so all
// partial products are signed 32 x 32.  The product of the low words, below
// one unit of the result, is dropped.
//
// The same source compiles for the host, where the tests run it.
#pragma once

#include <cuda_runtime.h>

#include <cmath>

#include "dfconv.h"

namespace s2g {
namespace {

#ifdef __CUDACC__
#define S2G_DI __device__ __forceinline__
#else
#define S2G_DI inline
#endif

S2G_DI long long mad_wide(int a, int b, long long c) {
#ifdef __CUDACC__
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
#else
  return (long long)((unsigned long long)((long long)a * b) + (unsigned long long)c);
#endif
}
S2G_DI int clz32(int v) {  // 32 for 0
#ifdef __CUDACC__
  return __clz(v);
#else
  return v ? __builtin_clz((unsigned)v) : 32;
#endif
}
S2G_DI int clz64(long long v) {
#ifdef __CUDACC__
  return __clzll(v);
#else
  return v ? __builtin_clzll((unsigned long long)v) : 64;
#endif
}
// v = h 2^32 + l with l signed
S2G_DI void fx_words(long long v, int &h, int &l) {
  l = (int)v;
  h = (int)(v >> 32) + (int)((unsigned)l >> 31);
}
S2G_DI long long fx_high(long long c) { return (long long)(int)(c >> 32); }
constexpr long long kFxHalf = 0x80000000ll;  // rounds the high word of a cross-product sum

S2G_DI longlong2 fx_add(longlong2 a, longlong2 b) { return make_longlong2(a.x + b.x, a.y + b.y); }
S2G_DI longlong2 fx_sub(longlong2 a, longlong2 b) { return make_longlong2(a.x - b.x, a.y - b.y); }
S2G_DI longlong2 fx_mul_i(longlong2 a) { return make_longlong2(-a.y, a.x); }
S2G_DI longlong2 fx_conj(longlong2 a) { return make_longlong2(a.x, -a.y); }
S2G_DI longlong2 fx_shl(longlong2 a, int k) {
  return make_longlong2((long long)((unsigned long long)a.x << k), (long long)((unsigned long long)a.y << k));
}
S2G_DI longlong2 fx_sar(longlong2 a, int k) { return make_longlong2(a.x >> k, a.y >> k); }

// high products p and cross-product sums c of a w (CONJ: a conj(w)):
// a w = 4 (p + c 2^-32) up to the dropped low products.  |a| < 2^62.5 with |w| <= 1,
// or |a| < 2^61.5 with |w| < 2, keeps |c| below 2^63: by Cauchy's inequality over
// the pairs of words, 2^30.5 2^31.5 + 2^31.5 2^30 and 2^29.5 2^31.5 + 2^31.5 2^31.
template <bool CONJ>
S2G_DI void fx_products(longlong2 a, int4 w, long long half, long long &pr, long long &cr,
                                            long long &pi, long long &ci) {
  int xh, xl, yh, yl;
  fx_words(a.x, xh, xl);
  fx_words(a.y, yh, yl);
  const int nh = -w.z, nl = -w.w;
  const int rh = CONJ ? w.z : nh, rl = CONJ ? w.w : nl;  // re = x w.re + y r
  const int ih = CONJ ? nh : w.z, il = CONJ ? nl : w.w;  // im = y w.re + x i
  cr = mad_wide(xh, w.y, half);
  cr = mad_wide(xl, w.x, cr);
  cr = mad_wide(yh, rl, cr);
  cr = mad_wide(yl, rh, cr);
  pr = mad_wide(xh, w.x, 0);
  pr = mad_wide(yh, rh, pr);
  ci = mad_wide(yh, w.y, half);
  ci = mad_wide(yl, w.x, ci);
  ci = mad_wide(xh, il, ci);
  ci = mad_wide(xl, ih, ci);
  pi = mad_wide(yh, w.x, 0);
  pi = mad_wide(xh, ih, pi);
}
// a w 2^(N-2) and a conj(w) 2^(N-2), rounded
template <int N, bool CONJ>
S2G_DI longlong2 fx_product(longlong2 a, int4 w) {
  long long pr, cr, pi, ci;
  fx_products<CONJ>(a, w, kFxHalf >> N, pr, cr, pi, ci);
  if (N == 0) return make_longlong2(pr + fx_high(cr), pi + fx_high(ci));
  return make_longlong2((pr << N) + (cr >> (32 - N)), (pi << N) + (ci >> (32 - N)));
}
S2G_DI longlong2 fx_mul4(longlong2 a, int4 w) { return fx_product<0, false>(a, w); }  // a w / 4: one radix-4 stage
S2G_DI longlong2 fx_mulc4(longlong2 a, int4 w) { return fx_product<0, true>(a, w); }
S2G_DI longlong2 fx_mul2(longlong2 a, int4 w) { return fx_product<1, false>(a, w); }  // a w / 2
S2G_DI longlong2 fx_mulc2(longlong2 a, int4 w) { return fx_product<1, true>(a, w); }
S2G_DI longlong2 fx_mul(longlong2 a, int4 w) { return fx_product<2, false>(a, w); }  // a w
S2G_DI longlong2 fx_mulc(longlong2 a, int4 w) { return fx_product<2, true>(a, w); }
// s + v w / 4 for reals, w = (wh, wl)
S2G_DI long long fx_mac4(long long s, long long v, int wh, int wl) {
  int h, l;
  fx_words(v, h, l);
  const long long c = mad_wide(l, wh, mad_wide(h, wl, kFxHalf));
  return mad_wide(h, wh, s + fx_high(c));
}

// exponent e of a block whose largest FP64 exponent field is emax: |v| < 2^e
S2G_DI int fx_exp(int emax) { return (emax > 1 ? emax : 1) - 1022; }
constexpr int kExpNonFinite = 2047;  // exponent field of infinities and NaN

// v 2^(BITS - e) rounded towards zero, |v| < 2^e (subnormals included)
template <int BITS>
S2G_DI long long fx_split(double v, int e) {
  const unsigned long long u = bits_of(v);
  const int E = (int)((u >> 52) & 0x7FF);
  const unsigned long long M = (u & 0xFFFFFFFFFFFFFull) | (E ? 1ull << 52 : 0ull);
  const int r = e + 1022 - (E ? E : 1);  // >= 0
  const unsigned long long q = r < 64 ? (M << (BITS - 53)) >> r : 0ull;
  return (long long)u < 0 ? -(long long)q : (long long)q;
}
template <int BITS>
S2G_DI longlong2 fx_split2(double2 v, int e) {
  return make_longlong2(fx_split<BITS>(v.x, e), fx_split<BITS>(v.y, e));
}
// q 2^k as a double, rounded to nearest (integer work; ldexp only for results
// outside the normal range)
S2G_DI double fx_join(long long q, int k) {
  if (q == 0) return 0.0;
  const unsigned long long s = (unsigned long long)q & (1ull << 63);
  unsigned long long a = (unsigned long long)(q < 0 ? -q : q);
  const int n = clz64((long long)a);
  a <<= n;
  const int E = 1023 + 63 + k - n;  // biased exponent of the leading bit
  if (E <= 0 || E >= 2046) {
    const double d = ldexp((double)(a >> 11), 63 + k - n - 52);
    return s ? -d : d;
  }
  // the rounding carry runs into the exponent field
  const unsigned long long m = (a >> 11) + ((a >> 10) & 1);
  return double_of(s | ((((unsigned long long)(E - 1)) << 52) + m));
}
S2G_DI double2 fx_join2(longlong2 q, int k) { return make_double2(fx_join(q.x, k), fx_join(q.y, k)); }


// Floats to doubles and back in integers (rounded to nearest, ties to even); zeros,
// subnormals, infinities, NaN and results outside the normal range of a float go to
// the conversion instructions, out of line.
#ifdef __CUDACC__
__device__ __noinline__ double widen_any(float x) { return (double)x; }
__device__ __noinline__ float narrow_any(double x) { return __double2float_rn(x); }
#else
inline double widen_any(float x) { return (double)x; }
inline float narrow_any(double x) { return (float)x; }
#endif
S2G_DI double widen(float x) {
  const uint32_t b = bits_of(x);
  if (((b >> 23) & 0xFF) - 1u >= 254u) return widen_any(x);
  return double_of(((uint64_t)((b & 0x80000000u) | (((b & 0x7FFFFFFFu) >> 3) + (896u << 20))) << 32) | (b << 29));
}
S2G_DI float narrow(double x) {
  const uint32_t hi = (uint32_t)(bits_of(x) >> 32), lo = (uint32_t)bits_of(x);
  if (((hi >> 20) & 0x7FF) - 897u >= 254u) return narrow_any(x);
  uint32_t f = (((hi & 0x7FFFFFFFu) - (896u << 20)) << 3) | (lo >> 29);
  const uint32_t rem = lo & 0x1FFFFFFFu;
  f += rem > 0x10000000u || (rem == 0x10000000u && (f & 1)) ? 1u : 0u;  // the carry runs into the exponent
  return float_of((hi & 0x80000000u) | f);
}
}  // namespace
}  // namespace s2g
