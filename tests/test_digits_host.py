"""Host check of the integer conversions behind the digit slices and the fixed-point
rings (s2let_gb300/csrc/digits.h, fxarith.h): random and edge values, exactly or to
the rounding that each states."""
import os
import shutil
import subprocess

import pytest

from test_ringcore import CSRC, CUDA

HARNESS = r"""
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include "digits.h"
using namespace s2g;
typedef __int128 i128;
static int fails = 0;
#define CHECK(c, ...) do { if (!(c) && ++fails < 20) { std::printf("%s:%d %s ", "h", __LINE__, #c); std::printf(__VA_ARGS__); std::printf("\n"); } } while (0)
static std::mt19937_64 g(5);
static double any_double(int span) {  // normal, exponents within +-span
  const uint64_t m = g() >> 12, e = 1023 + (long)(g() % (2 * span + 1)) - span;
  return double_of((g() << 63) | (e << 52) | (g() % 5 ? m : (g() % 2 ? 0xFFFFFFFFFFFFFull : 0)));
}
template <int S> void bytes_of(long long q) {
  uint32_t lo, hi;
  digit_bytes<S>(q, lo, hi);
  i128 sum = 0;
  for (int j = 0; j < S; ++j) {
    const int y = S - 1 - j, b = (int)((y < 4 ? lo >> (8 * y) : hi >> (8 * (y - 4))) & 0xFF), d = b - 64;
    CHECK(d >= -64 && d <= (j == 0 ? 64 : 63), "q %lld digit %d %d", q, j, d);
    sum = sum * 128 + d;
  }
  CHECK(sum == q, "q %lld", q);
  if (S == 7) CHECK(hi >> 24 == 0, "q %lld", q);
  if (S == 7) {
    int d[7];
    int_digits(q, d);
    for (int j = 0; j < 7; ++j) {
      const int y = 6 - j, b = (int)((y < 4 ? lo >> (8 * y) : hi >> (8 * (y - 4))) & 0xFF);
      CHECK(b == d[j] + 64, "q %lld digit %d", q, j);
    }
  }
}
int main() {
  // digits: every q of 48 and 55 bits, the ends and runs of the extreme digits among them
  for (int S : {7, 8}) {
    const int bits = 7 * S - 1;
    std::vector<long long> qs = {0, 1, -1};
    for (long long d : {-64, 63, 64, -1}) {
      long long q = 0;
      for (int j = 0; j < S; ++j) {
        q = q * 128 + (j == 0 && d == 63 ? 63 : d);
        qs.push_back(q);
        qs.push_back(-q);
      }
    }
    for (int k = 0; k <= bits; ++k)
      for (long long o : {-1, 0, 1}) {
        qs.push_back((1ll << k) + o);
        qs.push_back(-(1ll << k) + o);
      }
    for (int i = 0; i < 300000; ++i) qs.push_back((long long)(g() % (2ull << bits)) - (1ll << bits));
    for (long long q : qs)
      if (q <= 1ll << bits && q >= -(1ll << bits)) S == 7 ? bytes_of<7>(q) : bytes_of<8>(q);
  }
  // fixed-point images of doubles, |v| < 2^e: rounded to nearest
  for (int i = 0; i < 500000; ++i) {
    const int span = i % 3 ? 40 : 300;
    const double v = i % 50 ? any_double(span) : 0.0;
    const int e = block_scale(exp_field(v)) + (i % 2 ? 0 : (int)(g() % 70));
    const long double s = ldexpl((long double)v, -e);
    const long long q7 = fixed48(v, e), q8 = fixed55(v, e);
    CHECK(fabsl(ldexpl(s, 48) - q7) <= 0.5L, "v %a e %d", v, e);
    CHECK(fabsl(ldexpl(s, 55) - q8) <= 0.5L, "v %a e %d", v, e);
    const int d = eighth_digit(v, e);
    CHECK(d >= -64 && d <= 64 && q7 * 128 + d == q8, "v %a e %d digit %d", v, e, d);
    const int f = fx_exp(exp_field(v)) + (i % 2 ? 0 : (int)(g() % 70));
    CHECK(fabsl(ldexpl((long double)v, 62 - f) - fx_split<62>(v, f)) < 1.0L, "v %a e %d", v, f);
    CHECK(fx_split<61>(-v, f) == -fx_split<61>(v, f), "v %a", v);
    CHECK(fx_join(fx_split<62>(v, fx_exp(exp_field(v))), fx_exp(exp_field(v)) - 62) == v, "v %a", v);
  }
  {  // subnormals
    const double t = double_of(12345);
    CHECK(fx_join(fx_split<62>(t, fx_exp(0)), fx_exp(0) - 62) == t, "subnormal");
    CHECK(fx_join(-(1ll << 62), 1100) == -INFINITY && fx_join(3, 2000) == INFINITY, "overflow");
    CHECK(fx_join(3, -1076) == double_of(1) || fx_join(3, -1076) == double_of(0), "3/4 of the least");
  }
  for (int i = 0; i < 500000; ++i) {  // fx_join rounds to nearest
    const long long q = (long long)g() >> (i % 40);
    const int k = (int)(g() % 200) - 100;
    const double d = fx_join(q, k);
    const long double x = ldexpl((long double)q, k), u = q ? ldexpl(1.0L, ilogb(d) - 52) : 0;
    CHECK(fabsl((long double)d - x) <= 0.5L * u, "q %lld k %d", q, k);
  }
  // products: off the correctly rounded one only within 2^-10 ulp of a tie
  for (int i = 0; i < 1000000; ++i) {
    const double x = any_double(i % 7 ? 100 : 500), y = any_double(i % 7 ? 100 : 500), z = mul_int(x, y), r = x * y;
    if (z == r) continue;
    const i128 m = (i128)((bits_of(x) & 0xFFFFFFFFFFFFFull) | 1ull << 52) * ((bits_of(y) & 0xFFFFFFFFFFFFFull) | 1ull << 52);
    const int sh = m >> 105 ? 53 : 52;
    const i128 frac = m & (((i128)1 << sh) - 1), half = (i128)1 << (sh - 1);
    const i128 off = frac > half ? frac - half : half - frac;
    CHECK(off <= (i128)1 << (sh - 10), "x %a y %a: %a %a", x, y, z, r);
    CHECK(llabs((long long)(bits_of(z) - bits_of(r))) == 1, "x %a y %a: %a %a", x, y, z, r);
  }
  const double edge[] = {0.0, -0.0, 1.0, -1.0, INFINITY, -INFINITY, NAN, 0x1p-1074, 0x1.fffffffffffffp-1023, 0x1p-1022,
                         0x1.fffffffffffffp1023, 0x1p-511, 0x1.fffffffffffffp-512, 0x1p512, 0x1.fffffffffffffp511, 3.0};
  for (double x : edge)
    for (double y : edge) {
      const double z = mul_int(x, y), r = x * y;
      CHECK(z == r ? std::signbit(z) == std::signbit(r) : std::isnan(z) && std::isnan(r), "%a %a: %a %a", x, y, z, r);
    }
  // the 71-bit sums
  for (int i = 0; i < 1000000; ++i) {
    long long hi = (long long)g() >> (20 + i % 44), lo = (long long)g() >> (17 + i % 47);
    if (i % 11 == 0) hi = i % 2 ? -1 : 0;
    if (i % 13 == 0) lo = -(hi << 28) + (long long)(g() % 9) - 4;  // cancelling
    if (i % 13 == 0 && (hi > 1 << 17 || hi < -(1 << 17))) continue;
    const i128 n = ((i128)hi << 28) + lo;
    const int k = (int)(g() % 400) - 200;
    const double d = join71(hi, lo, k);
    if (n == 0) {
      CHECK(d == 0, "%lld %lld", hi, lo);
      continue;
    }
    const long double s = ldexpl((long double)d, -k);  // 53 bits: exact as an integer times a power of two
    const i128 back = s == floorl(s) ? (i128)s : (i128)0;
    const long double u = ldexpl(1.0L, ilogbl(s) - 52);
    if (u >= 1.0L) {
      const i128 diff = back > n ? back - n : n - back;
      CHECK((long double)diff <= u * (0.5L + 0x1p-10L), "%lld %lld k %d", hi, lo, k);
    } else {
      CHECK((i128)s == n && s == floorl(s), "%lld %lld k %d", hi, lo, k);
    }
  }
  CHECK(join71(1ll << 40, 0, 1000) == INFINITY && join71(-(1ll << 40), 0, 1000) == -INFINITY, "overflow");
  CHECK(join71(1, 0, -1102) == double_of(1) && join71(0, 5, -1074) == double_of(5), "subnormal");
  // floats
  for (int i = 0; i < 2000000; ++i) {
    uint32_t b = (uint32_t)g();
    if (i % 4 == 0) b = (b & 0x807FFFFFu) | ((uint32_t[]){0, 1, 254, 255}[i / 4 % 4] << 23);
    if (i % 64 == 0) b &= 0xFF800000u;
    float x;
    std::memcpy(&x, &b, 4);
    const double w = widen(x), e = (double)x;
    CHECK(bits_of(w) == bits_of(e) || (std::isnan(w) && std::isnan(e)), "float %08x", b);
    uint64_t u = g();
    if (i % 2) u = (u & 0x800FFFFFFFFFFFFFull) | ((uint64_t)(890 + g() % 270) << 52);  // around the range of a float
    if (i % 3 == 0) u = (u & ~0x1FFFFFFFull) | (uint64_t[]){0, 1, 0x0FFFFFFF, 0x10000000, 0x10000001, 0x1FFFFFFF}[g() % 6];
    if (i % 5 == 0) u |= 0x000FFFFFE0000000ull;
    const float f = narrow(double_of(u)), r = (float)double_of(u);
    CHECK(bits_of(f) == bits_of(r) || (std::isnan(f) && std::isnan(r)), "double %016llx", (unsigned long long)u);
  }
  std::printf("%d failures\n", fails);
  return fails != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or CUDA is None, reason="needs g++ and the CUDA headers")
def test_integer_conversions(tmp_path):
    (tmp_path / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=gnu++17", "-ffp-contract=off", f"-I{CSRC}", f"-I{CUDA}", str(tmp_path / "h.cpp"),
                    "-o", str(tmp_path / "h")], check=True)
    out = subprocess.run([str(tmp_path / "h")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout[-3000:]
