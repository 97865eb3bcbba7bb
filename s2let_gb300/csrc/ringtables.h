// The constants of a ring length's Bluestein transform (RingFFT, plan.h), in
// extended precision on the host.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdint>
#include <vector>

namespace s2g {

// re + i im (magnitude below 2) as (re.h, re.l, im.h, im.l), v = (h 2^32 + l) 2^-62, |l| < 2^31
inline int4 fixed62(long double re, long double im) {
  const auto words = [](long double v, int &h, int &l) {
    long long q = llroundl(ldexpl(v, 62));
    l = (int)(unsigned)(unsigned long long)q;
    if (l == INT32_MIN) l = (int)(unsigned)(unsigned long long)++q;  // |l| < 2^31
    h = (int)((q - l) >> 32);
  };
  int4 o;
  words(re, o.x, o.y);
  words(im, o.z, o.w);
  return o;
}

struct RingTables {
  int P = 8, logP = 3, eb = 0;
  std::vector<int4> chirp, bhat, tw;
};

// host FFT (radix-2, in extended precision) for the Bluestein kernel spectrum;
// w holds exp(-2 pi i k / n) for k < n/2
using cxl = std::complex<long double>;
inline cxl cxl_mul(cxl a, cxl b) {  // std::complex's product checks for NaN
  return {a.real() * b.real() - a.imag() * b.imag(), a.real() * b.imag() + a.imag() * b.real()};
}
inline void host_fft(std::vector<cxl> &x, const std::vector<cxl> &w) {
  const size_t n = x.size();
  for (size_t i = 1, j = 0; i < n; ++i) {
    size_t bit = n >> 1;
    for (; j & bit; bit >>= 1) j ^= bit;
    j ^= bit;
    if (i < j) std::swap(x[i], x[j]);
  }
  for (size_t len = 2; len <= n; len <<= 1)
    for (size_t i = 0; i < n; i += len)
      for (size_t k = 0; k < len / 2; ++k) {
        const cxl u = x[i + k], v = cxl_mul(x[i + k + len / 2], w[k * (n / len)]);
        x[i + k] = u + v;
        x[i + k + len / 2] = u - v;
      }
}

inline RingTables ring_tables(int K) {
  RingTables r;
  while (r.P < 2 * K - 1) {
    r.P <<= 1;
    ++r.logP;
  }
  const int P = r.P, logP = r.logP;
  const long double pi = 3.141592653589793238462643383279502884197L;
  std::vector<cxl> chirp(K), b(P, cxl(0.0L)), tw(3 * P / 4);
  for (long k = 0; k < K; ++k) {
    const long double x = pi * (long double)((k * k) % (2L * K)) / (long double)K;
    chirp[k] = {cosl(x), sinl(x)};
  }
  for (int k = 0; k < 3 * P / 4; ++k) {
    if (k >= P / 4) {  // w^k = -i w^(k - P/4)
      tw[k] = {tw[k - P / 4].imag(), -tw[k - P / 4].real()};
    } else {
      const long double x = 2.0L * pi * (long double)k / (long double)P;
      tw[k] = {cosl(x), -sinl(x)};
    }
  }
  b[0] = chirp[0];
  for (int k = 1; k < K; ++k) b[k] = b[P - k] = chirp[k];
  host_fft(b, tw);
  long double top = 0.0L;
  for (const cxl &v : b) top = std::max(top, std::abs(v));
  // at most 2 (1 - 2^-30) in magnitude: the factor 1/4 of the product with it then
  // costs one bit and not two, and the high words still fit
  r.eb = 0;
  while (ldexpl(2.0L - ldexpl(1.0L, -29), r.eb) < top) ++r.eb;
  const auto fixed = [](const std::vector<cxl> &v, int e) {
    std::vector<int4> o(v.size());
    for (size_t i = 0; i < v.size(); ++i) o[i] = fixed62(ldexpl(v[i].real(), -e), ldexpl(v[i].imag(), -e));
    return o;
  };
  // per level h of the radix-4 passes (P/4, P/16, ...): w^j, w^2j, w^3j for j = k P / (4h), k < h
  const int h0 = logP & 1 ? 2 : 4;
  std::vector<cxl> levels(P - h0);
  for (int h = h0; h <= P / 4; h *= 4)
    for (int c = 0; c < 3; ++c)
      for (int k = 0; k < h; ++k) levels[h - h0 + c * h + k] = tw[(c + 1) * (k * (P / (4 * h)))];
  r.chirp = fixed(chirp, 0);
  r.bhat = fixed(b, r.eb);
  r.tw = fixed(levels, 0);
  return r;
}

}  // namespace s2g
