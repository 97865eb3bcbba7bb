// Bluestein core of the ring DFTs: the padded transforms of one ring's buffer in
// 64-bit block fixed point (fxarith.h), written for the threads of one block, or
// (the tests) for one thread of the host.
//
// Scaling.  Forward and inverse transform are radix-4 with a factor 1/4 per pass,
// which never raises the largest magnitude, so nothing overflows whatever the
// data.  It lowers a noise-like block by one bit a pass and a spike by two, while a
// rounding error stays about one unit: a few passes in a row would cost an FP64
// transform's accuracy.  So at a few places (bluestein) the threads OR the
// magnitudes they write, and the next pass shifts the block up as it reads it,
// until its largest component is just below 2^61 (forward) or 2^60 (inverse).
// Bounds (|z| of a value; K <= P/2 samples):
//   after the chirp            < 2^60.5   (62-bit components, / 4)
//   first, unscaled pass       < 2^61.5   (two of its four inputs are zero)
//   forward passes             < 2^61.5   (also when shifted up)
//   times the kernel spectrum  < 2^60.5   (below 2 in magnitude, / 4)
//   inverse passes             < 2^60.5   (sums of four < 2^62.5 before their 1/4)
//   last, unscaled pass        < 2^62.5
// Measured on the CPU, normwise, against extended precision, beside an FP64
// Bluestein transform of the same length (white, steep, smooth, sparse, single-mode
// and chirp-shaped rings, P = 256 to 8192): at most 0.6 times its error; white
// rings 5e-17 to 1.2e-16 against 3e-16 to 4e-16.  With one upward shift, between the
// transforms, the same rings were up to 8 times FP64's error (K = 1023 white 1.7e-15
// against 8e-16, K = 4095 3.3e-15, chirp-shaped 2e-14).  The shifts, the ORs and the
// rounding of the inverse butterfly cost the ring kernels 4 to 6 % (8 maps at L =
// 1024, N = 4: 5.05 -> 5.30 ms analysis, 5.21 -> 5.41 synthesis; 64 at L = 128 0.772 ->
// 0.817, 0.793 -> 0.823); shifts after every pass would cost 11 to 14 %.
#pragma once

#include "fxarith.h"

namespace s2g {
namespace {

// what the core reads of a ring length (RingFFT, plan.h)
struct RingCore {
  int P, logP;
  int eb;  // the kernel spectrum is bhat 2^eb
  const int4 *bhat, *tw;
};

// Shared-memory layout: element i of the P = 2^lg point buffer (16-byte
// complex values, no padding) lives at swz(i) = i ^ X(i), where X(i) XORs bits
// 3-4 of i into bits 1-2, bits 3-5 into bits 0-2 and bits lg-3..lg-1 into bits
// 0-2 (the last term only for lg > 6).  X depends only on bits >= 3 and sets
// only bits 0-2, so swz is a bijection and its own inverse, and it is linear
// over GF(2): swz(a ^ b) = swz(a) ^ swz(b).  Every access pattern below (bit-
// reversed scatter and gather, the radix-4 passes at every span, stride-4 and
// linear sweeps) then touches 8 distinct 16-byte bank groups per quarter warp
// for P >= 256 (checked by enumerating the patterns on the CPU), without the
// 1/8 padding a skewed layout needs.
struct Swz {
  int top;  // lg - 3 when lg > 6, else 31 (the term vanishes for non-negative i)
};
S2G_DI Swz swz_of(int logP) { return Swz{logP > 6 ? logP - 3 : 31}; }
S2G_DI int swz(int i, Swz z) {
  return i ^ ((i >> 2) & 6) ^ ((i >> 3) & 7) ^ ((i >> z.top) & 7);
}
S2G_DI int brev(int k, int logP) {
#ifdef __CUDACC__
  return (int)(__brev((unsigned)k) >> (32 - logP));
#else
  unsigned r = 0;
  for (int i = 0; i < logP; ++i) r |= ((unsigned)k >> i & 1u) << (logP - 1 - i);
  return (int)r;
#endif
}
// buffer slot of bit-reversed position k
S2G_DI int slot_brev(int k, int logP) { return swz(brev(k, logP), swz_of(logP)); }

// The threads that transform one buffer.
#ifdef __CUDACC__
struct RingThreads {
  __device__ __forceinline__ int first() const { return threadIdx.x; }
  __device__ __forceinline__ int step() const { return blockDim.x; }
  __device__ __forceinline__ void sync() const { __syncthreads(); }
  // *slot |= v of every thread (no barrier)
  __device__ __forceinline__ void gather(int *slot, int v) const {
    v = __reduce_or_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) atomicOr(slot, v);
  }
};
#else
struct RingThreads {  // one thread
  int first() const { return 0; }
  int step() const { return 1; }
  void sync() const {}
  void gather(int *slot, int v) const { *slot |= v; }
};
#endif

// Read-only table loads with an L1 eviction priority: the twiddle table is
// read by every pass of every ring on the SM (kept: evict_last); the chirp and
// the chirp-kernel spectrum are read once per ring (evict_first).
#ifdef __CUDACC__
__device__ __forceinline__ int4 ld_keep(const int4 *p) {
  int4 v;
  asm("ld.global.nc.L1::evict_last.v4.s32 {%0, %1, %2, %3}, [%4];"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p));
  return v;
}
__device__ __forceinline__ int4 ld_once(const int4 *p) {
  int4 v;
  asm("ld.global.nc.L1::evict_first.v4.s32 {%0, %1, %2, %3}, [%4];"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p));
  return v;
}
#else
inline int4 ld_keep(const int4 *p) { return *p; }
inline int4 ld_once(const int4 *p) { return *p; }
#endif

// bits of the high words that differ from their sign, one place up (headroom tracking)
S2G_DI int high_bits(longlong2 v) {
  const int x = (int)(v.x >> 32), y = (int)(v.y >> 32);
  return (x ^ (x + x)) | (y ^ (y + y));
}
// left shift that brings the largest of the tracked components to 2^top at most
S2G_DI int headroom(int bits, int top) {
  const int k = clz32(bits) - (63 - top);
  return k > 0 ? k : 0;
}

S2G_DI void shift4(longlong2 &a0, longlong2 &a1, longlong2 &a2, longlong2 &a3, int k) {
  a0 = fx_shl(a0, k);
  a1 = fx_shl(a1, k);
  a2 = fx_shl(a2, k);
  a3 = fx_shl(a3, k);
}

// forward butterfly on bit-reversed data: stages s and s + 1 with
// w1 = w^2j (elements 1), w2 = w^j (elements 2), w3 = w^3j (elements 3), over 4
S2G_DI void dit4(longlong2 &a0, longlong2 &a1, longlong2 &a2, longlong2 &a3, int4 w1, int4 w2, int4 w3) {
  const longlong2 t0 = fx_sar(a0, 2), t1 = fx_mul4(a1, w1), t2 = fx_mul4(a2, w2), t3 = fx_mul4(a3, w3);
  const longlong2 b0 = fx_add(t0, t1), b1 = fx_sub(t0, t1), b2 = fx_add(t2, t3), b3 = fx_mul_i(fx_sub(t2, t3));
  a0 = fx_add(b0, b2);
  a2 = fx_sub(b0, b2);
  a1 = fx_sub(b1, b3);
  a3 = fx_add(b1, b3);
}
// a / 4, rounded to nearest, ties to even
S2G_DI longlong2 fx_quarter(longlong2 a) {
  return make_longlong2((a.x + 1 + ((a.x >> 2) & 1)) >> 2, (a.y + 1 + ((a.y >> 2) & 1)) >> 2);
}
// inverse butterfly, natural to bit-reversed order, over 4.  a0 is rounded without
// bias: y_0 is a sum along the a0 of every pass, so a downward shift gave the bin m = 0
// of every ring an error of the same sign (mean over white rings 2e-16 to 1.4e-15 of
// the level at P = 512 to 8192, against 1e-16 to 2e-16 in the worst bin of an FP64
// transform; so 5e-17 at most), and the monopole of a map ten times FP64's error.
// The forward butterfly's downward shift spreads over all bins (within the same 5e-17).
// Costs 1 to 2 % of the ring kernels, 2 to 3 % in both butterflies.
S2G_DI void dif4(longlong2 &a0, longlong2 &a1, longlong2 &a2, longlong2 &a3, int4 w1, int4 w2, int4 w3) {
  const longlong2 b0 = fx_add(a0, a2), b1 = fx_add(a1, a3), b2 = fx_sub(a0, a2), b3 = fx_mul_i(fx_sub(a1, a3));
  a0 = fx_quarter(fx_add(b0, b1));
  a1 = fx_mulc4(fx_sub(b0, b1), w1);
  a2 = fx_mulc4(fx_add(b2, b3), w2);
  a3 = fx_mulc4(fx_sub(b2, b3), w3);
}

// First pass of the core, fused with the producer: value(j) is the
// premultiplied a_j for j < P/2 (the second half of the padded sequence is zero
// and is not stored), written to the even bit-reversed positions and their
// neighbours.  Even log2 P: stages 1 and 2 of (a0, 0, a2, 0) with unit twiddles,
// where a0 and a2 are the elements j and j + P/4; odd: a copy (stage 1 of
// (a0, 0)).  Together with last_pass this
// leaves two sweeps over the buffer and two barriers of a ring to its neighbours:
// 64 maps at band-limit 128 0.800 -> 0.773 ms in the ring kernels, 32 at 256 1.385
// -> 1.350; 8 at 1024 5.12 -> 5.07 (analysis), 5.18 -> 5.20 (synthesis).
template <class V>
S2G_DI void first_pass(RingThreads th, longlong2 *buf, int P, int logP, V value) {
  if (logP & 1) {
    for (int j = th.first(); j < P / 2; j += th.step()) {
      const int b = slot_brev(j, logP);
      const longlong2 v = value(j);
      buf[b] = v;
      buf[b ^ 1] = v;
    }
  } else {
    for (int j = th.first(); j < P / 4; j += th.step()) {
      const int b = slot_brev(j, logP);
      const longlong2 a0 = value(j), a2 = value(j + P / 4), ia = fx_mul_i(a2);
      buf[b] = fx_add(a0, a2);
      buf[b ^ 1] = fx_sub(a0, ia);
      buf[b ^ 2] = fx_sub(a0, a2);
      buf[b ^ 3] = fx_add(a0, ia);
    }
  }
}
// Last pass, fused with the consumer: y_k for k < P/2 from the buffer that
// bluestein() leaves (unit twiddles; the other half of the outputs is not formed).
S2G_DI longlong2 last_pass(const longlong2 *buf, int P, int logP, int k) {
  if (logP & 1) {
    const int b = slot_brev(k, logP);
    return fx_add(buf[b], buf[b ^ 1]);
  }
  const int b = slot_brev(k & (P / 4 - 1), logP);
  const longlong2 a0 = buf[b], a1 = buf[b ^ 1], a2 = buf[b ^ 2], a3 = buf[b ^ 3];
  return k < P / 4 ? fx_add(fx_add(a0, a2), fx_add(a1, a3)) : fx_add(fx_sub(a0, a2), fx_mul_i(fx_sub(a1, a3)));
}
// the same in place, for consumers that read other CTAs' buffers:
// slot_brev(k) <- f(k, y_k) for k < n
template <class F>
S2G_DI void last_pass_in_place(RingThreads th, longlong2 *buf, int P, int logP, int n, F f) {
  if (logP & 1) {
    for (int k = th.first(); k < n; k += th.step()) {
      const int b = slot_brev(k, logP);
      buf[b] = f(k, fx_add(buf[b], buf[b ^ 1]));
    }
  } else {
    for (int k = th.first(); k < P / 4; k += th.step()) {
      const int b = slot_brev(k, logP);
      const longlong2 a0 = buf[b], a1 = buf[b ^ 1], a2 = buf[b ^ 2], a3 = buf[b ^ 3];
      if (k < n) buf[b] = f(k, fx_add(fx_add(a0, a2), fx_add(a1, a3)));
      if (k + P / 4 < n) buf[b ^ 2] = f(k + P / 4, fx_add(fx_sub(a0, a2), fx_mul_i(fx_sub(a1, a3))));
    }
  }
}

// One radix-4 pass of the forward transform (DIT: stages s and s + 1, span h =
// 2^(s-1)) or of the inverse (stages s and s - 1, h = 2^(s-2)); the block is read
// times 2^k if SHIFT; returns the bits of what it wrote if track.
template <bool DIT, bool SHIFT>
S2G_DI int radix4_pass(RingThreads th, longlong2 *buf, const RingCore &a, int lgh, int k, bool track) {
  const Swz z = swz_of(a.logP);
  const int h = 1 << lgh, h0 = a.logP & 1 ? 2 : 4;
  const int q1 = swz(h, z), q2 = swz(2 * h, z), q3 = swz(3 * h, z);
  int mx = 0;
  for (int i = th.first(); i < a.P / 4; i += th.step()) {
    const int jp = i & (h - 1);
    const int b = swz(((i >> lgh) << (lgh + 2)) + jp, z);
    const int4 *w = a.tw + (h - h0) + jp;
    const int4 w2 = ld_keep(w), w1 = ld_keep(w + h), w3 = ld_keep(w + 2 * h);
    longlong2 a0 = buf[b], a1 = buf[b ^ q1], a2 = buf[b ^ q2], a3 = buf[b ^ q3];
    if (SHIFT) shift4(a0, a1, a2, a3, k);
    if (DIT)
      dit4(a0, a1, a2, a3, w1, w2, w3);
    else
      dif4(a0, a1, a2, a3, w1, w2, w3);
    buf[b] = a0;
    buf[b ^ q1] = a1;
    buf[b ^ q2] = a2;
    buf[b ^ q3] = a3;
    if (track) mx |= high_bits(a0) | high_bits(a1) | high_bits(a2) | high_bits(a3);
  }
  return mx;
}
// The last forward pass, the kernel-spectrum product and the first inverse pass:
// they work on the same four elements, which stay in registers.
S2G_DI int middle_pass(RingThreads th, longlong2 *buf, const RingCore &a, int k) {
  const Swz z = swz_of(a.logP);
  const int h = a.P / 4, h0 = a.logP & 1 ? 2 : 4;
  const int q1 = swz(h, z), q2 = swz(2 * h, z), q3 = swz(3 * h, z);
  int mx = 0;
  for (int i = th.first(); i < h; i += th.step()) {
    const int b = swz(i, z);
    longlong2 a0 = buf[b], a1 = buf[b ^ q1], a2 = buf[b ^ q2], a3 = buf[b ^ q3];
    shift4(a0, a1, a2, a3, k);
    const int4 *w = a.tw + (h - h0) + i;
    const int4 w2 = ld_once(w), w1 = ld_once(w + h), w3 = ld_once(w + 2 * h);
    dit4(a0, a1, a2, a3, w1, w2, w3);
    a0 = fx_mul4(a0, ld_once(&a.bhat[i]));
    a1 = fx_mul4(a1, ld_once(&a.bhat[i + h]));
    a2 = fx_mul4(a2, ld_once(&a.bhat[i + 2 * h]));
    a3 = fx_mul4(a3, ld_once(&a.bhat[i + 3 * h]));
    dif4(a0, a1, a2, a3, w1, w2, w3);
    buf[b] = a0;
    buf[b ^ q1] = a1;
    buf[b ^ q2] = a2;
    buf[b ^ q3] = a3;
    mx |= high_bits(a0) | high_bits(a1) | high_bits(a2) | high_bits(a3);
  }
  return mx;
}

constexpr int kRingSlots = 4;   // headroom slots of a transform, zero before first_pass
constexpr int kLongRing = 13;   // log2 P from which the forward transform is rescaled twice before its end

// Between first_pass (barrier not yet passed) and last_pass (barrier passed): the
// buffer then holds y_k 2^S before the last pass, y the convolution times P, S the
// sum of the scalings.  Returns the sum of the upward shifts.  P >= 8.
// Shifted up: the second forward radix-4 pass, where a spike has lost two bits; the
// middle pass; the inverse pass after it, which has lost up to four; and from
// kLongRing the fourth forward pass (errors of steep rings over FP64's: P = 8192 1.6
// without it and 0.6 with it; P = 4096 0.5 without).
S2G_DI int bluestein(RingThreads th, longlong2 *buf, const RingCore &a, int *slots) {
  const int logP = a.logP;
  int sum = 0;
  bool known = false;  // *slots holds the bits of the buffer
  const auto shift = [&](int top) {
    const int k = known ? headroom(*slots++, top) : 0;
    sum += k;
    known = false;
    return k;
  };
  const auto done = [&](bool track, int mx) {
    if (track) th.gather(slots, mx);
    known = track;
    th.sync();
  };
  th.sync();
  int pass = 0;
  for (int s = logP & 1 ? 2 : 3; s + 1 < logP; s += 2, ++pass) {
    const bool track = pass == 0 || s + 3 >= logP || (pass == 2 && logP >= kLongRing);
    const int mx = known ? radix4_pass<true, true>(th, buf, a, s - 1, shift(61), track)
                         : radix4_pass<true, false>(th, buf, a, s - 1, 0, track);
    done(track, mx);
  }
  const int mx = middle_pass(th, buf, a, shift(61));
  int s = logP - 2;
  done(s >= 3, mx);
  if (s >= 3) {
    radix4_pass<false, true>(th, buf, a, s - 2, shift(60), false);
    th.sync();
  }
  for (s -= 2; s >= 3; s -= 2) {
    radix4_pass<false, false>(th, buf, a, s - 2, 0, false);
    th.sync();
  }
  return sum;
}
// values of first_pass are q 2^e0; those of last_pass then q 2^k, with 2 bits per
// radix-4 pass and the kernel spectrum's product, the shifts, the kernel spectrum's
// exponent, and the 1/P of the transforms
S2G_DI int core_exponent(const RingCore &a, int e0, int shifts) {
  const int passes = (a.logP - 1) >> 1;  // radix-4 passes of one direction
  return e0 + 4 * passes + 2 + a.eb - shifts - a.logP;
}

}  // namespace
}  // namespace s2g
