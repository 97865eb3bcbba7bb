// Ring DFTs: batched Bluestein transforms of the theta rings (length 2bl-1 on
// MW, 2bl on MWSS sampling) in shared memory, and the same fused with the
// gamma DFT across a thread-block cluster.
//
// Arithmetic.  Block fixed point on 64-bit integers (fxarith.h): each ring (or
// pair of real rings, or ring of all n-components) is scaled by one power of
// two from its largest exponent field, transformed in integers (ringcore.h, with
// the bounds and the accuracy: below an FP64 transform's error), and widened to
// FP64 once per output.  Both precision modes use it.
// A ring that holds an infinity or a NaN comes out as NaN.
//
// What bounds it: the wide multiply-adds (half rate) and the integer adds of
// the butterflies; a 4-point, two-stage butterfly takes 36 multiply-adds and
// 45 adds and shifts, against 256 FP32 instructions in double-float and 32
// FP64 instructions at 1/64 rate.  Measured, px2wav + wav2px at L = 1024, N = 4
// (real maps), rings and gamma DFTs: 2 maps in FP64 19.2 ms with FP64
// butterflies, 3.3 ms so; 32 maps at split precision 60.6 ms in double-float,
// 47.7 ms so.
//
// Table data comes as 62-bit fixed point (RingFFT, plan.h): chirp exp(i pi k^2
// / K), the passes' twiddles level by level (the passes below the first read
// 16 KB of them at P = 4096, contiguously, so they stay in L1), and the
// spectrum of the wrapped chirp over 2^eb.
#include <cooperative_groups.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <map>
#include <mutex>
#include <vector>

#include "common.h"
#include "ringcore.h"
#include "ringtables.h"
#include "kernels.h"
#include "smemlimit.h"
#include "timing.h"

namespace s2g {

namespace {

namespace cg = cooperative_groups;

struct RingArgs : RingCore {
  const void *rings;
  void *rings_out;  // inverse: output rings
  int64_t ring_stride;  // between rings of one map
  int64_t map_stride;   // between maps
  int rpm;              // rings per map
  const double2 *spec_in;
  double2 *spec_out;
  int64_t spec_stride;      // between spectra of one map
  int64_t spec_map_stride;  // between maps (spectra of ring r at spec_base(r))
  int spec_rpm;             // spectra per map
  int herm;                 // complex inverse: m < 0 taken as conj of m > 0 (real-valued ring)
  int sw, mlo;
  int nrings, bl, K;
  const int4 *chirp;
};

// Jobs of one launch: blocks (fused: clusters) first[q] .. first[q + 1] belong to
// job q.  The scales of small band-limits, a few microseconds each, share launches.
constexpr int kMaxJobs = 16;
struct RingGroup {
  int n;
  int first[kMaxJobs + 1];
  RingArgs a[kMaxJobs];
};

// One launch of ring DFTs fused with the gamma DFT (k_ring_inverse_gamma,
// k_gamma_ring_forward): NN <= kFuseMaxNN n-components per ring.
constexpr int kFuseMaxNN = 8;
constexpr int kFuseMaxTw = 128;
struct GammaItem {
  RingArgs a;
  const double2 *G;  // synthesis input: spectrum of component k of ring (b, t) at G + b gms + k gks + t W
  double2 *Gout;     // analysis output, the same addressing (all m from -(bl-1))
  int64_t gms, gks;
  int W, nt;
  void *fw;  // gamma slice g of ring (b, t) at fw + b fms + g npx + t K (double, or double2 unless real)
  int64_t fms, npx;
};
struct GammaFuse {
  int n;
  int first[kMaxJobs + 1];
  GammaItem it[kMaxJobs];
  int herm_k;  // real signals: the component with n = 0 (m >= 0 stored, at offset bl-1), else -1
  int ng;
  int et;               // the twiddles below are over 2^et
  int4 tw[kFuseMaxTw];  // [g NN + k] twiddles with their normalisation
};
template <class G>
__device__ __forceinline__ int job_of(const G &g, int block) {
  int q = 0;
  while (q + 1 < g.n && block >= g.first[q + 1]) ++q;
  return q;
}

// Pixels in memory: doubles, or floats that are widened as they are read and
// rounded to nearest as they are written, in integers; zeros, subnormals,
// infinities, NaN and results outside the normal range of a float go to the
// conversion instructions, out of line.  Complex floats are read and written as
// two 4-byte words, so that any float pointer will do.  Widening and rounding in
// passes of their own cost a gradient step with FP32 storage (band-limit 256, 32
// maps) 13.08 ms instead of 12.70, and the memory of the FP64 copies.  The type
// is a template parameter: as a run-time switch it slowed the FP64 launches by 1
// to 8 %.
template <bool F32>
__device__ __forceinline__ double ld_px(const void *p, int64_t i) {
  return F32 ? widen(((const float *)p)[i]) : ((const double *)p)[i];
}
template <bool F32>
__device__ __forceinline__ double2 ld_px2(const void *p, int64_t i) {
  if (F32) return make_double2(widen(((const float *)p)[2 * i]), widen(((const float *)p)[2 * i + 1]));
  return ((const double2 *)p)[i];
}
template <bool F32>
__device__ __forceinline__ void st_px(void *p, int64_t i, double v) {
  if (F32)
    ((float *)p)[i] = narrow(v);
  else
    ((double *)p)[i] = v;
}
template <bool F32>
__device__ __forceinline__ void st_px2(void *p, int64_t i, double2 v) {
  if (F32) {
    ((float *)p)[2 * i] = narrow(v.x);
    ((float *)p)[2 * i + 1] = narrow(v.y);
  } else {
    ((double2 *)p)[i] = v;
  }
}

// element offset of ring r (rings of a map are ring_stride apart, maps map_stride)
__device__ __forceinline__ int64_t ring_base(const RingArgs &a, int r) {
  return (int64_t)(r / a.rpm) * a.map_stride + (int64_t)(r % a.rpm) * a.ring_stride;
}
__device__ __forceinline__ int64_t spec_base(const RingArgs &a, int r) {
  return (int64_t)(r / a.spec_rpm) * a.spec_map_stride + (int64_t)(r % a.spec_rpm) * a.spec_stride;
}

// block-wide max of an int (blockDim.x <= 1024)
__device__ int block_max_int(int v) {
  __shared__ int redi[32];
  v = __reduce_max_sync(0xffffffffu, v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) redi[threadIdx.x >> 5] = v;
  __syncthreads();
  int m = 0;
  for (int i = 0; i < (int)((blockDim.x + 31) >> 5); ++i) m = max(m, redi[i]);
  return m;
}
__device__ __forceinline__ int emax2(int m, double2 z) { return max(m, max(exp_field(z.x), exp_field(z.y))); }

__device__ __forceinline__ double2 nan2() {
  const double n = double_of(0x7FF8000000000000ull);
  return make_double2(n, n);
}

constexpr int kRingThreads = 256;

template <bool REAL, bool F32>
__global__ void __launch_bounds__(kRingThreads, 3) k_ring_forward(const __grid_constant__ RingGroup grp) {
  extern __shared__ longlong2 buf[];
  __shared__ int s_mx[kRingSlots];
  const int job = job_of(grp, blockIdx.x), blk = blockIdx.x - grp.first[job];
  const RingArgs a = grp.a[job];  // by value: read once from the parameters
  const int K = a.K, P = a.P, logP = a.logP;
  const int r0 = REAL ? 2 * blk : blk;
  const bool has1 = REAL && (r0 + 1 < a.nrings);
  if (threadIdx.x < kRingSlots) s_mx[threadIdx.x] = 0;  // before the barriers of the maximum
  int em = 0;
  for (int j = threadIdx.x; j < K; j += blockDim.x) {
    if (REAL) {
      em = max(em, exp_field(ld_px<F32>(a.rings, ring_base(a, r0) + j)));
      if (has1) em = max(em, exp_field(ld_px<F32>(a.rings, ring_base(a, r0 + 1) + j)));
    } else {
      em = emax2(em, ld_px2<F32>(a.rings, ring_base(a, r0) + j));
    }
  }
  em = block_max_int(em);
  const int e = fx_exp(em);
  first_pass(RingThreads{}, buf, P, logP, [&](int j) {
    longlong2 v = make_longlong2(0, 0);
    if (j < K) {
      double2 x;
      if (REAL) {
        x.x = ld_px<F32>(a.rings, ring_base(a, r0) + j);
        x.y = has1 ? ld_px<F32>(a.rings, ring_base(a, r0 + 1) + j) : 0.0;
      } else {
        x = ld_px2<F32>(a.rings, ring_base(a, r0) + j);
      }
      v = fx_mulc4(fx_split2<62>(x, e), ld_once(&a.chirp[j]));  // x_j conj(c_j) / 4
    }
    return v;
  });
  const int sh = bluestein(RingThreads{}, buf, a, s_mx);
  const int k0 = core_exponent(a, e - 60, sh);
  if (!REAL) {
    double2 *out = a.spec_out + spec_base(a, r0);
    for (int c = threadIdx.x; c < a.sw; c += blockDim.x) {
      const int m = a.mlo + c;
      const int k = m < 0 ? m + K : m;
      const longlong2 y = fx_mulc(last_pass(buf, P, logP, k), ld_once(&a.chirp[k]));
      out[c] = em == kExpNonFinite ? nan2() : fx_join2(y, k0);
    }
  } else {
    double2 *out0 = a.spec_out + spec_base(a, r0);
    for (int m = threadIdx.x; m < a.sw; m += blockDim.x) {
      const int km = m ? K - m : 0;
      const longlong2 zm = fx_mulc2(last_pass(buf, P, logP, m), ld_once(&a.chirp[m]));
      const longlong2 zc = fx_conj(fx_mulc2(last_pass(buf, P, logP, km), ld_once(&a.chirp[km])));
      // A = (Z_m + conj Z_{-m})/2,  B = (Z_m - conj Z_{-m})/(2i)
      out0[m] = em == kExpNonFinite ? nan2() : fx_join2(fx_add(zm, zc), k0);
      if (has1) {
        const longlong2 d = fx_sub(zm, zc);
        out0[a.spec_stride + m] = em == kExpNonFinite ? nan2() : fx_join2(make_longlong2(d.y, -d.x), k0);
      }
    }
  }
}

template <bool REAL, bool F32>
__global__ void __launch_bounds__(kRingThreads, 3) k_ring_inverse(const __grid_constant__ RingGroup grp) {
  extern __shared__ longlong2 buf[];
  __shared__ int s_mx[kRingSlots];
  const int job = job_of(grp, blockIdx.x), blk = blockIdx.x - grp.first[job];
  const RingArgs a = grp.a[job];  // by value: read once from the parameters
  constexpr int BITS = REAL ? 61 : 62;  // A + i B of two rings
  const int K = a.K, P = a.P, logP = a.logP, bl = a.bl;
  const int r0 = REAL ? 2 * blk : blk;
  const bool has1 = REAL && (r0 + 1 < a.nrings);
  const double2 *s0 = a.spec_in + spec_base(a, r0);
  if (threadIdx.x < kRingSlots) s_mx[threadIdx.x] = 0;  // before the barriers of the maximum
  int em = 0;
  for (int c = threadIdx.x; c < a.sw; c += blockDim.x) {
    em = emax2(em, s0[c]);
    if (has1) em = emax2(em, s0[a.spec_stride + c]);
  }
  em = block_max_int(em);
  const int e = fx_exp(em);
  first_pass(RingThreads{}, buf, P, logP, [&](int j) {
    longlong2 v = make_longlong2(0, 0);
    if (j < K) {
      const int m = (j < bl) ? j : j - K;  // frequency of DFT bin j
      if (REAL) {
        const int am = m < 0 ? -m : m;
        if (am < a.sw) {
          longlong2 A = fx_split2<BITS>(s0[am], e);
          longlong2 B = has1 ? fx_split2<BITS>(s0[a.spec_stride + am], e) : make_longlong2(0, 0);
          if (m < 0) {
            A = fx_conj(A);
            B = fx_conj(B);
          }
          v = fx_add(A, fx_mul_i(B));
        }
      } else {
        const int c = m - a.mlo;
        if (c >= 0 && c < a.sw)
          v = fx_split2<BITS>(s0[c], e);
        else if (a.herm && m < 0 && -m - a.mlo < a.sw)
          v = fx_conj(fx_split2<BITS>(s0[-m - a.mlo], e));
      }
      // inverse DFT = conj(forward(conj z)):  a_j = conj(z_j) conj(c_j)
      v = fx_conj(fx_mul4(v, ld_once(&a.chirp[j])));
    }
    return v;
  });
  const int sh = bluestein(RingThreads{}, buf, a, s_mx);
  const int k0 = core_exponent(a, e - BITS + 2, sh);
  for (int p = threadIdx.x; p < K; p += blockDim.x) {
    // f_p = c_p conj(y_p)
    const longlong2 y = fx_mul(fx_conj(last_pass(buf, P, logP, p)), ld_once(&a.chirp[p]));
    const double2 f = em == kExpNonFinite ? nan2() : fx_join2(y, k0);
    if (REAL) {
      st_px<F32>(a.rings_out, ring_base(a, r0) + p, f.x);
      if (has1) st_px<F32>(a.rings_out, ring_base(a, r0 + 1) + p, f.y);
    } else {
      st_px2<F32>(a.rings_out, ring_base(a, r0) + p, f);
    }
  }
}

// ---------------------------------------------------------------------------
// Ring DFTs and gamma DFT in one launch
//
// The n-components F_k(t, p) (k < NN) of one theta-ring are transformed by a
// thread-block cluster of NN CTAs, one per component, each with the padded
// Bluestein buffer of the single-ring kernels.  The gamma DFT exchanges values
// between the components of a pixel through distributed shared memory, so the
// n-components never go to HBM:
//   synthesis: each CTA runs the inverse ring DFT of its component and leaves
//              F_k(p) in its buffer; after a cluster barrier each CTA computes
//              the gamma slices f_g(p) of its share of the pixels from all NN
//              buffers and writes them to f_wav.
//   analysis:  each CTA reads the gamma slices of its share of the pixels,
//              forms every component F_k(p), premultiplies by the chirp and
//              stores it into CTA k's buffer; after a cluster barrier each CTA
//              runs the forward ring DFT of its component and writes its
//              spectrum.
// One power-of-two scale per ring, the largest over the cluster; after the
// synthesis transforms the components are aligned to the largest exponent.
// gamma_g and gamma_{ng-g} have conjugate twiddles, so each pair of slices
// shares its products.
// ---------------------------------------------------------------------------

__device__ __forceinline__ int cluster_max_int(cg::cluster_group &cl, int *slot, int v, int nn) {
  const int m = block_max_int(v);
  if (threadIdx.x == 0) *slot = m;
  cl.sync();
  int r = 0;
  for (int j = 0; j < nn; ++j) r = max(r, *cl.map_shared_rank(slot, j));
  return r;
}

template <int NN, bool REAL, bool F32>
__global__ void __launch_bounds__(kRingThreads, 3) k_ring_inverse_gamma(const __grid_constant__ GammaFuse grp) {
  extern __shared__ longlong2 buf[];
  __shared__ int s_mx[kRingSlots], s_em, s_k;
  cg::cluster_group cl = cg::this_cluster();
  const int k = (int)cl.block_rank();
  const int job = job_of(grp, blockIdx.x / NN), r = blockIdx.x / NN - grp.first[job];
  const GammaItem gf = grp.it[job];  // by value: read once from the parameters
  const RingArgs &a = gf.a;
  const int b = r / gf.nt, t = r - b * gf.nt;
  const int K = a.K, P = a.P, logP = a.logP, bl = a.bl;
  const bool herm = (k == grp.herm_k);
  const int sw = herm ? bl : gf.W, mlo = herm ? 0 : -(bl - 1);
  const double2 *s0 = gf.G + (int64_t)b * gf.gms + (int64_t)k * gf.gks + (int64_t)t * gf.W + (herm ? bl - 1 : 0);
  if (threadIdx.x < kRingSlots) s_mx[threadIdx.x] = 0;  // before the barriers of the maximum
  int em = 0;
  for (int c = threadIdx.x; c < sw; c += blockDim.x) em = emax2(em, s0[c]);
  em = cluster_max_int(cl, &s_em, em, NN);
  const int e = fx_exp(em);
  first_pass(RingThreads{}, buf, P, logP, [&](int j) {
    longlong2 v = make_longlong2(0, 0);
    if (j < K) {
      const int m = (j < bl) ? j : j - K;
      const int c = m - mlo;
      if (c >= 0 && c < sw)
        v = fx_split2<62>(s0[c], e);
      else if (herm && m < 0 && -m < sw)
        v = fx_conj(fx_split2<62>(s0[-m], e));
      v = fx_conj(fx_mul4(v, ld_once(&a.chirp[j])));
    }
    return v;
  });
  const int sh = bluestein(RingThreads{}, buf, a, s_mx);
  // F_k(p) / 2 = c_p conj(y_p) / 2, in place (p -> brev(p) is one-to-one); components < 2^61.5
  last_pass_in_place(RingThreads{}, buf, P, logP, K,
                     [&](int p, longlong2 y) { return fx_mul2(fx_conj(y), ld_once(&a.chirp[p])); });
  if (threadIdx.x == 0) s_k = core_exponent(a, e - 60, sh) + 1;
  cl.sync();
  // gamma slices of this CTA's share of the pixels
  int kj[NN], km = INT_MIN;
#pragma unroll
  for (int j = 0; j < NN; ++j) {
    kj[j] = *cl.map_shared_rank(&s_k, j);
    km = max(km, kj[j]);
  }
  const int ko = km + 2 + grp.et;
  const bool bad = em == kExpNonFinite;
  const int chunk = (K + NN - 1) / NN;
  const int p1 = min(K, (k + 1) * chunk);
  const int64_t obase = (int64_t)b * gf.fms + (int64_t)t * K;
  // with w = C + i S (each product over 4: sums of 8 stay below 2^62.5):
  //   real:    f_g = A - B, f_{ng-g} = A + B, A = sum_k C Re z_k, B = sum_k S Im z_k
  //   complex: f_g = U + i V, f_{ng-g} = U - i V, U = sum_k C z_k, V = sum_k S z_k
  for (int p = k * chunk + threadIdx.x; p < p1; p += blockDim.x) {
    const int i = slot_brev(p, logP);
    longlong2 z[NN];
#pragma unroll
    for (int j = 0; j < NN; ++j) z[j] = fx_sar(*cl.map_shared_rank(buf + i, j), min(63, km - kj[j]));
    for (int g = 0; 2 * g <= grp.ng; ++g) {
      const int g2 = grp.ng - g;  // the conjugate partner (g = 0 and g2 == g have none)
      const int64_t o = obase + (int64_t)g * gf.npx + p, o2 = obase + (int64_t)g2 * gf.npx + p;
      const bool pair = g > 0 && g2 != g;
      if (REAL) {
        long long A = 0, B = 0;
#pragma unroll
        for (int j = 0; j < NN; ++j) {
          const int4 w = grp.tw[g * NN + j];
          A = fx_mac4(A, z[j].x, w.x, w.y);
          B = fx_mac4(B, z[j].y, w.z, w.w);
        }
        st_px<F32>(gf.fw, o, bad ? nan2().x : fx_join(A - B, ko));
        if (pair) st_px<F32>(gf.fw, o2, bad ? nan2().x : fx_join(A + B, ko));
      } else {
        longlong2 U = make_longlong2(0, 0), V = make_longlong2(0, 0);
#pragma unroll
        for (int j = 0; j < NN; ++j) {
          const int4 w = grp.tw[g * NN + j];
          U = make_longlong2(fx_mac4(U.x, z[j].x, w.x, w.y), fx_mac4(U.y, z[j].y, w.x, w.y));
          V = make_longlong2(fx_mac4(V.x, z[j].x, w.z, w.w), fx_mac4(V.y, z[j].y, w.z, w.w));
        }
        const longlong2 iV = fx_mul_i(V);
        st_px2<F32>(gf.fw, o, bad ? nan2() : fx_join2(fx_add(U, iV), ko));
        if (pair) st_px2<F32>(gf.fw, o2, bad ? nan2() : fx_join2(fx_sub(U, iV), ko));
      }
    }
  }
  cl.sync();  // peers read this buffer until here
}

template <int NN, bool REAL, bool F32>
__global__ void __launch_bounds__(kRingThreads, 3) k_gamma_ring_forward(const __grid_constant__ GammaFuse grp) {
  extern __shared__ longlong2 buf[];
  __shared__ int s_mx[kRingSlots], s_em;
  cg::cluster_group cl = cg::this_cluster();
  const int k = (int)cl.block_rank();
  const int job = job_of(grp, blockIdx.x / NN), r = blockIdx.x / NN - grp.first[job];
  const GammaItem gf = grp.it[job];  // by value: read once from the parameters
  const RingArgs &a = gf.a;
  const int b = r / gf.nt, t = r - b * gf.nt;
  const int K = a.K, P = a.P, logP = a.logP;
  const int chunk = (K + NN - 1) / NN;
  const int p0 = k * chunk, p1 = min(K, p0 + chunk);
  const int64_t ibase = (int64_t)b * gf.fms + (int64_t)t * K;
  if (threadIdx.x < kRingSlots) s_mx[threadIdx.x] = 0;  // before the barriers of the maximum
  int em = 0;
  for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x)
    for (int g = 0; g < grp.ng; ++g) {
      const int64_t o = ibase + (int64_t)g * gf.npx + p;
      if (REAL)
        em = max(em, exp_field(ld_px<F32>(gf.fw, o)));
      else
        em = emax2(em, ld_px2<F32>(gf.fw, o));
    }
  em = cluster_max_int(cl, &s_em, em, NN);
  const int e = fx_exp(em);
  // the zero padding of this CTA's own buffer
  for (int j = K + threadIdx.x; j < P / 2; j += blockDim.x) buf[slot_brev(j, logP)] = make_longlong2(0, 0);
  // gamma_g and gamma_{ng-g} have conjugate twiddles w = C + i S and C - i S:
  // each pair contributes C (f_g + f_{ng-g}) + i S (f_g - f_{ng-g}).  The
  // twiddles' magnitudes sum to at most 1 over g (et), so F_k / 4 stays below
  // 2^59.5 and leaves the chirp twice as large.
  for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
    longlong2 acc[NN];
#pragma unroll
    for (int j = 0; j < NN; ++j) acc[j] = make_longlong2(0, 0);
    for (int g = 0; 2 * g <= grp.ng; ++g) {
      const int g2 = grp.ng - g;
      const bool pair = g > 0 && g2 != g;
      const int64_t o = ibase + (int64_t)g * gf.npx + p, o2 = ibase + (int64_t)g2 * gf.npx + p;
      if (REAL) {
        const long long fa = fx_split<61>(ld_px<F32>(gf.fw, o), e);
        const long long fb = pair ? fx_split<61>(ld_px<F32>(gf.fw, o2), e) : 0;
        const long long Pp = fa + fb, Q = fa - fb;
#pragma unroll
        for (int j = 0; j < NN; ++j) {
          const int4 w = grp.tw[g * NN + j];
          acc[j] = make_longlong2(fx_mac4(acc[j].x, Pp, w.x, w.y), fx_mac4(acc[j].y, Q, w.z, w.w));
        }
      } else {
        const longlong2 fa = fx_split2<61>(ld_px2<F32>(gf.fw, o), e);
        const longlong2 fb = pair ? fx_split2<61>(ld_px2<F32>(gf.fw, o2), e) : make_longlong2(0, 0);
        const longlong2 Pp = fx_add(fa, fb), Q = fx_sub(fa, fb);
#pragma unroll
        for (int j = 0; j < NN; ++j) {
          const int4 w = grp.tw[g * NN + j];
          // C P + i S Q
          acc[j] = make_longlong2(fx_mac4(fx_mac4(acc[j].x, Pp.x, w.x, w.y), -Q.y, w.z, w.w),
                                  fx_mac4(fx_mac4(acc[j].y, Pp.y, w.x, w.y), Q.x, w.z, w.w));
        }
      }
    }
    const int4 ch = ld_once(&a.chirp[p]);
    const int i = slot_brev(p, logP);
#pragma unroll
    for (int j = 0; j < NN; ++j) *cl.map_shared_rank(buf + i, j) = fx_product<3, true>(acc[j], ch);
  }
  cl.sync();  // every component's buffer is complete
  // in place: a thread reads only the slots that it writes
  first_pass(RingThreads{}, buf, P, logP, [&](int j) { return buf[slot_brev(j, logP)]; });
  const int sh = bluestein(RingThreads{}, buf, a, s_mx);
  const int k0 = core_exponent(a, e - 60 + grp.et, sh);
  double2 *out = gf.Gout + (int64_t)b * gf.gms + (int64_t)k * gf.gks + (int64_t)t * gf.W;
  for (int c = threadIdx.x; c < gf.W; c += blockDim.x) {
    const int m = c - (a.bl - 1);
    const int q = m < 0 ? m + K : m;
    const longlong2 y = fx_mulc(last_pass(buf, P, logP, q), ld_once(&a.chirp[q]));
    out[c] = em == kExpNonFinite ? nan2() : fx_join2(y, k0);
  }
}

// ---------------------------------------------------------------------------
// launches
// ---------------------------------------------------------------------------

RingArgs ring_args(const RingFFT &rf, int bl, int nrings) {
  RingArgs a{};
  a.spec_rpm = 1 << 30;  // single-level spectrum addressing unless set
  a.spec_map_stride = 0;
  a.K = rf.K;
  a.P = rf.P;
  a.logP = rf.logP;
  a.eb = rf.eb;
  a.bl = bl;
  a.nrings = nrings;
  a.chirp = rf.chirp;
  a.bhat = rf.bhat;
  a.tw = rf.tw;
  return a;
}

int ring_threads(int P) { return std::min(kRingThreads, std::max(32, P / 4)); }
size_t ring_smem(int P) { return sizeof(longlong2) * (size_t)P; }

// Shared memory of the ring kernels: one P-point buffer of 16-byte values, and
// the smallest carveout that holds the CTAs an SM's registers allow (3 of 256
// threads at 80 registers; with the 1 KB the system takes per CTA and the static
// arrays): 164 of 228 KB would not hold three at P = 4096, 196 does and leaves
// the rest to the L1.  Room for only three CTAs whatever their size kept the
// small rings' CTAs of 32 to 128 threads from filling the SM: 64 maps at
// band-limit 128 took 1.19 ms in the ring kernels and take 0.80, at 48 0.34 and
// 0.21; band-limit 1024 is unchanged.
void ring_smem_attrs(const void *kernel, int P) {
  const size_t smem = ring_smem(P);
  const int ctas = std::min(32, 3 * kRingThreads / ring_threads(P));
  constexpr int kSizes[] = {8, 16, 32, 64, 100, 132, 164, 196, 228};  // KB of shared memory an SM can set aside
  int kb = 228;
  for (int k : kSizes)
    if (ctas * (smem + 1024 + 256) <= (size_t)k * 1024) {
      kb = k;
      break;
    }
  static SharedMemoryLimits limits;
  limits.prepare(
      kernel, smem, 100 * kb / 228,
      [&](size_t b) { S2G_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b)); },
      [&](int c) { S2G_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, c)); });
}

int largest_P(const RingGroup &g) {
  int P = 0;
  for (int q = 0; q < g.n; ++q) P = std::max(P, g.a[q].P);
  return P;
}

template <class KF>
void launch_ring(KF kernel, const RingGroup &g, cudaStream_t st) {
  const int P = largest_P(g);
  ring_smem_attrs((const void *)kernel, P);
  kernel<<<g.first[g.n], ring_threads(P), ring_smem(P), st>>>(g);
  S2G_LAUNCHED();
}

// Work model of one Bluestein transform of padded length P (for the timing
// report), in 32 x 32 + 64 multiply-adds: 12 per complex product; 3 products
// per 4 points and radix-4 pass ((log2 P - 1)/2 passes each way), one per
// point for the kernel spectrum and two per sample for the chirps.
double ring_work(const RingArgs &a, int nblk) {
  const double P = a.P, passes = (a.logP - 1) / 2;
  return (double)nblk * 12.0 * (2.0 * passes * 0.75 * P + P + 2.0 * a.K);
}

// launches of up to kMaxJobs jobs
template <class LAUNCH>
void run_rings(const std::vector<RingJob> &jobs, int ss, bool real, bool forward, LAUNCH &&launch, cudaStream_t st) {
  RingGroup g;
  double fl = 0, by = 0;
  bool f32 = false;
  g.n = 0;
  g.first[0] = 0;
  const auto flush = [&] {
    if (!g.n) return;
    KTimer kt(KC_RING, st, fl, by);
    launch(g, f32);
    g.n = 0;
    fl = by = 0;
  };
  for (const RingJob &j : jobs) {
    if (j.nrings <= 0) continue;
    if (j.f32 != f32) flush();  // one storage type per launch
    f32 = j.f32;
    RingArgs a = ring_args(ring_fft(grid_ring_len(j.bl, ss)), j.bl, j.nrings);
    a.ring_stride = j.ring_stride;
    a.map_stride = j.map_stride;
    a.rpm = j.rpm;
    a.spec_stride = j.spec_stride;
    a.spec_map_stride = j.spec_map_stride;
    a.spec_rpm = j.spec_rpm;
    a.herm = j.herm ? 1 : 0;
    a.sw = j.sw;
    a.mlo = j.mlo;
    if (forward) {
      a.rings = j.in;
      a.spec_out = (double2 *)j.out;
    } else {
      a.spec_in = (const double2 *)j.in;
      a.rings_out = j.out;
    }
    const int nblk = real ? (j.nrings + 1) / 2 : j.nrings;
    if (timing_enabled()) fl += ring_work(a, nblk);
    by += (double)j.nrings * a.K * (real ? 8.0 : 16.0) * (j.f32 ? 0.5 : 1.0) + (double)j.nrings * a.sw * 16.0;
    g.a[g.n] = a;
    g.first[g.n + 1] = g.first[g.n] + nblk;
    if (++g.n == kMaxJobs) flush();
  }
  flush();
}

// Twiddles of the fused gamma DFT: synthesis c e^{i n_k gamma_g} (x2 for
// n_k != 0 on real signals, which stand for the +-n pair), analysis
// c e^{-i n_k gamma_g}; gamma_g = 2 pi g / ng.  Stored over 2^et: synthesis
// |w| <= 1, analysis sum_g |w| <= 1.
void fuse_twiddles(GammaFuse &gf, const std::vector<int> &ns, int ng, bool real, double c, bool synth) {
  const int nn = (int)ns.size();
  const double top = synth ? (real ? 2.0 * c : c) : ng * c;
  gf.et = 0;
  while (std::ldexp(1.0, gf.et) < top) ++gf.et;
  while (std::ldexp(1.0, gf.et - 1) >= top) --gf.et;
  for (int g = 0; g < ng; ++g)
    for (int k = 0; k < nn; ++k) {
      const long double x = 2.0L * (long double)((ns[k] * g) % ng) / (long double)ng;  // angle / pi
      const long double pi = 3.141592653589793238462643383279502884L;
      const long double f = ldexpl(synth && real && ns[k] != 0 ? 2.0L * c : (long double)c, -gf.et);
      gf.tw[g * nn + k] = fixed62(f * cosl(pi * x), (synth ? f : -f) * sinl(pi * x));
    }
}

cudaLaunchConfig_t fused_config(int nctas, int nn, int P, cudaLaunchAttribute *at, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nctas);
  cfg.blockDim = dim3(ring_threads(P));
  cfg.dynamicSmemBytes = ring_smem(P);
  cfg.stream = st;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)nn;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

template <class KF>
void launch_fused(KF kernel, const GammaFuse &gf, int nn, cudaStream_t st) {
  int P = 0;
  for (int q = 0; q < gf.n; ++q) P = std::max(P, gf.it[q].a.P);
  ring_smem_attrs((const void *)kernel, P);
  cudaLaunchAttribute at[1];
  const cudaLaunchConfig_t cfg = fused_config(gf.first[gf.n] * nn, nn, P, at, st);
  S2G_CUDA(cudaLaunchKernelEx(&cfg, kernel, gf));
  S2G_LAUNCHED();
}

// Whether a cluster of nn CTAs of the fused kernels (P-point buffers) can be
// resident on this GPU: asked once per (nn, P) of the device in use.
bool cluster_fits(int nn, int P) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, bool> known;
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_pair(nn, P);
  auto it = known.find(key);
  if (it != known.end()) return it->second;
  const void *kern = nullptr;
  switch (nn) {
    case 2: kern = (const void *)k_ring_inverse_gamma<2, false, false>; break;
    case 3: kern = (const void *)k_ring_inverse_gamma<3, false, false>; break;
    case 4: kern = (const void *)k_ring_inverse_gamma<4, false, false>; break;
    case 5: kern = (const void *)k_ring_inverse_gamma<5, false, false>; break;
    case 6: kern = (const void *)k_ring_inverse_gamma<6, false, false>; break;
    case 7: kern = (const void *)k_ring_inverse_gamma<7, false, false>; break;
    default: kern = (const void *)k_ring_inverse_gamma<8, false, false>; break;
  }
  bool ok = ring_smem(P) <= 227 * 1024;
  if (ok) {
    ring_smem_attrs(kern, P);
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = fused_config(nn, nn, P, at, nullptr);
    int nclusters = 0;
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&nclusters, kern, &cfg);
    if (e != cudaSuccess) {  // not fusable in this call; asked again by the next
      cudaGetLastError();
      return false;
    }
    ok = nclusters > 0;
  }
  known[key] = ok;
  return ok;
}

}  // namespace

bool ring_gamma_fusable(int nn, int ng, int bl, int ss) {
  if (nn < 2 || nn > kFuseMaxNN || ng * nn > kFuseMaxTw) return false;
  return cluster_fits(nn, ring_fft(grid_ring_len(bl, ss)).P);
}

namespace {
// multiply-adds of the gamma products: 3 per real product, (ng + 1)/2 slice pairs
double gamma_work(double px, int ng, int nn, bool real) { return px * ((ng + 1) / 2) * nn * (real ? 6.0 : 12.0); }

// launches of up to kMaxJobs jobs of one direction
template <class LAUNCH>
void run_fused(const std::vector<GammaJob> &jobs, const std::vector<int> &ns, int ng, bool real, double c, int ss,
               bool synth, LAUNCH &&launch, cudaStream_t st) {
  const int nn = (int)ns.size();
  GammaFuse g;
  double fl = 0, by = 0;
  bool f32 = false;
  g.n = 0;
  g.first[0] = 0;
  g.ng = ng;
  g.herm_k = -1;
  for (int k = 0; k < nn; ++k)
    if (synth && real && ns[k] == 0) g.herm_k = k;
  const auto flush = [&] {
    if (!g.n) return;
    KTimer kt(KC_RING, st, fl, by);
    launch(g, f32);
    g.n = 0;
    fl = by = 0;
  };
  bool tw = false;
  for (const GammaJob &j : jobs) {
    S2G_REQUIRE(ring_gamma_fusable(nn, ng, j.bl, ss), ERR_UNSUPPORTED, "fused ring/gamma DFT: unsupported shape");
    const int nt = grid_rings(j.bl, ss), nrings = j.nb * nt;
    if (nrings <= 0) continue;
    if (j.f32 != f32) flush();  // one storage type per launch
    f32 = j.f32;
    if (!tw) fuse_twiddles(g, ns, ng, real, c, synth);
    tw = true;
    GammaItem &it = g.it[g.n];
    it.a = ring_args(ring_fft(grid_ring_len(j.bl, ss)), j.bl, nrings);
    it.G = j.G;
    it.Gout = j.Gout;
    it.gms = j.gms;
    it.gks = j.gks;
    it.W = 2 * j.bl - 1;
    it.nt = nt;
    it.fw = j.fw;
    it.fms = j.fms;
    it.npx = (int64_t)nt * it.a.K;
    const double px = (double)nrings * it.a.K;
    if (timing_enabled()) fl += ring_work(it.a, nrings * nn) + gamma_work(px, ng, nn, real);
    by += (double)nrings * nn * it.W * 16.0 + px * ng * (real ? 8.0 : 16.0) * (j.f32 ? 0.5 : 1.0);
    g.first[g.n + 1] = g.first[g.n] + nrings;
    if (++g.n == kMaxJobs) flush();
  }
  flush();
}
}  // namespace

void ring_inverse_gamma(const std::vector<GammaJob> &jobs, const std::vector<int> &ns, int ng, bool real, double c,
                        int ss, cudaStream_t st) {
  run_fused(jobs, ns, ng, real, c, ss, true, [&](const GammaFuse &gf, bool f32) {
    switch ((int)ns.size()) {
#define S2G_FUSE(N)                                               \
  case N:                                                         \
    if (f32)                                                      \
      real ? launch_fused(k_ring_inverse_gamma<N, true, true>, gf, N, st)           \
           : launch_fused(k_ring_inverse_gamma<N, false, true>, gf, N, st);         \
    else                                                          \
      real ? launch_fused(k_ring_inverse_gamma<N, true, false>, gf, N, st)          \
           : launch_fused(k_ring_inverse_gamma<N, false, false>, gf, N, st);        \
    break;
      S2G_FUSE(2) S2G_FUSE(3) S2G_FUSE(4) S2G_FUSE(5) S2G_FUSE(6) S2G_FUSE(7) S2G_FUSE(8)
#undef S2G_FUSE
      default: break;
    }
  }, st);
}

void gamma_ring_forward(const std::vector<GammaJob> &jobs, const std::vector<int> &ns, int ng, bool real, double c,
                        int ss, cudaStream_t st) {
  run_fused(jobs, ns, ng, real, c, ss, false, [&](const GammaFuse &gf, bool f32) {
    switch ((int)ns.size()) {
#define S2G_FUSE(N)                                               \
  case N:                                                         \
    if (f32)                                                      \
      real ? launch_fused(k_gamma_ring_forward<N, true, true>, gf, N, st)           \
           : launch_fused(k_gamma_ring_forward<N, false, true>, gf, N, st);         \
    else                                                          \
      real ? launch_fused(k_gamma_ring_forward<N, true, false>, gf, N, st)          \
           : launch_fused(k_gamma_ring_forward<N, false, false>, gf, N, st);        \
    break;
      S2G_FUSE(2) S2G_FUSE(3) S2G_FUSE(4) S2G_FUSE(5) S2G_FUSE(6) S2G_FUSE(7) S2G_FUSE(8)
#undef S2G_FUSE
      default: break;
    }
  }, st);
}

void ring_forward_many(const std::vector<RingJob> &jobs, int ss, bool real, cudaStream_t st) {
  run_rings(jobs, ss, real, true, [&](const RingGroup &g, bool f32) {
    if (f32)
      real ? launch_ring(k_ring_forward<true, true>, g, st) : launch_ring(k_ring_forward<false, true>, g, st);
    else
      real ? launch_ring(k_ring_forward<true, false>, g, st) : launch_ring(k_ring_forward<false, false>, g, st);
  }, st);
}
void ring_inverse_many(const std::vector<RingJob> &jobs, int ss, bool real, cudaStream_t st) {
  run_rings(jobs, ss, real, false, [&](const RingGroup &g, bool f32) {
    if (f32)
      real ? launch_ring(k_ring_inverse<true, true>, g, st) : launch_ring(k_ring_inverse<false, true>, g, st);
    else
      real ? launch_ring(k_ring_inverse<true, false>, g, st) : launch_ring(k_ring_inverse<false, false>, g, st);
  }, st);
}

}  // namespace s2g
