// Contractions against recomputed (checkpointed) Wigner tables: FP64, and at split
// precision the multiply-adds in double-float.
//
// A recomputed table keeps, per m, theta ring t and segment of kSeg degrees,
// the pair (d^{lc}, d^{lc+1}) = (a, b) 2^E from the double-double recursion
// (plan.cu).  The kernels here regenerate each segment in FP64 with the
// three-term recursion in l, written with u = 2 sin^2(theta/2) (north) or
// u = 2 cos^2(theta/2) (south) so that the large integer parts cancel exactly:
//   d^{l+1} = (q_l + p_l u) d^l - c2_l d^{l-1}
//   north: p_l = -r l(l+1), q_l = r (l(l+1) - m n);  south: p_l = r l(l+1), q_l = -r (l(l+1) + m n)
//   r = (2l+1) / (l S_{l+1}),  c2_l = (l+1) S_l / (l S_{l+1}),  S_l = sqrt((l^2-m^2)(l^2-n^2))
// rescaled within a segment: with d^l = lam_l w_l, lam_{lc} = lam_{lc+1} = 1 and
// lam_{l+1} = c2_l lam_{l-1}, it is w_{l+1} = (p' u + q') w_l - w_{l-1} with (p', q') =
// (p, q) lam_l / (c2_l lam_{l-1}): two FP64 instructions per value.  lam depends on
// (l, m) only and is folded into the coefficients (l -> t) or the output weight (t
// -> l).  p', q' and lam are part of the table (WignerTable::rec): computing them
// per launch and ring tile (two square roots and two divisions per degree, and a
// serial product over the segment) cost a third of the FP64 work.  Restarting
// every kSeg degrees from the double-double checkpoints keeps the recursion's
// rounding growth to a few ulps (a plain FP64 run over l < 2048 drifts by ~3e-12
// near the poles).
// One regenerated row serves every problem on its table at once (parts): the
// scales of one band-limit, and directions n and -n (d_{m,-n} = (-1)^{m+n}
// d_{-m,n}), up to 4 parts per launch.
// Values are carried scaled by 2^-E, one scale per ring and segment, applied
// once per segment: to the partial sums (l -> t) or to the inputs (t -> l).
//
//   k_rc_l2t   out[b][t][m] = sign sum_l d^l(theta_t) w(l) x_b(l, m)       one thread per ring t
//   k_rc_t2l   y_b(l, m)   = sign w(l) sum_t d^l(theta_t) in_b(t, m)       a 128 x 64 d tile in shared memory
//   k_apply_w  the forward quadrature W_eps(m) (or its transpose) on ring spectra: the
//              stored path's Q = D^T W becomes D^T applied after W (FP64 tiled GEMM)
#include <algorithm>
#include <vector>

#include "autotune.h"
#include "common.h"
#include "ddarith.h"
#include "dfarith.h"
#include "kernels.h"
#include "mixed.h"
#include "recompute.h"
#include "runtime.h"
#include "timing.h"

namespace s2g {

namespace {

constexpr int kRcT = 128;  // threads per CTA: rings per tile
static_assert(kRcT == 2 * kSeg, "t -> l maps two threads per degree of a segment");

constexpr int kRcParts = 4;
// One problem on the table: row mt of the table is its m = mt, or -mt (neg).
struct RcPart {
  int mlo, mhi, lmin;
  int neg;
  const double2 *w;
  const double2 *src;  // l -> t: x (l^2 + l + m);  t -> l: spectra [t][m - s_mlo]
  double2 *dst;        // l -> t: spectra [t][m - d_mlo];  t -> l: y (l^2 + l + m)
};
struct RcArgs {
  int bl, nt, an, tmlo;
  const int64_t *coff;
  const double2 *ck;
  const int *ck_e;
  const double2 *uq;
  const RcRec *rec;
  const int64_t *roff;
  int np, lmin;  // parts, smallest lmin
  RcPart part[kRcParts];
  double wscale;
  int wconj;
  int64_t ss;
  int sw, s_mlo, x_half;
  int64_t ds;
  int dw, d_mlo;
  int nb, mpc;  // maps, maps per CTA: column c = part c / mpc, map b0 + c % mpc
};

// explicit roundings: every instantiation (columns per CTA) gives the same bits
__device__ __forceinline__ double2 cmul_(double2 a, double2 b) {
  return make_double2(__fma_rn(a.x, b.x, __dmul_rn(-a.y, b.y)), __fma_rn(a.x, b.y, __dmul_rn(a.y, b.x)));
}
__device__ __forceinline__ double2 weight_of(const RcArgs &a, const RcPart &P, int l) {
  double2 w = P.w ? P.w[l] : make_double2(1.0, 0.0);
  if (a.wconj) w.y = -w.y;
  return make_double2(w.x * a.wscale, w.y * a.wscale);
}
// m of a part at table row mt, whether the part has it, and its sign
struct RcM {
  int m;
  bool on;
  double sign;
};
__device__ __forceinline__ RcM rc_m(const RcArgs &a, const RcPart &P, int mt) {
  RcM r;
  r.m = P.neg ? -mt : mt;
  r.on = r.m >= P.mlo && r.m <= P.mhi;
  r.sign = P.neg && ((r.m + a.an) & 1) ? -1.0 : 1.0;
  return r;
}
// l -> t coefficient of a column: x(l, m) w(l) f
__device__ __forceinline__ double2 rc_coef(const RcArgs &a, const RcPart &P, int m, int b, int l, double f) {
  const int64_t base = (int64_t)b * a.ss + (int64_t)l * l + l;
  double2 v;
  if (a.x_half && m < 0) {
    v = P.src[base - m];
    v.y = -v.y;
    if (m & 1) v = make_double2(-v.x, -v.y);
  } else {
    v = P.src[base + m];
  }
  const double2 w = weight_of(a, P, l);
  return cmul_(v, make_double2(w.x * f, w.y * f));
}

// The rescaled recursion of every (m, segment): rec[roff[mi] + l - l0] = (p', q'
// north, q' south, lam) of degree l (p', q' unused at a segment's first degree).
//   p' = (2l+1)(l+1) / S_{l+1} f,  q' = (2l+1)(l(l+1) -+ m n) / (l S_{l+1}) f,  f = lam_l / lam_{l+1}
// in double-double, rounded once: lam is a product over the segment, and in FP64 its
// roundings and those of f made the contractions less accurate than the unscaled
// recursion (inverse transforms of white maps on 30 tables of 64 <= L <= 700, rms: 1.17
// times its error; so 0.74 times, having fewer roundings per value).
__global__ void k_rc_rec(RcRec *__restrict__ rec, const int64_t *__restrict__ roff, int bl, int an, int mlo,
                         int nm, int maxseg) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (int64_t)nm * maxseg) return;
  const int mi = (int)(gid / maxseg), c = (int)(gid % maxseg);
  const int m = mlo + mi, am = m < 0 ? -m : m, l0 = am > an ? am : an;
  const int lc = l0 + c * kSeg, n = min(kSeg, bl - lc);
  if (n <= 0) return;
  RcRec *out = rec + roff[mi] + c * kSeg;
  out[0] = RcRec{0.0, 0.0, 0.0, 1.0};
  // the integers below stay under 2^53 up to the largest band-limit
  const double mn = (double)m * an, m2 = (double)m * m, n2 = (double)an * an;
  dd lam0{1.0, 0.0}, lam1{1.0, 0.0};  // lam of degrees lc + i - 1 and lc + i
  for (int i = 1; i < n; ++i) {
    const double l = lc + i, ll1 = l * (l + 1.0);
    const dd s1 = dd_sqrt_d(((l + 1.0) * (l + 1.0) - m2) * ((l + 1.0) * (l + 1.0) - n2));
    const dd s0 = dd_sqrt_d((l * l - m2) * (l * l - n2));
    const dd ls1 = dd_mul_d(s1, l);
    const dd lam2 = dd_mul(dd_div(dd_mul_d(s0, l + 1.0), ls1), lam0);  // c2_l lam_{l-1}
    const dd f = dd_div(lam1, dd_mul(ls1, lam2));                      // lam_l / (l S_{l+1} lam_{l+1})
    const auto times = [&](double k) { return dd_mul_d(f, k).hi; };
    out[i] = RcRec{-times((2.0 * l + 1.0) * ll1), times((2.0 * l + 1.0) * (ll1 - mn)),
                   -times((2.0 * l + 1.0) * (ll1 + mn)), lam1.hi};
    lam0 = lam1;
    lam1 = lam2;
  }
}
// p' (negated south of the equator), q' of one degree
__device__ __forceinline__ double2 rec_pq(const RcRec &r, bool north) {
  return north ? make_double2(r.p, r.qn) : make_double2(-r.p, r.qs);
}

__device__ __forceinline__ int exp_bits(double v) { return (int)((__double_as_longlong(v) >> 52) & 0x7FF); }
constexpr int kRenorm = 600;  // rescale step when a carried value passes 2^kRenorm

// 2^E as a double (0 below the subnormal range)
__device__ __forceinline__ double pow2(int E) { return E < -1074 ? 0.0 : ldexp(1.0, E); }

// ---------------------------------------------------------------------------
// l -> t
// ---------------------------------------------------------------------------

template <int NBT>
__global__ void __launch_bounds__(kRcT) k_rc_l2t(const __grid_constant__ RcArgs a) {
  __shared__ RcRec srec[kSeg];
  __shared__ double2 sx[kSeg][NBT];
  const int mt = a.tmlo + blockIdx.x;
  const int amt = mt < 0 ? -mt : mt;
  const int l0 = amt > a.an ? amt : a.an, bl = a.bl, nl = bl - l0;
  const int lst = l0 > a.lmin ? l0 : a.lmin;
  const int t = blockIdx.y * kRcT + threadIdx.x;
  const bool live = t < a.nt;
  const int b0 = blockIdx.z * a.mpc;
  double2 acc[NBT];
#pragma unroll
  for (int b = 0; b < NBT; ++b) acc[b] = make_double2(0.0, 0.0);
  double u = 0.0;
  bool north = true;
  if (live) {
    const double2 q = a.uq[t];
    u = q.x;
    north = q.y != 0.0;
  }
  if (nl > 0 && lst < bl) {
    const int nseg = (nl + kSeg - 1) / kSeg, c0 = (lst - l0) / kSeg;
    const double2 *ck = a.ck + a.coff[blockIdx.x];
    const int *cke = a.ck_e + a.coff[blockIdx.x];
    const RcRec *rec = a.rec + a.roff[blockIdx.x];
    for (int c = c0; c < nseg; ++c) {
      const int lc = l0 + c * kSeg, n = min(kSeg, bl - lc);
      __syncthreads();
      for (int i = threadIdx.x; i < n; i += kRcT) srec[i] = rec[c * kSeg + i];
      __syncthreads();
      for (int i = threadIdx.x; i < kSeg * NBT; i += kRcT) {
        const int kk = i / NBT, col = i % NBT, l = lc + kk, p = col / a.mpc, b = b0 + col % a.mpc;
        double2 v = make_double2(0.0, 0.0);
        if (kk < n && p < a.np && b < a.nb) {
          const RcPart &P = a.part[p];
          const RcM rm = rc_m(a, P, mt);
          if (rm.on && l >= P.lmin) v = rc_coef(a, P, rm.m, b, l, srec[kk].lam);
        }
        sx[kk][col] = v;
      }
      __syncthreads();
      if (!live) continue;
      int E = cke[(int64_t)c * a.nt + t];
      if (E < -1074 - 2 * kRenorm) continue;  // the whole segment is below the double range
      const double2 ab = ck[(int64_t)c * a.nt + t];
      double vp = ab.x, v = ab.y;
      double2 s[NBT];
#pragma unroll
      for (int b = 0; b < NBT; ++b) {
        s[b].x = vp * sx[0][b].x;
        s[b].y = vp * sx[0][b].y;
        if (n > 1) {
          s[b].x = fma(v, sx[1][b].x, s[b].x);
          s[b].y = fma(v, sx[1][b].y, s[b].y);
        }
      }
      for (int i = 1; i + 1 < n; ++i) {
        const double2 k = rec_pq(srec[i], north);
        const double xt = fma(k.x, u, k.y);
        const double vn = fma(xt, v, -vp);
        vp = v;
        v = vn;
        if (exp_bits(v) > 1023 + kRenorm) {  // flush at the old scale, continue at the new one
          const double sc = pow2(E);
#pragma unroll
          for (int b = 0; b < NBT; ++b) {
            acc[b].x = fma(s[b].x, sc, acc[b].x);
            acc[b].y = fma(s[b].y, sc, acc[b].y);
            s[b] = make_double2(0.0, 0.0);
          }
          v = ldexp(v, -kRenorm);
          vp = ldexp(vp, -kRenorm);
          E += kRenorm;
        }
#pragma unroll
        for (int b = 0; b < NBT; ++b) {
          s[b].x = fma(v, sx[i + 1][b].x, s[b].x);
          s[b].y = fma(v, sx[i + 1][b].y, s[b].y);
        }
      }
      const double sc = pow2(E);
#pragma unroll
      for (int b = 0; b < NBT; ++b) {
        acc[b].x = fma(s[b].x, sc, acc[b].x);
        acc[b].y = fma(s[b].y, sc, acc[b].y);
      }
    }
  }
  if (!live) return;
#pragma unroll
  for (int col = 0; col < NBT; ++col) {
    const int p = col / a.mpc, b = b0 + col % a.mpc;
    if (p >= a.np || b >= a.nb) continue;
    const RcM rm = rc_m(a, a.part[p], mt);
    if (!rm.on) continue;
    a.part[p].dst[(int64_t)b * a.ds + (int64_t)t * a.dw + (rm.m - a.d_mlo)] =
        make_double2(acc[col].x * rm.sign, acc[col].y * rm.sign);
  }
}

// ---------------------------------------------------------------------------
// t -> l
// ---------------------------------------------------------------------------

constexpr int kTileLd = kSeg + 1;  // padded row of the d tile

template <int NBT>
size_t rc_t2l_smem() {
  return sizeof(double) * kRcT * kTileLd + sizeof(double2) * kRcT * NBT;
}

// grid: x = table row, y = segment, z = batch chunk.  Threads generate one ring's
// row of the tile each, then contract as (degree li = tid % kSeg, half bh = tid /
// kSeg): with NBT >= 2 each half takes half of the columns over all rings of the
// tile; with NBT = 1 each half takes half of the rings, and the halves add up at
// the end.
template <int NBT>
__global__ void __launch_bounds__(kRcT) k_rc_t2l(const __grid_constant__ RcArgs a) {
  static_assert(NBT == 1 || NBT % 2 == 0, "one column, or two column halves");
  constexpr int NH = NBT == 1 ? 1 : NBT / 2;
  constexpr bool SPLIT_T = NBT == 1;
  extern __shared__ double smem_rc[];
  double *tile = smem_rc;                                   // [kRcT][kTileLd]
  double2 *sg = (double2 *)(smem_rc + kRcT * kTileLd);      // [kRcT][NBT]
  __shared__ RcRec srec[kSeg];
  const int mt = a.tmlo + blockIdx.x, c = blockIdx.y;
  const int amt = mt < 0 ? -mt : mt;
  const int l0 = amt > a.an ? amt : a.an, bl = a.bl, nl = bl - l0;
  const int lst = l0 > a.lmin ? l0 : a.lmin;
  const int nseg = nl > 0 ? (nl + kSeg - 1) / kSeg : 0;
  if (c >= nseg) return;
  const int lc = l0 + c * kSeg, n = min(kSeg, bl - lc);
  if (lc + n <= lst) return;  // every degree of the segment is below lmin: no output
  const int b0 = blockIdx.z * a.mpc;
  const int tid = threadIdx.x;
  const RcRec *rec = a.rec + a.roff[blockIdx.x] + c * kSeg;
  for (int i = tid; i < n; i += kRcT) srec[i] = rec[i];
  const double2 *ck = a.ck + a.coff[blockIdx.x] + (int64_t)c * a.nt;
  const int *cke = a.ck_e + a.coff[blockIdx.x] + (int64_t)c * a.nt;
  const int li = tid % kSeg, bh = tid / kSeg;
  double2 acc[NH];
#pragma unroll
  for (int j = 0; j < NH; ++j) acc[j] = make_double2(0.0, 0.0);
  __syncthreads();
  for (int t0 = 0; t0 < a.nt; t0 += kRcT) {
    const int t = t0 + tid;
    double *row = tile + tid * kTileLd;
    double scale = 0.0;
    int E = kCkZeroExp;
    if (t < a.nt) E = cke[t];
    if (E >= -1074 - 2 * kRenorm) {
      const double2 q = a.uq[t];
      const double u = q.x;
      const bool north = q.y != 0.0;
      const double2 ab = ck[t];
      double vp = ab.x, v = ab.y;
      row[0] = vp;
      if (n > 1) row[1] = v;
      for (int i = 1; i + 1 < n; ++i) {
        const double2 k = rec_pq(srec[i], north);
        const double xt = fma(k.x, u, k.y);
        const double vn = fma(xt, v, -vp);
        vp = v;
        v = vn;
        if (exp_bits(v) > 1023 + kRenorm) {  // keep one scale per row: rescale what is written
          for (int j = 0; j <= i; ++j) row[j] = ldexp(row[j], -kRenorm);
          v = ldexp(v, -kRenorm);
          vp = ldexp(vp, -kRenorm);
          E += kRenorm;
        }
        row[i + 1] = v;
      }
      for (int i = n; i < kSeg; ++i) row[i] = 0.0;
      scale = pow2(E);
    } else {
      for (int i = 0; i < kSeg; ++i) row[i] = 0.0;
    }
#pragma unroll
    for (int col = 0; col < NBT; ++col) {
      const int p = col / a.mpc, b = b0 + col % a.mpc;
      double2 g = make_double2(0.0, 0.0);
      if (t < a.nt && p < a.np && b < a.nb && scale != 0.0) {
        const RcM rm = rc_m(a, a.part[p], mt);
        if (rm.on) g = a.part[p].src[(int64_t)b * a.ss + (int64_t)t * a.sw + (rm.m - a.s_mlo)];
        g = make_double2(g.x * scale, g.y * scale);
      }
      sg[tid * NBT + col] = g;
    }
    __syncthreads();
    const int tl_end = min(kRcT, a.nt - t0);
    const int tl_lo = SPLIT_T ? bh * (kRcT / 2) : 0;
    const int tl_hi = SPLIT_T ? min(tl_end, tl_lo + kRcT / 2) : tl_end;
#pragma unroll 4
    for (int tl = tl_lo; tl < tl_hi; ++tl) {
      const double d = tile[tl * kTileLd + li];
#pragma unroll
      for (int j = 0; j < NH; ++j) {
        const double2 g = sg[tl * NBT + (SPLIT_T ? 0 : bh * NH) + j];
        acc[j].x = fma(d, g.x, acc[j].x);
        acc[j].y = fma(d, g.y, acc[j].y);
      }
    }
    __syncthreads();
  }
  if (SPLIT_T) {  // second half of the rings hands its sums to the first
    double2 *red = sg;  // free after the last tile
    if (bh == 1) red[li] = acc[0];
    __syncthreads();
    if (bh == 1) return;
    acc[0].x += red[li].x;
    acc[0].y += red[li].y;
  }
  const int l = lc + li;
  if (li >= n) return;
  const double lam = srec[li].lam;  // the rescaled recursion's lam_l
#pragma unroll
  for (int j = 0; j < NH; ++j) {
    const int col = (SPLIT_T ? 0 : bh * NH) + j, p = col / a.mpc, b = b0 + col % a.mpc;
    if (p >= a.np || b >= a.nb) continue;
    const RcPart &P = a.part[p];
    const RcM rm = rc_m(a, P, mt);
    if (!rm.on || l < P.lmin) continue;
    const double sl = rm.sign * lam;
    P.dst[(int64_t)b * a.ds + (int64_t)l * l + l + rm.m] =
        cmul_(make_double2(acc[j].x * sl, acc[j].y * sl), weight_of(a, P, l));
  }
}

// ---------------------------------------------------------------------------
// double-float variants (split-precision path on recomputed tables)
//
// The same two contractions with the per-map multiply-adds in double-float
// arithmetic on the FP32 pipe (dfarith.h), which GB300 issues at about 64
// times its FP64 rate.  The three-term recursion stays in FP64 (3 instructions
// per value, shared by all maps): in double-float its cancellation near the
// turning points cost 1e-11 of accuracy (2^-47 against 2^-53 per step over a
// 64-degree segment).  Each value is split into a double-float pair once
// (integer bit operations, dfconv.h) and multiplied into every map's partial
// sum; FP64 is otherwise left to the flush of the partial sums (two adds per
// output value and segment, or per tile of rings for t -> l).  Values are
// carried scaled by 2^-E per ring and segment as in the FP64 kernels, with a
// lower rescaling threshold (2^kRenormDf) so that they stay in the float
// range.  Coefficients (l -> t) and spectra (t -> l) enter as double-float
// scaled by the largest power of two of their block (segment or tile, per
// map).  The sums are renormalised after every term: Dot2 sums (dfarith.h), 12
// instructions a term instead of 15, gather their corrections in single precision and
// came out 3 to 8 times as far off over 32 to 128 terms of one sign (df_mac 4e-15 to
// 8e-15, emulated).
// ---------------------------------------------------------------------------

constexpr int kRenormDf = 60;

__device__ __forceinline__ float2 df_of(double v) {  // |v| within the float range
  float h, l;
  split_scaled(v, 0, h, l);
  return make_float2(h, l);
}
__device__ __forceinline__ float2 df_scale(float2 a, int k) { return make_float2(scale_pow2(a.x, k), scale_pow2(a.y, k)); }
template <int NBT>
__global__ void __launch_bounds__(kRcT) k_rc_l2t_df(const __grid_constant__ RcArgs a) {
  __shared__ RcRec srec[kSeg];
  __shared__ double2 sxd[kSeg][NBT];  // weighted coefficients of the segment
  __shared__ float4 sx[kSeg][NBT];    // the same as double-float, scaled by 2^-sxs[b]
  __shared__ int sxm[NBT], sxs[NBT];
  const int mt = a.tmlo + blockIdx.x;
  const int amt = mt < 0 ? -mt : mt;
  const int l0 = amt > a.an ? amt : a.an, bl = a.bl, nl = bl - l0;
  const int lst = l0 > a.lmin ? l0 : a.lmin;
  const int t = blockIdx.y * kRcT + threadIdx.x;
  const bool live = t < a.nt;
  const int b0 = blockIdx.z * a.mpc;
  double2 acc[NBT];
#pragma unroll
  for (int b = 0; b < NBT; ++b) acc[b] = make_double2(0.0, 0.0);
  double u = 0.0;
  bool north = true;
  if (live) {
    const double2 q = a.uq[t];
    u = q.x;
    north = q.y != 0.0;
  }
  if (nl > 0 && lst < bl) {
    const int nseg = (nl + kSeg - 1) / kSeg, c0 = (lst - l0) / kSeg;
    const double2 *ck = a.ck + a.coff[blockIdx.x];
    const int *cke = a.ck_e + a.coff[blockIdx.x];
    const RcRec *rec = a.rec + a.roff[blockIdx.x];
    for (int c = c0; c < nseg; ++c) {
      const int lc = l0 + c * kSeg, n = min(kSeg, bl - lc);
      __syncthreads();
      for (int i = threadIdx.x; i < n; i += kRcT) srec[i] = rec[c * kSeg + i];
      if (threadIdx.x < NBT) sxm[threadIdx.x] = 0;
      __syncthreads();
      for (int i = threadIdx.x; i < kSeg * NBT; i += kRcT) {
        const int kk = i / NBT, b = i % NBT, l = lc + kk, p = b / a.mpc, bm = b0 + b % a.mpc;
        double2 v = make_double2(0.0, 0.0);
        if (kk < n && p < a.np && bm < a.nb) {
          const RcPart &P = a.part[p];
          const RcM rm = rc_m(a, P, mt);
          if (rm.on && l >= P.lmin) v = rc_coef(a, P, rm.m, bm, l, srec[kk].lam);
        }
        sxd[kk][b] = v;
        atomicMax(&sxm[b], max(exp_bits(v.x), exp_bits(v.y)));
      }
      __syncthreads();
      if (threadIdx.x < NBT) sxs[threadIdx.x] = block_scale(sxm[threadIdx.x]);
      __syncthreads();
      for (int i = threadIdx.x; i < kSeg * NBT; i += kRcT) {
        const int kk = i / NBT, b = i % NBT;
        sx[kk][b] = dc_split(sxd[kk][b], sxs[b]);
      }
      __syncthreads();
      if (!live) continue;
      int E = cke[(int64_t)c * a.nt + t];
      if (E < -1074 - 2 * kRenorm) continue;  // the whole segment is below the double range
      const double2 ab = ck[(int64_t)c * a.nt + t];
      double vp = ab.x, v = ab.y;
      float4 sum[NBT];
      {
        const float2 dvp = df_of(vp), dv = df_of(v);
#pragma unroll
        for (int b = 0; b < NBT; ++b) {
          sum[b] = make_float4(0.f, 0.f, 0.f, 0.f);
          df_mac(sum[b], dvp, sx[0][b]);
          if (n > 1) df_mac(sum[b], dv, sx[1][b]);
        }
      }
      for (int i = 1; i + 1 < n; ++i) {
        const double2 k = rec_pq(srec[i], north);
        const double xt = fma(k.x, u, k.y);
        const double vn = fma(xt, v, -vp);  // rescaled recursion
        vp = v;
        v = vn;
        if (exp_bits(v) > 1023 + kRenormDf) {  // flush at the old scale, continue at the new one
#pragma unroll
          for (int b = 0; b < NBT; ++b) {
            const double2 f = dc_to(sum[b], E + sxs[b]);
            acc[b].x += f.x;
            acc[b].y += f.y;
            sum[b] = make_float4(0.f, 0.f, 0.f, 0.f);
          }
          v = ldexp(v, -kRenormDf);
          vp = ldexp(vp, -kRenormDf);
          E += kRenormDf;
        }
        const float2 dv = df_of(v);
#pragma unroll
        for (int b = 0; b < NBT; ++b) df_mac(sum[b], dv, sx[i + 1][b]);
      }
#pragma unroll
      for (int b = 0; b < NBT; ++b) {
        const double2 f = dc_to(sum[b], E + sxs[b]);
        acc[b].x += f.x;
        acc[b].y += f.y;
      }
    }
  }
  if (!live) return;
#pragma unroll
  for (int col = 0; col < NBT; ++col) {
    const int p = col / a.mpc, b = b0 + col % a.mpc;
    if (p >= a.np || b >= a.nb) continue;
    const RcM rm = rc_m(a, a.part[p], mt);
    if (!rm.on) continue;
    a.part[p].dst[(int64_t)b * a.ds + (int64_t)t * a.dw + (rm.m - a.d_mlo)] =
        make_double2(acc[col].x * rm.sign, acc[col].y * rm.sign);
  }
}

template <int NBT>
size_t rc_t2l_df_smem() {
  return sizeof(float2) * kRcT * kTileLd + sizeof(float4) * kRcT * NBT;
}

// t -> l in double-float: the tile rows (one ring each, scaled by 2^-E_t)
// as double-float pairs; the spectra enter scaled by 2^(E_t - es[b]) with es[b]
// the largest exponent of spectrum times ring scale over the tile, so the
// sums over the tile's rings share one power of two and are flushed to FP64
// once per tile.
template <int NBT>
__global__ void __launch_bounds__(kRcT) k_rc_t2l_df(const __grid_constant__ RcArgs a) {
  static_assert(NBT == 1 || NBT % 2 == 0, "one column, or two column halves");
  constexpr int NH = NBT == 1 ? 1 : NBT / 2;
  constexpr bool SPLIT_T = NBT == 1;
  extern __shared__ float2 smem_df[];
  float2 *tile = smem_df;                                  // [kRcT][kTileLd]
  float4 *sg = (float4 *)(smem_df + kRcT * kTileLd);       // [kRcT][NBT]
  __shared__ RcRec srec[kSeg];
  __shared__ int sgm[NBT];
  const int mt = a.tmlo + blockIdx.x, c = blockIdx.y;
  const int amt = mt < 0 ? -mt : mt;
  const int l0 = amt > a.an ? amt : a.an, bl = a.bl, nl = bl - l0;
  const int lst = l0 > a.lmin ? l0 : a.lmin;
  const int nseg = nl > 0 ? (nl + kSeg - 1) / kSeg : 0;
  if (c >= nseg) return;
  const int lc = l0 + c * kSeg, n = min(kSeg, bl - lc);
  if (lc + n <= lst) return;  // every degree of the segment is below lmin: no output
  const int b0 = blockIdx.z * a.mpc;
  const int tid = threadIdx.x;
  const RcRec *rec = a.rec + a.roff[blockIdx.x] + c * kSeg;
  for (int i = tid; i < n; i += kRcT) srec[i] = rec[i];
  __syncthreads();
  const double2 *ck = a.ck + a.coff[blockIdx.x] + (int64_t)c * a.nt;
  const int *cke = a.ck_e + a.coff[blockIdx.x] + (int64_t)c * a.nt;
  const int li = tid % kSeg, bh = tid / kSeg;
  double2 acc[NH];
#pragma unroll
  for (int j = 0; j < NH; ++j) acc[j] = make_double2(0.0, 0.0);
  for (int t0 = 0; t0 < a.nt; t0 += kRcT) {
    const int t = t0 + tid;
    float2 *row = tile + tid * kTileLd;
    int E = kCkZeroExp;
    if (t < a.nt) E = cke[t];
    const bool on = E >= -1074 - 2 * kRenorm;
    if (on) {
      const double2 q = a.uq[t];
      const double u = q.x;
      const bool north = q.y != 0.0;
      const double2 ab = ck[t];
      double vp = ab.x, v = ab.y;
      row[0] = df_of(vp);
      if (n > 1) row[1] = df_of(v);
      for (int i = 1; i + 1 < n; ++i) {
        const double2 k = rec_pq(srec[i], north);
        const double xt = fma(k.x, u, k.y);
        const double vn = fma(xt, v, -vp);  // rescaled recursion
        vp = v;
        v = vn;
        if (exp_bits(v) > 1023 + kRenormDf) {  // keep one scale per row: rescale what is written
          for (int j = 0; j <= i; ++j) row[j] = df_scale(row[j], -kRenormDf);
          v = ldexp(v, -kRenormDf);
          vp = ldexp(vp, -kRenormDf);
          E += kRenormDf;
        }
        row[i + 1] = df_of(v);
      }
      for (int i = n; i < kSeg; ++i) row[i] = make_float2(0.f, 0.f);
    } else {
      for (int i = 0; i < kSeg; ++i) row[i] = make_float2(0.f, 0.f);
    }
    // the spectra of this ring times 2^E, and the tile's largest exponent per map
    if (tid < NBT) sgm[tid] = -(1 << 30);
    __syncthreads();
    double2 g[NBT];
#pragma unroll
    for (int b = 0; b < NBT; ++b) {
      g[b] = make_double2(0.0, 0.0);
      const int p = b / a.mpc, bm = b0 + b % a.mpc;
      if (on && p < a.np && bm < a.nb) {
        const RcM rm = rc_m(a, a.part[p], mt);
        if (rm.on) g[b] = a.part[p].src[(int64_t)bm * a.ss + (int64_t)t * a.sw + (rm.m - a.s_mlo)];
        const int ex = max(exp_bits(g[b].x), exp_bits(g[b].y));
        if (ex > 0) atomicMax(&sgm[b], ex + E);
      }
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < NBT; ++b) {
      const int es = sgm[b] > -(1 << 29) ? block_scale(sgm[b]) : 0;
      sg[tid * NBT + b] = on ? dc_split(g[b], es - E) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    const int tl_end = min(kRcT, a.nt - t0);
    const int tl_lo = SPLIT_T ? bh * (kRcT / 2) : 0;
    const int tl_hi = SPLIT_T ? min(tl_end, tl_lo + kRcT / 2) : tl_end;
    float4 sum[NH];
#pragma unroll
    for (int j = 0; j < NH; ++j) sum[j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int tl = tl_lo; tl < tl_hi; ++tl) {
      const float2 d = tile[tl * kTileLd + li];
#pragma unroll
      for (int j = 0; j < NH; ++j) df_mac(sum[j], d, sg[tl * NBT + (SPLIT_T ? 0 : bh * NH) + j]);
    }
#pragma unroll
    for (int j = 0; j < NH; ++j) {
      const int b = (SPLIT_T ? 0 : bh * NH) + j;
      const int es = sgm[b] > -(1 << 29) ? block_scale(sgm[b]) : 0;
      const double2 f = dc_to(sum[j], es);
      acc[j].x += f.x;
      acc[j].y += f.y;
    }
    __syncthreads();
  }
  if (SPLIT_T) {  // second half of the rings hands its sums to the first
    double2 *red = (double2 *)sg;  // free after the last tile
    if (bh == 1) red[li] = acc[0];
    __syncthreads();
    if (bh == 1) return;
    acc[0].x += red[li].x;
    acc[0].y += red[li].y;
  }
  const int l = lc + li;
  if (li >= n) return;
  const double lam = srec[li].lam;  // the rescaled recursion's lam_l
#pragma unroll
  for (int j = 0; j < NH; ++j) {
    const int col = (SPLIT_T ? 0 : bh * NH) + j, p = col / a.mpc, b = b0 + col % a.mpc;
    if (p >= a.np || b >= a.nb) continue;
    const RcPart &P = a.part[p];
    const RcM rm = rc_m(a, P, mt);
    if (!rm.on || l < P.lmin) continue;
    const double sl = rm.sign * lam;
    P.dst[(int64_t)b * a.ds + (int64_t)l * l + l + rm.m] =
        cmul_(make_double2(acc[j].x * sl, acc[j].y * sl), weight_of(a, P, l));
  }
}

// ---------------------------------------------------------------------------
// quadrature operator on ring spectra
// ---------------------------------------------------------------------------

// out[b][i][m - o_mlo] = sum_k A_m[i][k] in[b][k][m - i_mlo], i, k < nt, for the
// m in [mlo, mhi] with (m + an) even (parity 0, W_+) or odd (parity 1, W_-);
// A = W (trans = 0) or W^T (trans = 1).  Columns are the (map, m) pairs of the
// parity, each complex column two real ones.  64 x 64 output tile per CTA.
constexpr int AW_T = 64, AW_K = 16;
// problems of one launch (blockIdx.z = parity + 2 problem), strides in common
constexpr int kWItems = kMaxParts;
struct WItems {
  int n;
  const double2 *in[kWItems];
  double2 *out[kWItems];
  int mlo[kWItems], mhi[kWItems];
};
__global__ void __launch_bounds__(256) k_apply_w(const double *__restrict__ Wp, const double *__restrict__ Wm, int trans,
                                          int nt, int an, const __grid_constant__ WItems items, int64_t is, int iw,
                                          int i_mlo, int64_t os, int ow, int o_mlo, int nb) {
  const int par = blockIdx.z & 1, item = blockIdx.z >> 1;
  const int mlo = items.mlo[item], mhi = items.mhi[item];
  const double2 *__restrict__ in = items.in[item];
  double2 *__restrict__ out = items.out[item];
  const int m_first = ((mlo + an) & 1) == par ? mlo : mlo + 1;
  if (m_first > mhi) return;
  const int nmp = (mhi - m_first) / 2 + 1;  // m's of this parity
  const int ncols = 2 * nmp * nb;           // real columns
  const int row0 = blockIdx.y * AW_T, col0 = blockIdx.x * AW_T;
  if (row0 >= nt || col0 >= ncols) return;
  const double *W = par == 0 ? Wp : Wm;
  __shared__ double sA[AW_K][AW_T + 1];  // [k][row]
  __shared__ double sB[AW_K][AW_T + 1];  // [k][col]
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  double acc[4][4] = {};
  for (int k0 = 0; k0 < nt; k0 += AW_K) {
    for (int i = threadIdx.x; i < AW_K * AW_T; i += 256) {
      // W rows are contiguous in k (trans = 0) or in the row index (trans = 1)
      const int kk = trans ? i / AW_T : i % AW_K, cc = trans ? i % AW_T : i / AW_K;
      const int k = k0 + kk;
      double av = 0.0;
      if (k < nt && row0 + cc < nt)
        av = trans ? W[(int64_t)k * nt + row0 + cc] : W[(int64_t)(row0 + cc) * nt + k];
      sA[kk][cc] = av;
    }
    for (int i = threadIdx.x; i < AW_K * AW_T; i += 256) {
      const int kk = i / AW_T, cc = i % AW_T;
      const int k = k0 + kk, col = col0 + cc;
      double bv = 0.0;
      if (k < nt && col < ncols) {
        const int pair = col >> 1, im = col & 1;
        const int b = pair / nmp, m = m_first + 2 * (pair % nmp);
        const double2 z = in[(int64_t)b * is + (int64_t)k * iw + (m - i_mlo)];
        bv = im ? z.y : z.x;
      }
      sB[kk][cc] = bv;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < AW_K; ++kk) {
      double x[4], y[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = sA[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) y[j] = sB[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma(x[i], y[j], acc[i][j]);
    }
    __syncthreads();
  }
  // columns tx*4 .. tx*4+3 are two complex columns (re, im pairs start even)
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rr = row0 + ty * 4 + i;
    if (rr >= nt) continue;
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
      const int col = col0 + tx * 4 + j;
      if (col >= ncols) continue;
      const int pair = col >> 1;
      const int b = pair / nmp, m = m_first + 2 * (pair % nmp);
      out[(int64_t)b * os + (int64_t)rr * ow + (m - o_mlo)] = make_double2(acc[i][j], acc[i][j + 1]);
    }
  }
}

// The same operator in double-float (split-precision path).  Per K-slab of
// AWD_K: W values as double-float pairs (unscaled: the operator's entries sit
// well inside the float range), each real column's slab as double-float
// scaled by its largest power of two; the slab's partial sums are flushed
// into FP64 accumulators with that power of two.  15 FP32 instructions per
// multiply-add against one FP64 instruction at 1/64 of the rate.
constexpr int AWD_K = 32;
__global__ void __launch_bounds__(256) k_apply_w_df(const double *__restrict__ Wp, const double *__restrict__ Wm, int trans,
                                          int nt, int an, const __grid_constant__ WItems items, int64_t is, int iw,
                                          int i_mlo, int64_t os, int ow, int o_mlo, int nb) {
  const int par = blockIdx.z & 1, item = blockIdx.z >> 1;
  const int mlo = items.mlo[item], mhi = items.mhi[item];
  const double2 *__restrict__ in = items.in[item];
  double2 *__restrict__ out = items.out[item];
  const int m_first = ((mlo + an) & 1) == par ? mlo : mlo + 1;
  if (m_first > mhi) return;
  const int nmp = (mhi - m_first) / 2 + 1;  // m's of this parity
  const int ncols = 2 * nmp * nb;           // real columns
  const int row0 = blockIdx.y * AW_T, col0 = blockIdx.x * AW_T;
  if (row0 >= nt || col0 >= ncols) return;
  const double *W = par == 0 ? Wp : Wm;
  __shared__ float2 sA[AWD_K][AW_T + 1];  // [k][row]
  // [k][col]: first the FP64 values, then (in place, each thread converting the
  // entries it stored) their double-float pairs scaled by 2^-sBe[col]
  __shared__ float2 sB[AWD_K][AW_T + 1];
  __shared__ int sBm[AW_T], sBe[AW_T];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  double acc[4][4] = {};
  for (int k0 = 0; k0 < nt; k0 += AWD_K) {
    if (threadIdx.x < AW_T) sBm[threadIdx.x] = 0;
    for (int i = threadIdx.x; i < AWD_K * AW_T; i += 256) {
      const int kk = trans ? i / AW_T : i % AWD_K, cc = trans ? i % AW_T : i / AWD_K;
      const int k = k0 + kk;
      double av = 0.0;
      if (k < nt && row0 + cc < nt)
        av = trans ? W[(int64_t)k * nt + row0 + cc] : W[(int64_t)(row0 + cc) * nt + k];
      sA[kk][cc] = df_of(av);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < AWD_K * AW_T; i += 256) {
      const int kk = i / AW_T, cc = i % AW_T;
      const int k = k0 + kk, col = col0 + cc;
      double bv = 0.0;
      if (k < nt && col < ncols) {
        const int pair = col >> 1, im = col & 1;
        const int b = pair / nmp, m = m_first + 2 * (pair % nmp);
        const double2 z = in[(int64_t)b * is + (int64_t)k * iw + (m - i_mlo)];
        bv = im ? z.y : z.x;
      }
      *reinterpret_cast<double *>(&sB[kk][cc]) = bv;
      atomicMax(&sBm[cc], exp_bits(bv));
    }
    __syncthreads();
    if (threadIdx.x < AW_T) sBe[threadIdx.x] = block_scale(sBm[threadIdx.x]);
    __syncthreads();
    for (int i = threadIdx.x; i < AWD_K * AW_T; i += 256) {
      const int kk = i / AW_T, cc = i % AW_T;
      sB[kk][cc] = df_split(*reinterpret_cast<const double *>(&sB[kk][cc]), sBe[cc]);
    }
    __syncthreads();
    float2 sum[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[i][j] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int kk = 0; kk < AWD_K; ++kk) {
      float2 x[4], y[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = sA[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) y[j] = sB[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) sum[i][j] = df_add_norm(sum[i][j], df_mul(x[i], y[j]));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int e = sBe[tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i][j] += join_scaled(sum[i][j].x, sum[i][j].y, e);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rr = row0 + ty * 4 + i;
    if (rr >= nt) continue;
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
      const int col = col0 + tx * 4 + j;
      if (col >= ncols) continue;
      const int pair = col >> 1;
      const int b = pair / nmp, m = m_first + 2 * (pair % nmp);
      out[(int64_t)b * os + (int64_t)rr * ow + (m - o_mlo)] = make_double2(acc[i][j], acc[i][j + 1]);
    }
  }
}

RcArgs rc_args(const WignerTable &tb, double wscale, bool wconj, int nb) {
  RcArgs a{};
  a.bl = tb.bl;
  a.nt = tb.nt;
  a.an = tb.an;
  a.tmlo = tb.mlo;
  a.coff = tb.d_coff;
  a.ck = tb.ck;
  a.ck_e = tb.ck_e;
  a.uq = tb.uq;
  a.rec = tb.rec;
  a.roff = tb.d_roff;
  a.wscale = wscale;
  a.wconj = wconj ? 1 : 0;
  a.nb = nb;
  a.lmin = tb.bl;
  return a;
}

// The parts of one problem: n > 0 reads table row m, n < 0 row -m, n = 0 both.
template <class A>
std::vector<RcPart> parts_of(const A &p, const double2 *src, double2 *dst) {
  RcPart P{};
  P.mlo = p.mlo;
  P.mhi = p.mhi;
  P.lmin = p.lmin;
  P.w = p.w;
  P.src = src;
  P.dst = dst;
  P.neg = p.n < 0 ? 1 : 0;
  if (p.n != 0 || p.mlo >= 0) return {P};
  RcPart N = P;
  P.mlo = 0;
  N.mhi = std::min(p.mhi, -1);
  N.neg = 1;
  return {P, N};
}

// algorithmic work of one launch, as the stored path counts it (one complex x
// real MAC per (l, m, t) per map) plus the recursion (3 FP64 per value)
void rc_work(const WignerTable &tb, int mlo, int mhi, int lmin, int nb, double *flops, double *bytes) {
  double macs = 0;
  for (int m = mlo; m <= mhi; ++m) {
    const int am = m < 0 ? -m : m, l0 = std::max(am, tb.an), lst = std::max(l0, lmin);
    if (lst < tb.bl) macs += (double)(tb.bl - lst) * tb.nt;
  }
  *flops = 4.0 * macs * nb;
  *bytes = 16.0 * nb * (double)(mhi - mlo + 1) * (tb.nt + tb.bl);
}

void apply_w(const WignerTable &tb, bool trans, const WItems &items, int64_t is, int iw, int i_mlo, int64_t os, int ow,
             int o_mlo, int nb, cudaStream_t st) {
  int nm = 0, nmtot = 0;
  for (int i = 0; i < items.n; ++i) {
    nm = std::max(nm, items.mhi[i] - items.mlo[i] + 1);
    nmtot += items.mhi[i] - items.mlo[i] + 1;
  }
  const int ncols = 2 * ((nm + 1) / 2) * nb;
  KTimer kt(KC_QUAD, st, 2.0 * tb.nt * (double)tb.nt * nmtot * nb * 2.0, 16.0 * nb * (double)nmtot * tb.nt * 2.0);
  dim3 grid(ceil_div(ncols, AW_T), ceil_div(tb.nt, AW_T), 2 * items.n);
  if (t_precision == 1)  // split precision: double-float multiply-adds
    k_apply_w_df<<<grid, 256, 0, st>>>(tb.W[0], tb.W[1], trans ? 1 : 0, tb.nt, tb.an, items, is, iw, i_mlo, os, ow,
                                       o_mlo, nb);
  else
    k_apply_w<<<grid, 256, 0, st>>>(tb.W[0], tb.W[1], trans ? 1 : 0, tb.nt, tb.an, items, is, iw, i_mlo, os, ow,
                                    o_mlo, nb);
  S2G_LAUNCHED();
}

template <int NBT>
void launch_l2t(const RcArgs &a, int nm, cudaStream_t st) {
  dim3 grid(nm, ceil_div(a.nt, kRcT), ceil_div(a.nb, a.mpc));
  k_rc_l2t<NBT><<<grid, kRcT, 0, st>>>(a);
  S2G_LAUNCHED();
}

template <int NBT>
void launch_t2l(const RcArgs &a, int nm, int maxseg, cudaStream_t st) {
  const size_t smem = rc_t2l_smem<NBT>();
  static const bool attr = [smem] {  // once per instantiation (thread-safe static initialisation)
    S2G_CUDA(cudaFuncSetAttribute(k_rc_t2l<NBT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return true;
  }();
  (void)attr;
  dim3 grid(nm, maxseg, ceil_div(a.nb, a.mpc));
  k_rc_t2l<NBT><<<grid, kRcT, smem, st>>>(a);
  S2G_LAUNCHED();
}

template <int NBT>
void launch_l2t_df(const RcArgs &a, int nm, cudaStream_t st) {
  dim3 grid(nm, ceil_div(a.nt, kRcT), ceil_div(a.nb, a.mpc));
  k_rc_l2t_df<NBT><<<grid, kRcT, 0, st>>>(a);
  S2G_LAUNCHED();
}

template <int NBT>
void launch_t2l_df(const RcArgs &a, int nm, int maxseg, cudaStream_t st) {
  const size_t smem = rc_t2l_df_smem<NBT>();
  static const bool attr = [smem] {  // once per instantiation (thread-safe static initialisation)
    S2G_CUDA(cudaFuncSetAttribute(k_rc_t2l_df<NBT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return true;
  }();
  (void)attr;
  dim3 grid(nm, maxseg, ceil_div(a.nb, a.mpc));
  k_rc_t2l_df<NBT><<<grid, kRcT, smem, st>>>(a);
  S2G_LAUNCHED();
}

}  // namespace

namespace {
void run_l2t(const RcArgs &a, int nm, int nbt, cudaStream_t st) {
  const bool df = t_precision == 1;  // split precision: the double-float kernels (same results to about 1e-13)
  switch (nbt) {
    case 8: df ? launch_l2t_df<8>(a, nm, st) : launch_l2t<8>(a, nm, st); break;
    case 4: df ? launch_l2t_df<4>(a, nm, st) : launch_l2t<4>(a, nm, st); break;
    case 2: df ? launch_l2t_df<2>(a, nm, st) : launch_l2t<2>(a, nm, st); break;
    default: df ? launch_l2t_df<1>(a, nm, st) : launch_l2t<1>(a, nm, st); break;
  }
}
void run_t2l(const RcArgs &a, int nm, int maxseg, int nbt, cudaStream_t st) {
  const bool df = t_precision == 1;
  switch (nbt) {
    case 16: df ? launch_t2l_df<16>(a, nm, maxseg, st) : launch_t2l<16>(a, nm, maxseg, st); break;
    case 8: df ? launch_t2l_df<8>(a, nm, maxseg, st) : launch_t2l<8>(a, nm, maxseg, st); break;
    case 4: df ? launch_t2l_df<4>(a, nm, maxseg, st) : launch_t2l<4>(a, nm, maxseg, st); break;
    case 2: df ? launch_t2l_df<2>(a, nm, maxseg, st) : launch_t2l<2>(a, nm, maxseg, st); break;
    default: df ? launch_t2l_df<1>(a, nm, maxseg, st) : launch_t2l<1>(a, nm, maxseg, st); break;
  }
}

// Launches over up to kRcParts parts each.  Columns per CTA (parts x maps): the
// largest power of two up to maxcols that parts and batch fill, or the autotuned
// choice of maps per CTA.
// mincols: a batch takes at least so many (the t -> l kernel sums one column in
// another order than several).
template <class RUN>
void launch_parts(RcArgs a, const std::vector<RcPart> &parts, const WignerTable &tb, int family, int mincols,
                  int maxcols, cudaStream_t st, RUN &&run) {
  for (size_t i = 0; i < parts.size(); i += kRcParts) {
    a.np = (int)std::min<size_t>(kRcParts, parts.size() - i);
    a.lmin = tb.bl;
    double fl = 0, by = 0;
    for (int p = 0; p < a.np; ++p) {
      a.part[p] = parts[i + p];
      a.lmin = std::min(a.lmin, a.part[p].lmin);
      if (timing_enabled()) {
        double f1 = 0, b1 = 0;
        rc_work(tb, a.part[p].mlo, a.part[p].mhi, a.part[p].lmin, a.nb, &f1, &b1);
        fl += f1;
        by += b1;
      }
    }
    const int np2 = a.np > 2 ? 4 : a.np;
    const int c0 = a.nb > 1 && np2 < mincols ? 1 : 0;  // log2 of the fewest maps per CTA
    int ncand = 1;
    while ((2 << (c0 + ncand - 1)) <= a.nb && np2 << (c0 + ncand) <= maxcols) ++ncand;
    const auto go = [&](int c) {
      a.mpc = 1 << (c0 + c);
      run(a, np2 << (c0 + c));
    };
    const int c = tuned(family, tune_bucket(tb.bl), tune_bucket(a.nb), (t_precision == 1 ? 1 : 0) + 2 * (np2 / 2),
                        ncand, ncand - 1, st, go);
    KTimer kt(KC_RECOMPUTE, st, fl, by);
    go(c);
  }
}

bool same_form(const L2T &p, const L2T &q) {
  return p.tb == q.tb && p.use_q == q.use_q && p.xs == q.xs && p.x_half == q.x_half && p.wscale == q.wscale &&
         p.wconj == q.wconj && p.os == q.os && p.ow == q.ow && p.omlo == q.omlo && p.nb == q.nb;
}
bool same_form(const T2L &p, const T2L &q) {
  return p.tb == q.tb && p.use_q == q.use_q && p.is == q.is && p.iw == q.iw && p.imlo == q.imlo &&
         p.wscale == q.wscale && p.wconj == q.wconj && p.ys == q.ys && p.nb == q.nb;
}

// Quadrature of n problems, as many of one m range as a pass takes.
// FP64 mode: the FP64 kernel.  Eight slices on the tensor cores are faster, but the
// operator's rows are peaked (the largest entry, on the diagonal, stands far above the
// rest), and slices err relative to it: forward transforms of white maps at L = 512 and
// 700 came out 1.2 and 1.3 times as far off (at L = 128 1.07), while on the Wigner
// tables, whose rows oscillate at one level, slices are the more accurate.
// Split precision: on the tensor cores from band-limit 513; up to 512 by the
// double-float kernel.  That one takes twice the time alone (32 maps of 64 <= L <= 320,
// one by one: 15.7 against 8.3 ms), but it shares the GPU with the other maps of a
// multi-map call, which the tensor-core kernel's shared memory does not (20.9 against
// 21.8 ms).  The rule looks at the band-limit only: calls of one map or one batch take
// it too.
constexpr int kQuadDfMaxBl = 512;
template <class A, class F>
void quadrature(const A *p, int n, bool trans, F &&io, int64_t is, int iw, int i_mlo, int64_t os, int ow, int o_mlo,
                cudaStream_t st) {
  const WignerTable &tb = *p[0].tb;
  for (int i0 = 0; i0 < n;) {
    QuadIO q[kMaxParts];
    int k = 0;
    for (; k < kMaxParts && i0 + k < n && p[i0 + k].mlo == p[i0].mlo && p[i0 + k].mhi == p[i0].mhi; ++k)
      io(i0 + k, &q[k].in, &q[k].out);
    const bool tensor = t_precision == 1 && tb.bl > kQuadDfMaxBl;
    if (!tensor || !quadrature_mixed(tb, trans, q, k, p[i0].mlo, p[i0].mhi, is, iw, i_mlo, os, ow, o_mlo, p[0].nb, st)) {
      WItems w{};
      w.n = k;
      for (int i = 0; i < k; ++i) {
        w.in[i] = q[i].in;
        w.out[i] = q[i].out;
        w.mlo[i] = p[i0].mlo;
        w.mhi[i] = p[i0].mhi;
      }
      apply_w(tb, trans, w, is, iw, i_mlo, os, ow, o_mlo, p[0].nb, st);
    }
    i0 += k;
  }
}

void l2t_rc(const L2T *v, int n, cudaStream_t st) {
  const L2T &p = v[0];
  const WignerTable &tb = *p.tb;
  RcArgs a = rc_args(tb, p.wscale, p.wconj, p.nb);
  a.ss = p.xs;
  a.x_half = p.x_half ? 1 : 0;
  a.dw = p.ow;
  a.d_mlo = p.omlo;
  // Q^T x = W^T (D x): D x into scratch of the output's layout, then W^T
  Scratch S(st);
  const int64_t one = (int64_t)p.nb * tb.nt * p.ow;
  double2 *tmp = p.use_q ? S.get<double2>(one * n) : nullptr;
  a.ds = p.use_q ? (int64_t)tb.nt * p.ow : p.os;
  std::vector<RcPart> parts;
  for (int i = 0; i < n; ++i)
    for (const RcPart &q : parts_of(v[i], v[i].x, p.use_q ? tmp + i * one : v[i].out)) parts.push_back(q);
  launch_parts(a, parts, tb, TF_RC_L2T, 1, 8, st, [&](const RcArgs &x, int nbt) { run_l2t(x, tb.nm, nbt, st); });
  if (p.use_q) {
    quadrature(v, n, true, [&](int i, const double2 **in, double2 **out) {
      *in = tmp + i * one;
      *out = v[i].out;
    }, a.ds, p.ow, p.omlo, p.os, p.ow, p.omlo, st);
  }
}

void t2l_rc(const T2L *v, int n, cudaStream_t st) {
  const T2L &p = v[0];
  const WignerTable &tb = *p.tb;
  RcArgs a = rc_args(tb, p.wscale, p.wconj, p.nb);
  // Q in = D^T (W in): the quadrature on the spectra first
  Scratch S(st);
  double2 *tmp = nullptr;
  const int64_t one = (int64_t)p.nb * tb.nt * p.iw;
  a.ss = p.use_q ? (int64_t)tb.nt * p.iw : p.is;
  if (p.use_q) {
    tmp = S.get<double2>(one * n);
    quadrature(v, n, false, [&](int i, const double2 **in, double2 **out) {
      *in = v[i].in;
      *out = tmp + i * one;
    }, p.is, p.iw, p.imlo, a.ss, p.iw, p.imlo, st);
  }
  a.sw = p.iw;
  a.s_mlo = p.imlo;
  a.ds = p.ys;
  int maxseg = 1;
  for (int m = 0; m < tb.bl; ++m) maxseg = std::max(maxseg, tb.nseg(m));
  std::vector<RcPart> parts;
  for (int i = 0; i < n; ++i)
    for (const RcPart &q : parts_of(v[i], p.use_q ? tmp + i * one : v[i].in, v[i].y)) parts.push_back(q);
  launch_parts(a, parts, tb, TF_RC_T2L, 2, 16, st,
               [&](const RcArgs &x, int nbt) { run_t2l(x, tb.nm, maxseg, nbt, st); });
}

// problems of one form in shared launches, in order
template <class A, class F>
void by_form(const A *p, int n, F &&f) {
  std::vector<A> same;
  for (int i = 0; i < n; ++i) {
    if (!same.empty() && !same_form(same[0], p[i])) {
      f(same.data(), (int)same.size());
      same.clear();
    }
    if (p[i].nb > 0 && p[i].mhi >= p[i].mlo) same.push_back(p[i]);
  }
  if (!same.empty()) f(same.data(), (int)same.size());
}
}  // namespace

RcRec *build_rec(int bl, int an, int mlo, int nm, const int64_t *d_roff, int64_t n) {
  RcRec *rec = nullptr;
  S2G_CUDA(device_malloc((void **)&rec, sizeof(RcRec) * (size_t)(n > 0 ? n : 1)));
  const int maxseg = ceil_div(bl, kSeg);
  k_rc_rec<<<ceil_div((int64_t)nm * maxseg, 128), 128>>>(rec, d_roff, bl, an, mlo, nm, maxseg);
  S2G_LAUNCHED();
  return rec;
}

void contract_l2t_rc(const L2T *p, int n, cudaStream_t st) {
  by_form(p, n, [&](const L2T *v, int k) { l2t_rc(v, k, st); });
}
void contract_t2l_rc(const T2L *p, int n, cudaStream_t st) {
  by_form(p, n, [&](const T2L *v, int k) { t2l_rc(v, k, st); });
}

}  // namespace s2g
