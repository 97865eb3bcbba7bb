// Contractions on tcgen05 by digit slicing (see mixed.h for the number format).
//
// Two forms: 7 slices (28 digit products, the split-precision mode's forward
// contractions) and 8 slices (36 products, FP64 results: the FP64 mode, and the
// adjoint contractions of both modes).
//
// Layout in HBM
//   Sliced table, one per (band-limit, |n|, kind: D or Q, read along or across):
//     for each table m, for each 128-row tile rt, for each 64-wide K-chunk kc,
//     for each digit slice j, an 8 KB block [4 K groups][128 rows][16 bytes] of
//     digits + 64; rows and K are zero-padded to the block.  One byte per digit:
//     7 or 8 bytes per table entry, half of what bf16 panels take, so that the
//     table stream (the bound of small batches) and the L2-to-SM traffic (of
//     large ones) halve.  The eighth slice has an array of its own (it is the
//     remainder of the first seven, which both forms share).  Row exponents eA
//     (int16) per (m, row).
//   Sliced coefficients, per call and per problem m: for each kc one panel
//     [S slices x NC columns][64 bf16], column exponents eX (int32) per (m,
//     column).
//
// Kernel k_contract_mx<NC, S>: persistent, one CTA per SM; NC real
// coefficient columns (16, 32 or 64) per table pass.
//   warp 0    producer: cp.async.bulk of digit blocks into a ring of 8 KB stages
//             and of coefficient panels into a ring of 2 or 3 (S slices x NC
//             columns x 64 K).
//   converter warps (5; 2 at NC = 64): digit block -> 16 KB panel [128 rows][64
//             bf16] in the 128-byte-swizzled K-major image that tcgen05 reads,
//             in a ring of 16 KB stages: a byte permute puts digit + 64 under the
//             exponent of 128 (bf16 has 8 significant bits), one packed
//             subtraction of 192 leaves the digit, 2 instructions per 2 digits.
//   warp 1    MMA issuer: per K-chunk and digit slice j, one 128 x N x 64
//             product (tcgen05.mma of K=16, N <= 256 each) of table slice j
//             against the first S-j coefficient slices, written to the
//             accumulator columns of classes j..S-1 (N = NC (S-j)); two TMEM
//             accumulators alternate between tiles (one at NC = 64).
//   epilogue warps (NC / 4): one per TMEM lane quarter and 16 columns:
//             tcgen05.ld of the S class accumulators, combine (double-float
//             for 7, integers for 8), row/column exponents, sign, per-l
//             weight, store; the accumulator is released as soon as its values
//             are in registers.
// Measured (2 maps at L = 1024, N = 4, FP64, 16 columns): 13.0 ms against 15.8 with
// bf16 panels in HBM; 32 maps, split precision, 64 columns: 31.1 against 33.5.
// With a quarter of the MMAs the 16-column launches take 24 % less, without the
// conversion's stores 10 %, without the combination 4 %: no single unit paces
// them (one map at L = 512, bl = 512: DRAM 51 % busy, tensor pipe 23 %, issue 27-30
// %); what is left is the latency of 32 MMAs of N <= 128 per K-chunk behind one
// another.  At 64 columns, 32 maps: DRAM 39 %, tensor pipe 47 %, issue 36 %.
// Every wait is bounded (about 2 s); on expiry the kernel raises an error flag,
// drains its own copies and MMAs, frees TMEM and returns.
#include <chrono>
#include <cstdint>
#include <cstdlib>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <vector>

#include "autotune.h"
#include "common.h"
#include "dfconv.h"
#include "digits.h"
#include "kernels.h"
#include "mixed.h"
#include "plan.h"
#include "runtime.h"
#include "timing.h"

namespace s2g {

namespace {

constexpr int kB0 = 6;                 // bits of the first digit (later digits: 7)
constexpr int kPK = 64;                // K per panel
constexpr int kPM = 128;               // rows per panel
constexpr int kPanelA = kPM * kPK;     // digits of a block, elements of a panel
constexpr int kGrpK = 16;              // consecutive K of one row in a digit block
constexpr int kMinBl = 128;            // 7 slices from this band-limit
// 8 slices from this band-limit, whatever the batch (so that a map's result does
// not depend on its batch).  Per contraction at bl = 64, FP64 kernel against
// slicing + contraction: 1 map 16 / 26 us, 8 complex maps 50 / 28, 32 maps 77 /
// 38; at bl = 32 8 maps 28 / 29, 32 maps 37 / 30.
constexpr int kMinBl8 = kTensorMinBl;
constexpr long long kWaitCycles = 4000000000LL;

// NC real coefficient columns per CTA (16, 32 or 64): parts x maps x {re, im};
// S digit slices (7, or 8 for FP64 results).  NC <= 32: two TMEM accumulators
// alternate between tiles; NC = 64: one accumulator of 64 S columns (all of
// TMEM at S = 8).  The table rings take what the coefficient stages leave of
// shared memory; the digit blocks in flight (48 KB and more) cover the latency
// at an SM's share of the HBM bandwidth (28 KB).
template <int NC, int S>
struct Cfg {
  static constexpr int kXST = NC == 16 ? 3 : 2;                                    // coefficient ring
  static constexpr int kAST = NC == 64 ? 3 : 5;                                    // panel ring
  static constexpr int kRST = NC == 64 ? (S == 8 ? 6 : 8) : (NC == 32 ? 10 : 12);  // digit-block ring
  static constexpr int kNBuf = NC == 64 ? 1 : 2;                                   // TMEM accumulators
  static constexpr int kConvWarps = NC == 64 ? 2 : 5;  // 2: 640 threads, so that 96 registers hold the epilogue
  static constexpr int kEpiWarps = NC / 4;  // one per TMEM lane quarter and 16-column chunk
  static constexpr int kThreads = 32 * (2 + kConvWarps + kEpiWarps);
  static constexpr int kPanelX = S * NC * kPK;  // elements
  static constexpr int kAccCols = S * NC;       // TMEM columns per accumulator
  static constexpr int kTmemCols = NC == 16 ? 256 : 512;
  static constexpr size_t kSmemA = (size_t)kAST * kPanelA * 2;
  static constexpr size_t kSmemR = (size_t)kRST * kPanelA;
  static constexpr size_t kSmemX = (size_t)kXST * kPanelX * 2;
  static constexpr int kNumBars = 2 * kAST + 2 * kRST + 2 * kXST + 4 + 1;
  static constexpr size_t kSmemBytes = 1024 + kSmemA + kSmemX + kSmemR + kNumBars * 8 + 16;
  static_assert(kSmemBytes <= 232448, "shared memory");
  // The converter warps take blocks out of order, and a parity wait tells only
  // neighbouring phases of a stage apart.  A warp waits for block c after its
  // block c - kConvWarps, whose panel stage was free, so the MMAs (in order) had
  // consumed every block up to c - kConvWarps - kAST: the panel stage of c is at
  // most one phase behind if kConvWarps <= kAST, and the digit block before c in
  // its stage (c - kRST) has been loaded if kConvWarps + kAST <= kRST.
  static_assert(kConvWarps <= kAST && kConvWarps + kAST <= kRST, "ring depths");
  static_assert(kNBuf * kAccCols <= kTmemCols, "TMEM");
};

// What a launch computes.
enum MxMode {
  MX_L2T = 0,   // sums over l: rows t, K = l
  MX_T2L = 1,   // sums over theta: rows l, K = t
  MX_QUAD = 2,  // the quadrature operator on ring spectra: rows t, K = t', one block per parity of m + n
};

struct Geom {
  int l0, nl, rows, K, nkc, nrt;
};
// Tile geometry of one m block of a table with nt theta samples: l -> t has
// rows t < nt and reduction K = l - l0; t -> l has rows l - l0 and K = t.
__host__ __device__ inline Geom geom(int bl, int nt, int an, int m, int mode) {
  Geom g;
  const int am = m < 0 ? -m : m;
  g.l0 = mode == MX_QUAD ? 0 : (am > an ? am : an);
  g.nl = bl - g.l0 > 0 ? bl - g.l0 : 0;
  g.rows = mode == MX_T2L ? g.nl : nt;
  g.K = mode == MX_L2T ? g.nl : nt;
  g.nkc = g.nl > 0 ? (g.K + kPK - 1) / kPK : 0;
  g.nrt = (g.rows + kPM - 1) / kPM;  // l -> t keeps its rows (written as zeros) when nl = 0
  return g;
}

// element index of (row, col) inside a [rows][64] bf16 K-major panel with the
// 128-byte swizzle: 16-byte chunk index XOR (row mod 8), 8-row atoms of 1024 B
__host__ __device__ inline int swz(int row, int col) {
  const int chunk = (col >> 3) ^ (row & 7);
  return (row >> 3) * 512 + (row & 7) * 64 + chunk * 8 + (col & 7);
}


// Two digits (bytes d + 64 of w, chosen by sel) as bf16: 0x4300 | x is 128 + x
// for x < 128 and 256 for x = 128, all exact, so subtracting 192 leaves d.
__device__ __forceinline__ uint32_t digits2_bf16(uint32_t w, uint32_t sel) {
  const uint32_t v = __byte_perm(w, 0x43434343u, sel);
  uint32_t r;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(0x43404340u));
  return r;
}

struct TableRefM {
  int mi;
  double sign;
};
__device__ __forceinline__ TableRefM table_ref_m(int tmlo, int n, int m) {
  TableRefM r;
  if (n > 0 || (n == 0 && m >= 0)) {
    r.mi = m - tmlo;
    r.sign = 1.0;
  } else {
    const int an = n < 0 ? -n : n;
    r.mi = -m - tmlo;
    r.sign = ((m + an) & 1) ? -1.0 : 1.0;
  }
  return r;
}

// ---------------------------------------------------------------------------
// table slicing (plan time)
// ---------------------------------------------------------------------------

// mode: MxMode; tr: the source block holds the transpose (row k, column row).  panels8 (nullable with panels set, or the reverse):
// the eighth digit's blocks, one per (row tile, K-chunk).
__global__ void __launch_bounds__(128) k_slice_table(const double *__restrict__ T,
                                                     const int64_t *__restrict__ off, int bl, int nt,
                                                     int an, int tmlo, int mode, int tr, uint8_t *__restrict__ panels,
                                                     uint8_t *__restrict__ panels8,
                                                     const int64_t *__restrict__ pan_off,
                                                     int16_t *__restrict__ eA,
                                                     const int64_t *__restrict__ e_off) {
  const int mi = blockIdx.x, rt = blockIdx.y;
  const Geom g = geom(bl, nt, an, tmlo + mi, mode);
  if (rt >= g.nrt) return;
  const double *Tm = T + off[mi];
  const int64_t rs = tr ? 1 : g.K, ks = tr ? g.rows : 1;  // strides of the row and of k
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kpad = g.nkc * kPK;
  for (int rr = warp; rr < kPM; rr += 4) {
    const int row = rt * kPM + rr;
    const bool live = row < g.rows;
    int e;
    if (panels) {
      int mx = 0;
      if (live)
        for (int k = lane; k < g.K; k += 32) mx = max(mx, exp_field(Tm[row * rs + k * ks]));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      e = block_scale(mx);
      if (lane == 0) eA[e_off[mi] + row] = (int16_t)e;
    } else {
      e = eA[e_off[mi] + row];
    }
    for (int k = lane; k < kpad; k += 32) {
      const double v = (live && k < g.K) ? Tm[row * rs + k * ks] : 0.0;
      const int kc = k / kPK;
      const int64_t tile = (int64_t)(rt * g.nkc + kc);
      const int idx = (k % kPK / kGrpK * kPM + rr) * kGrpK + k % kGrpK;
      if (panels) {
        int dg[kS];
        int_digits(fixed48(v, e), dg);
        uint8_t *p = panels + pan_off[mi] + tile * kS * kPanelA;
#pragma unroll
        for (int j = 0; j < kS; ++j) p[(int64_t)j * kPanelA + idx] = (uint8_t)(dg[j] + 64);
      }
      if (panels8) panels8[pan_off[mi] / kS + tile * kPanelA + idx] = (uint8_t)(eighth_digit(v, e) + 64);
    }
  }
}

// ---------------------------------------------------------------------------
// coefficient slicing (per call)
// ---------------------------------------------------------------------------

// One scale's coefficients and outputs inside a fused table pass.
struct Part {
  const double2 *src;  // l -> t: flm-like (l^2 + l + m); t -> l: spectra [t][m - s_mlo]
  int64_t ss;
  int sw, s_mlo, x_half;
  const double2 *w;  // per-l weight (l -> t: on the input; t -> l: on the output)
  double wscale;
  int wconj;
  int wkind;  // WKIND_* of w
  int lmin;
  double2 *dst;  // l -> t: spectra [t][m - d_mlo] (row width dw); t -> l: l^2 + l + m
  int64_t ds;
  int dw, d_mlo;
};

struct XArgs {
  int mode;  // MxMode
  int bl, nt, an, mlo, lmin;  // lmin: smallest lmin over the parts
  int nparts;
  Part part[kMaxParts];
  int nb, b0, mpp;  // maps per part in this launch: column pair cp -> part cp / mpp, map b0 + cp % mpp
  int nmp;          // problem m count
  int nkcmax, kst;  // largest K-chunk count over the problem m; staged column stride (double2)
  const int64_t *xoff;
  uint16_t *xpan;
  int *eX;
};

__device__ __forceinline__ double2 weight_of(const double2 *w, double wscale, int wconj, int l) {
  double2 v = w ? w[l] : make_double2(1.0, 0.0);
  if (wconj) v.y = -v.y;
  return make_double2(v.x * wscale, v.y * wscale);
}
// (out of line like mul_fp64)
__device__ __noinline__ double2 weighted_complex(double2 x, double2 w, double wscale, int wconj) {
  if (wconj) w.y = -w.y;
  const double2 v = make_double2(w.x * wscale, w.y * wscale);
  return make_double2(x.x * v.x - x.y * v.y, x.x * v.y + x.y * v.x);
}
// x times the part's weight at degree l (x times wscale without a weight).  A
// real or imaginary weight takes three FP64 products instead of the eight of a
// scaled complex product; the terms dropped are exact zeros, so the result is
// the same.
__device__ __forceinline__ double2 weighted(const Part &P, double2 x, int l) {
  if (!P.w) return make_double2(x.x * P.wscale, x.y * P.wscale);
  if (P.wkind == WKIND_REAL) {
    const double r = P.w[l].x * P.wscale;
    return make_double2(x.x * r, x.y * r);
  }
  if (P.wkind == WKIND_IMAG) {  // x (i r)
    const double r = (P.wconj ? -P.w[l].y : P.w[l].y) * P.wscale;
    return make_double2(-(x.y * r), x.x * r);
  }
  const double2 wt = weight_of(P.w, P.wscale, P.wconj, l);
  return make_double2(x.x * wt.x - x.y * wt.y, x.x * wt.y + x.y * wt.x);
}

// Coefficient slicing: one block per (kMG consecutive problem m, column pair
// cp = part cp / mpp, map b0 + cp % mpp).  Phase 1 stages the kMG complex
// columns in shared memory, reading the source with m as the contiguous index
// (flm-like l^2 + l + m for l -> t, spectra [t][m] for t -> l), so that a warp
// load covers 64-byte runs, and records the largest exponent field of each
// real and imaginary column.  Phase 2 writes the digit panels: 8 consecutive
// lanes build one 128-byte panel row from 8 K values each.  The FP64 values
// are read once and the panels written once; columns without a map are left
// alone (with one map and one part, seven of eight column pairs).
//
// What bounds it: integer instructions and the latency of the two phases, at
// 3-4 CTAs per SM, not the bytes (50 % of the DRAM rate from spectra, 20 % from
// coefficients, whose panels stay in L2).  One launch at L = 512, 32 maps:
// from spectra 195 -> 159 us with the digits spread in integers (digit_bytes)
// instead of peeled off a double-float; from coefficients 191 -> 137 us with the
// weight products in integers (mul_int) as well, as the FP64 unit they kept
// busy is shared by the SM.  64 registers: the fourth CTA is worth 10 %.
constexpr int kMG = 4;
constexpr int kSliceThreads = 256;
constexpr int kNonFinite = 1 << 20;  // column exponent of a column that holds an infinity or a NaN
// staged index of K position k: one double2 of padding per 8, so that the
// 16-byte reads of 8 lanes at K stride 8 fall in distinct banks
__host__ __device__ __forceinline__ int sv_idx(int k) { return k + (k >> 3); }

template <int NC, int S>
__global__ void __launch_bounds__(kSliceThreads, 4) k_slice_x(XArgs a) {
  extern __shared__ double2 sv[];  // [kMG][a.kst]
  __shared__ int gl0[kMG], gnkc[kMG], gkc0[kMG], gls[kMG], gex[kMG][2];
  constexpr int PX = Cfg<NC, S>::kPanelX;
  const int cp = blockIdx.y, pm0 = blockIdx.x * kMG, c0 = 2 * cp;
  const int part = cp / a.mpp, b = a.b0 + cp % a.mpp;
  if (part >= a.nparts || b >= a.nb) {
    // no map in these columns: their panels are never written and their sums
    // never stored; ordinary exponents keep the epilogue on its straight path
    if (threadIdx.x < 2 * kMG && pm0 + (int)threadIdx.x / 2 < a.nmp)
      a.eX[(pm0 + threadIdx.x / 2) * NC + c0 + threadIdx.x % 2] = 0;
    return;
  }
  if (threadIdx.x < kMG) {
    const int pm = pm0 + threadIdx.x;
    int l0 = 0, nkc = 0, kc0 = 0, ls = 0;
    if (pm < a.nmp) {
      const Geom g = geom(a.bl, a.nt, a.an, a.mlo + pm, a.mode);
      l0 = g.l0;
      nkc = g.nkc;
      if (a.mode == MX_L2T) {
        const int lst = g.l0 > a.lmin ? g.l0 : a.lmin;
        kc0 = lst >= a.bl ? g.nkc : (lst - g.l0) / kPK;
        // first degree with a value: below its part's lmin the column is zero
        ls = a.part[part].lmin > g.l0 ? a.part[part].lmin : g.l0;
      }
    }
    gl0[threadIdx.x] = l0;
    gnkc[threadIdx.x] = nkc;
    gkc0[threadIdx.x] = kc0;
    gls[threadIdx.x] = ls;
    gex[threadIdx.x][0] = gex[threadIdx.x][1] = 0;
  }
  for (int i = threadIdx.x; i < kMG * a.kst; i += kSliceThreads) ((int4 *)sv)[i] = make_int4(0, 0, 0, 0);
  __syncthreads();
  {
    const Part &P = a.part[part];
    const int mi = threadIdx.x % kMG;  // fixed per thread: kSliceThreads is a multiple of kMG
    const int pm = pm0 + mi, m = a.mlo + pm, am = m < 0 ? -m : m;
    const bool has = pm < a.nmp && gnkc[mi] > gkc0[mi];
    double2 *col = sv + mi * a.kst;
    int er = 0, ei = 0;
    constexpr int kStep = kSliceThreads / kMG, kU = 4;  // kU loads in flight per thread
    if (a.mode == MX_L2T) {
      // every lane walks the same degrees, so the kMG m of one degree are adjacent
      int lb = a.bl;
      for (int i = 0; i < kMG; ++i)
        if (pm0 + i < a.nmp && gnkc[i] > gkc0[i]) lb = min(lb, gls[i]);
      const int l0 = gl0[mi], ls = gls[mi];
      const bool neg = P.x_half && m < 0;
      const int mm = neg ? -m : m;
      // warp-uniform bounds: the weights travel by shuffles
      static_assert(kU == kMG, "lane mi forms the scaled weight of step u = mi");
      for (int lw = lb + (threadIdx.x & ~31) / kMG; lw < a.bl; lw += kU * kStep) {
        const int l1 = lw + (threadIdx.x & 31) / kMG;
        double2 v[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int l = l1 + u * kStep;
          v[u] = make_double2(0.0, 0.0);
          if (has && l >= ls && l < a.bl) v[u] = P.src[(int64_t)b * P.ss + (int64_t)l * l + l + mm];
        }
        double r = P.wscale;  // lane mi: the scaled weight of degree l1 + mi kStep
        if (P.w && P.wkind != WKIND_COMPLEX && l1 + mi * kStep < a.bl) {
          const double2 w = P.w[l1 + mi * kStep];
          r = mul_int(P.wkind == WKIND_REAL ? w.x : flip_sign(w.y, P.wconj), r);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int l = l1 + u * kStep;
          const double ru = __shfl_sync(0xffffffffu, r, u, kMG);
          if (!has || l < ls || l >= a.bl) continue;
          double2 x = v[u];
          // sign changes as bit flips (a negation can cost an FP64 instruction)
          if (neg) x = make_double2(flip_sign(x.x, am), flip_sign(x.y, am + 1));
          if (P.w && P.wkind == WKIND_COMPLEX)
            x = weighted_complex(x, P.w[l], P.wscale, P.wconj);
          else if (P.w && P.wkind == WKIND_IMAG)  // x (i r)
            x = make_double2(flip_sign(mul_int(x.y, ru), 1), mul_int(x.x, ru));
          else
            x = make_double2(mul_int(x.x, ru), mul_int(x.y, ru));
          col[sv_idx(l - l0)] = x;
          er = max(er, exp_field(x.x));
          ei = max(ei, exp_field(x.y));
        }
      }
    } else if (has) {
      const double2 *src = P.src + (int64_t)b * P.ss + (m - P.s_mlo);
      for (int t1 = threadIdx.x / kMG; t1 < a.nt; t1 += kU * kStep) {
        double2 v[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int t = t1 + u * kStep;
          v[u] = t < a.nt ? src[(int64_t)t * P.sw] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int t = t1 + u * kStep;
          if (t >= a.nt) continue;
          col[sv_idx(t)] = v[u];
          er = max(er, exp_field(v[u].x));
          ei = max(ei, exp_field(v[u].y));
        }
      }
    }
    // lanes with the same m are kMG apart
#pragma unroll
    for (int o = kMG; o < 32; o <<= 1) {
      er = max(er, __shfl_xor_sync(0xffffffffu, er, o));
      ei = max(ei, __shfl_xor_sync(0xffffffffu, ei, o));
    }
    if ((threadIdx.x & 31) < kMG) {
      atomicMax(&gex[mi][0], er);
      atomicMax(&gex[mi][1], ei);
    }
  }
  __syncthreads();
  if (threadIdx.x < kMG) {
    const int pm = pm0 + threadIdx.x;
    // |v| < 2^e for every value of the column (e = largest unbiased exponent + 1)
    for (int ri = 0; ri < 2; ++ri) {
      const int mx = gex[threadIdx.x][ri];
      const int e = S == kS ? block_scale(mx) : (mx > 1 ? mx : 1) - 1022;
      gex[threadIdx.x][ri] = e;
      if (pm < a.nmp) a.eX[pm * NC + c0 + ri] = mx == 2047 ? kNonFinite : e;
    }
  }
  __syncthreads();
  const int units = kMG * a.nkcmax * 8;
  for (int u = threadIdx.x; u < units; u += kSliceThreads) {
    const int h = u & 7, rest = u >> 3;
    const int kc = rest % a.nkcmax, mi = rest / a.nkcmax;
    const int pm = pm0 + mi;
    if (pm >= a.nmp || kc < gkc0[mi] || kc >= gnkc[mi]) continue;
    uint16_t *p = a.xpan + a.xoff[pm] * (NC / 16 * S) + (int64_t)kc * PX;
    const double *col = (const double *)(sv + mi * a.kst);
#pragma unroll 1
    for (int ri = 0; ri < 2; ++ri) {  // real part (column c0), then imaginary part (c0 + 1)
      uint32_t pk[S][4];
      const int e = gex[mi][ri];
#pragma unroll
      for (int q = 0; q < 4; ++q) {  // K values 2 q and 2 q + 1
        uint32_t lo[2], hi[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const double v = col[2 * sv_idx(kc * kPK + h * 8 + 2 * q + r) + ri];
          digit_bytes<S>(S == kS ? fixed48(v, e) : fixed55(v, e), lo[r], hi[r]);
        }
        // bytes of one digit of both values side by side, two digits per word
        const uint32_t w[4] = {__byte_perm(lo[0], lo[1], 0x5140), __byte_perm(lo[0], lo[1], 0x7362),
                               __byte_perm(hi[0], hi[1], 0x5140), __byte_perm(hi[0], hi[1], 0x7362)};
#pragma unroll
        for (int j = 0; j < S; ++j) {
          const int y = S - 1 - j;  // byte position of digit j
          pk[j][q] = digits2_bf16(w[y >> 1], y & 1 ? 0x4342 : 0x4140);
        }
      }
#pragma unroll
      for (int j = 0; j < S; ++j)
        *(uint4 *)(p + swz(j * NC + c0 + ri, h * 8)) = make_uint4(pk[j][0], pk[j][1], pk[j][2], pk[j][3]);
    }
  }
}

// ---------------------------------------------------------------------------
// tcgen05 / mbarrier / bulk-copy primitives
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t saddr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void bar_init(uint64_t *b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t *b) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(saddr(b))
               : "memory");
}
__device__ __forceinline__ void bar_expect_tx(uint64_t *b, uint32_t bytes) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(
                   saddr(b)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t *b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, "
      "p;\n\t}"
      : "=r"(ok)
      : "r"(saddr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait that ignores the abort flag (draining before TMEM release).
__device__ __noinline__ bool bar_wait_timed(uint64_t *b, uint32_t parity) {
  const long long t0 = clock64();
  while (!bar_try(b, parity))
    if (clock64() - t0 > kWaitCycles) return false;
  return true;
}
// Bounded wait; false when the CTA is aborting or the wait expired (then it
// raises the CTA abort flag and the global error flag).
__device__ __noinline__ bool bar_wait_slow(uint64_t *b, uint32_t parity, volatile int *abort_flag, int *err) {
  const long long t0 = clock64();
  for (uint32_t it = 0;; ++it) {
    if (bar_try(b, parity)) return true;
    if ((it & 255u) == 255u) {
      if (*abort_flag) return false;
      if (clock64() - t0 > kWaitCycles) {
        *abort_flag = 1;
        atomicExch(err, 1);
        return false;
      }
    }
  }
}
__device__ __forceinline__ bool bar_wait(uint64_t *b, uint32_t parity, volatile int *abort_flag, int *err) {
  return bar_try(b, parity) || bar_wait_slow(b, parity, abort_flag, err);
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   saddr(dst)),
               "l"(src), "r"(bytes), "r"(saddr(bar))
               : "memory");
}
__device__ __forceinline__ uint64_t sw128_desc(const void *p) {
  const uint32_t a = saddr(p);
  uint64_t d = 0;
  d |= (uint64_t)((a >> 4) & 0x3FFFu);  // start address
  d |= (uint64_t)1 << 16;               // leading byte offset (unused with 128B swizzle)
  d |= (uint64_t)(1024 >> 4) << 32;     // stride byte offset: 8-row groups 1024 B apart
  d |= (uint64_t)1 << 46;               // descriptor version
  d |= (uint64_t)2 << 61;               // 128-byte swizzle
  return d;
}
__device__ __forceinline__ uint32_t idesc_bf16(int M, int N) {
  return (1u << 4)                    // D: f32
         | (1u << 7) | (1u << 10)     // A, B: bf16
         | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);  // K-major A and B
}
__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, "
      "p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(bar))
               : "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}


// ---------------------------------------------------------------------------
// the contraction
// ---------------------------------------------------------------------------

// 8 digits, bytes d + 64 of two words, as bf16
__device__ __forceinline__ uint4 digits_bf16(uint32_t lo, uint32_t hi) {
  return make_uint4(digits2_bf16(lo, 0x4140), digits2_bf16(lo, 0x4342), digits2_bf16(hi, 0x4140),
                    digits2_bf16(hi, 0x4342));
}

struct MxArgs {
  int mode;  // MxMode
  const uint8_t *panels, *panels8;
  const int64_t *pan_off;
  const int16_t *eA;
  const int64_t *e_off;
  int bl, nt, an, tmlo, n, mlo, lmin;  // lmin: smallest over the parts
  const uint16_t *xpan;
  const int64_t *xoff;
  const int *eX;
  const int2 *tiles;
  int ntiles;
  int nparts;
  Part part[kMaxParts];
  int nb, mpp;
  // map groups of one launch: group g holds maps [b0 + g mpp, b0 + (g + 1) mpp)
  // of every part, its coefficient panels at xpan + g xg and exponents at
  // eX + g eXg.  Work item v is tile v / ngroups of group v % ngroups, so that
  // neighbouring CTAs run the same table tile for different groups and the
  // second read of the tile's panels is served by L2.
  int b0, ngroups, eXg;
  int64_t xg;
  int *err;
};

struct TileInfo {
  int pm, m, mi, rt, kc0, nkc, l0;
  int g;  // map group
  double sign;
};
// tile entry of work item v (read one item ahead of its use)
__device__ __forceinline__ int2 tile_of(const MxArgs &a, int v) {
  return v < a.ntiles * a.ngroups ? a.tiles[v / a.ngroups] : make_int2(0, 0);
}
__device__ __forceinline__ TileInfo tile_info(const MxArgs &a, int v, int2 tl) {
  TileInfo ti;
  ti.g = v % a.ngroups;
  ti.pm = tl.x;
  ti.rt = tl.y;
  ti.m = a.mlo + ti.pm;
  if (a.mode == MX_QUAD) {
    ti.mi = (ti.m + a.an) & 1;
    ti.sign = 1.0;
  } else {
    const TableRefM r = table_ref_m(a.tmlo, a.n, ti.m);
    ti.mi = r.mi;
    ti.sign = r.sign;
  }
  const Geom g = geom(a.bl, a.nt, a.an, ti.m, a.mode);
  ti.l0 = g.l0;
  ti.nkc = g.nkc;
  const int lst = g.l0 > a.lmin ? g.l0 : a.lmin;
  ti.kc0 = 0;
  if (a.mode == MX_L2T) ti.kc0 = lst >= a.bl ? g.nkc : (lst - g.l0) / kPK;
  return ti;
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float *v) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
// the S class accumulators of 8 columns into registers (waits for the loads)
template <int S>
__device__ __forceinline__ void load_classes8(uint32_t taddr, int ncols_per_class, float (*acc)[8]) {
#pragma unroll
  for (int c = 0; c < S; ++c) tmem_ld8(taddr + (uint32_t)(c * ncols_per_class), acc[c]);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// Combine the 7 class accumulators of 8 columns for this thread's row:
// S = sum_c acc_c 2^(-7c) by Horner in double-float on the FP32 pipe (the class
// values and 2^-7 scalings are exact floats), then one widening to FP64 with
// the power of two 2^(ea + eX - 12) applied while widening (dfconv.h).
__device__ __forceinline__ int ex_at(int4 e0, int4 e1, int col) {
  const int4 e = col < 4 ? e0 : e1;
  const int c = col & 3;
  return c == 0 ? e.x : (c == 1 ? e.y : (c == 2 ? e.z : e.w));
}
// eX of the 8 columns in e0 (columns 0-3) and e1 (4-7)
__device__ __forceinline__ void combine8(float (*acc)[8], int ea, int4 e0, int4 e1, double sign, double *y) {
#pragma unroll
  for (int col = 0; col < 8; ++col) {
    float hi = acc[kS - 1][col], lo = 0.0f;
#pragma unroll
    for (int c = kS - 2; c >= 0; --c) {
      hi = __fmul_rn(hi, 0.0078125f);
      lo = __fmul_rn(lo, 0.0078125f);
      const float s = __fadd_rn(acc[c][col], hi);
      const float v = __fsub_rn(s, acc[c][col]);
      float e = __fadd_rn(__fsub_rn(acc[c][col], __fsub_rn(s, v)), __fsub_rn(hi, v));
      e = __fadd_rn(e, lo);
      hi = __fadd_rn(s, e);
      lo = __fsub_rn(e, __fsub_rn(hi, s));
    }
    if (sign < 0.0) {
      hi = -hi;
      lo = -lo;
    }
    const int ex = ex_at(e0, e1, col);
    y[col] = ex == kNonFinite ? double_of(0x7FF8000000000000ull) : join_scaled(hi, lo, ea + ex - 2 * kB0);
  }
}
// The same for 8 slices and FP64 results: the class sums are integers; classes
// 0-3 and 4-7 go to two 64-bit words of 43 and 46 bits, their 71-bit sum is
// normalised and rounded once, in integer arithmetic (an FP64 conversion and
// sum would take three FP64 instructions per value, more than the tile's MMAs).
__device__ __forceinline__ void combine8_int(float (*acc)[8], int ea, int4 e0, int4 e1, double sign, double *y) {
#pragma unroll
  for (int col = 0; col < 8; ++col) {
    long long hi = 0, lo = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      hi += (long long)__float2int_rn(acc[c][col]) << (7 * (3 - c));
      lo += (long long)__float2int_rn(acc[c + 4][col]) << (7 * (3 - c));
    }
    if (sign < 0.0) {
      hi = -hi;
      lo = -lo;
    }
    const int ex = ex_at(e0, e1, col);
    y[col] = ex == kNonFinite ? double_of(0x7FF8000000000000ull) : join71(hi, lo, ea + ex - 2 * kB0 - 49);
  }
}

template <int NC, int S>
__global__ void __launch_bounds__(Cfg<NC, S>::kThreads, 1) k_contract_mx(MxArgs a) {
  using C = Cfg<NC, S>;
  constexpr int PX = C::kPanelX;
  constexpr int ACC = C::kAccCols;
  constexpr int TMC = C::kTmemCols;
  constexpr int kAST = C::kAST, kRST = C::kRST, kXST = C::kXST;
  constexpr int NBUF = C::kNBuf;
  constexpr int kEpi0 = 2 + C::kConvWarps;  // first epilogue warp
  constexpr int kNumBars = C::kNumBars;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint16_t *sA = (uint16_t *)smem;
  uint16_t *sX = (uint16_t *)(smem + C::kSmemA);
  uint8_t *sR = smem + C::kSmemA + C::kSmemX;
  uint64_t *bars = (uint64_t *)(smem + C::kSmemA + C::kSmemX + C::kSmemR);
  uint64_t *fullA = bars, *emptyA = fullA + kAST, *fullR = emptyA + kAST, *emptyR = fullR + kRST;
  uint64_t *fullX = emptyR + kRST, *emptyX = fullX + kXST;
  uint64_t *tfull = emptyX + kXST, *tempty = tfull + 2, *mma_done = tfull + 4;
  volatile int *abort_flag = (volatile int *)(bars + kNumBars);
  uint32_t *tmem_slot = (uint32_t *)(bars + kNumBars) + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kAST; ++i) {
      bar_init(&fullA[i], 1);
      bar_init(&emptyA[i], 1);
    }
    for (int i = 0; i < kRST; ++i) {
      bar_init(&fullR[i], 1);
      bar_init(&emptyR[i], 1);
    }
    for (int i = 0; i < kXST; ++i) {
      bar_init(&fullX[i], 1);
      bar_init(&emptyX[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      bar_init(&tfull[i], 1);
      bar_init(&tempty[i], 32 * C::kEpiWarps);
    }
    bar_init(mma_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(tmem_slot)),
                 "r"(TMC)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  int issuedR = 0, issuedX = 0;
  if (warp == 0 && lane == 0) {
    // ---------------- producer ----------------
    bool ok = true;
    int2 next = tile_of(a, blockIdx.x);
    for (int t = blockIdx.x; ok && t < a.ntiles * a.ngroups; t += gridDim.x) {
      const TileInfo ti = tile_info(a, t, next);
      next = tile_of(a, t + gridDim.x);
      const uint8_t *pan = a.panels + a.pan_off[ti.mi] + (int64_t)ti.rt * ti.nkc * kS * kPanelA;
      const uint8_t *pan8 = S == kSmax ? a.panels8 + a.pan_off[ti.mi] / kS + (int64_t)ti.rt * ti.nkc * kPanelA : nullptr;
      const uint16_t *xp = a.xpan + ti.g * a.xg + a.xoff[ti.pm] * (NC / 16 * S);
      for (int kc = ti.kc0; ok && kc < ti.nkc; ++kc) {
        const int xs = issuedX % kXST;
        if (!(ok = bar_wait(&emptyX[xs], ((issuedX / kXST) & 1) ^ 1, abort_flag, a.err))) break;
        bar_expect_tx(&fullX[xs], PX * 2);
        bulk_g2s(sX + (size_t)xs * PX, xp + (int64_t)kc * PX, PX * 2, &fullX[xs]);
        ++issuedX;
        for (int j = 0; j < S; ++j) {
          const int rs = issuedR % kRST;
          if (!(ok = bar_wait(&emptyR[rs], ((issuedR / kRST) & 1) ^ 1, abort_flag, a.err))) break;
          bar_expect_tx(&fullR[rs], kPanelA);
          const uint8_t *src = j < kS ? pan + ((int64_t)kc * kS + j) * kPanelA : pan8 + (int64_t)kc * kPanelA;
          bulk_g2s(sR + (size_t)rs * kPanelA, src, kPanelA, &fullR[rs]);
          ++issuedR;
        }
      }
    }
  } else if (warp == 1 && lane == 0) {
    // ---------------- MMA issuer ----------------
    int ca = 0, cx = 0, ti_n = 0;
    bool ok = true, any = false;
    int2 next = tile_of(a, blockIdx.x);
    for (int t = blockIdx.x; ok && t < a.ntiles * a.ngroups; t += gridDim.x, ++ti_n) {
      const TileInfo ti = tile_info(a, t, next);
      next = tile_of(a, t + gridDim.x);
      const int ab = ti_n % NBUF;
      if (!(ok = bar_wait(&tempty[ab], ((ti_n / NBUF) & 1) ^ 1, abort_flag, a.err))) break;
      tc_fence_after();
      const uint32_t d0 = tmem + (uint32_t)(ab * ACC);
      if (ti.kc0 >= ti.nkc) {
        bar_arrive(&tfull[ab]);  // nothing to accumulate: the epilogue writes zeros
        continue;
      }
      for (int kc = ti.kc0; ok && kc < ti.nkc; ++kc) {
        const int xs = cx % kXST;
        if (!(ok = bar_wait(&fullX[xs], (cx / kXST) & 1, abort_flag, a.err))) break;
        tc_fence_after();
        const uint64_t bdesc = sw128_desc(sX + (size_t)xs * PX);
        for (int j = 0; j < S; ++j) {
          const int as = ca % kAST;
          if (!(ok = bar_wait(&fullA[as], (ca / kAST) & 1, abort_flag, a.err))) break;
          tc_fence_after();
          const uint64_t adesc = sw128_desc(sA + (size_t)as * kPanelA);
          // B rows [0, NC (S - j)) -> accumulator columns NC j + row, in MMAs of N <= 256
          const int ntot = NC * (S - j);
          for (int off = 0; off < ntot; off += 256) {
            const int n = ntot - off < 256 ? ntot - off : 256;
            const uint32_t idesc = idesc_bf16(kPM, n);
            // 8-row atoms of 128 B: a row offset of `off` moves the start by off * 128 B
            const uint64_t bd = bdesc + (uint64_t)(off * 8);
#pragma unroll
            for (int k = 0; k < kPK / 16; ++k) {
              // K advance of 16 bf16 = 32 bytes inside the swizzle atom
              mma_bf16(d0 + (uint32_t)(NC * j + off), adesc + (uint64_t)(2 * k), bd + (uint64_t)(2 * k), idesc,
                       (kc == ti.kc0 && j == 0 && k == 0) ? 0u : 1u);
            }
          }
          any = true;
          mma_commit(&emptyA[as]);
          ++ca;
        }
        if (!ok) break;
        mma_commit(&emptyX[xs]);
        ++cx;
      }
      if (!ok) break;
      mma_commit(&tfull[ab]);
    }
    if (any) {  // every MMA of this thread has completed before TMEM is released
      mma_commit(mma_done);
      if (!bar_wait_timed(mma_done, 0)) atomicExch(a.err, 2);
    }
  } else if (warp >= 2 && warp < kEpi0) {
    // ---------------- converters ----------------
    // every warp takes whole blocks, warp w the w-th, (w + kConvWarps)-th, ...:
    // the waits, the proxy fence and the arrivals (several hundred cycles a
    // block) of the warps overlap.  Lane -> rows lane + 32 i, all 4 K groups.
    const int w = warp - 2;
    int done = 0;  // blocks of earlier tiles
    bool ok = true;
    int2 next = tile_of(a, blockIdx.x);
    for (int t = blockIdx.x; ok && t < a.ntiles * a.ngroups; t += gridDim.x) {
      const TileInfo ti = tile_info(a, t, next);
      next = tile_of(a, t + gridDim.x);
      const int n = (ti.nkc - ti.kc0) * S;
      for (int c = done + (w - done % C::kConvWarps + C::kConvWarps) % C::kConvWarps; c < done + n;
           c += C::kConvWarps) {
        const int rs = c % kRST, as = c % kAST;
        ok = bar_wait(&fullR[rs], (c / kRST) & 1, abort_flag, a.err) &&
             bar_wait(&emptyA[as], ((c / kAST) & 1) ^ 1, abort_flag, a.err);
        if (!__all_sync(0xffffffffu, ok)) {
          ok = false;
          break;
        }
        const uint4 *src = (const uint4 *)(sR + (size_t)rs * kPanelA) + lane;
        uint16_t *dst = sA + (size_t)as * kPanelA;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint4 d[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) d[i] = src[q * kPM + 32 * i];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            *(uint4 *)(dst + swz(lane + 32 * i, q * kGrpK)) = digits_bf16(d[i].x, d[i].y);
            *(uint4 *)(dst + swz(lane + 32 * i, q * kGrpK + 8)) = digits_bf16(d[i].z, d[i].w);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // visible to the MMAs' reads
        __syncwarp();
        if (lane == 0) {
          bar_arrive(&fullA[as]);
          bar_arrive(&emptyR[rs]);
        }
      }
      done += n;
    }
  } else if (warp >= kEpi0) {
    // ---------------- epilogue ----------------
    // warp -> TMEM lane quarter (warp mod 4, the quarter it may address) and one
    // 16-column chunk pi, read as two 8-column halves; the accumulator is
    // handed back right after the second half is in registers, before it is
    // combined and stored, so that the next tile's MMAs wait as little as possible
    const int quarter = warp & 3;
    const int pi = (warp - kEpi0) / 4;
    const int rr = quarter * 32 + lane;
    int ti_n = 0;
    int2 next = tile_of(a, blockIdx.x);
    for (int t = blockIdx.x; t < a.ntiles * a.ngroups; t += gridDim.x, ++ti_n) {
      const TileInfo ti = tile_info(a, t, next);
      next = tile_of(a, t + gridDim.x);
      const int ab = ti_n % NBUF;
      const bool live = ti.kc0 < ti.nkc;
      // the row and column exponents do not depend on the accumulator: read
      // them before waiting, so that their latency is not spent holding TMEM
      int ea = 0;
      int4 ex4[4];
      if (live) {
        ea = (int)a.eA[a.e_off[ti.mi] + ti.rt * kPM + rr];
        const int4 *ep = (const int4 *)(a.eX + ti.g * a.eXg + ti.pm * NC + pi * 16);
#pragma unroll
        for (int q = 0; q < 4; ++q) ex4[q] = ep[q];
      }
      // warp-uniform outcome: tcgen05.ld below is .sync.aligned
      if (!__all_sync(0xffffffffu, bar_wait(&tfull[ab], (ti_n / NBUF) & 1, abort_flag, a.err))) break;
      tc_fence_after();
      if (!live) {  // nothing accumulated: release at once
        tc_fence_before();
        bar_arrive(&tempty[ab]);
      }
      const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ab * ACC);
      const int t_row = ti.rt * kPM + rr;
      const int l = ti.l0 + ti.rt * kPM + rr;
#pragma unroll 1
      for (int hh = 0; hh < 2; ++hh) {
        const int c0 = pi * 16 + hh * 8;  // first column of this half
        double y[8];
        if (live) {
          float acc[S][8];
          load_classes8<S>(taddr + (uint32_t)c0, NC, acc);
          if (hh == 1) {  // every column of this warp is in registers: hand the accumulator back
            tc_fence_before();
            bar_arrive(&tempty[ab]);
          }
          if constexpr (S == kS)
            combine8(acc, ea, hh ? ex4[2] : ex4[0], hh ? ex4[3] : ex4[1], ti.sign, y);
          else
            combine8_int(acc, ea, hh ? ex4[2] : ex4[0], hh ? ex4[3] : ex4[1], ti.sign, y);
        } else {
#pragma unroll
          for (int col = 0; col < 8; ++col) y[col] = 0.0;
        }
        // column pair cp = c0 / 2 + bb: part cp / mpp, map b0 + cp % mpp
#pragma unroll
        for (int bb = 0; bb < 4; ++bb) {
          const int cp = c0 / 2 + bb;
          const int part = cp / a.mpp;
          const int b = a.b0 + ti.g * a.mpp + cp % a.mpp;
          if (part >= a.nparts || b >= a.nb) continue;
          const Part &P = a.part[part];
          if (a.mode != MX_T2L) {
            if (t_row < a.nt)
              P.dst[(int64_t)b * P.ds + (int64_t)t_row * P.dw + (ti.m - P.d_mlo)] =
                  make_double2(y[2 * bb], y[2 * bb + 1]);
          } else {
            const int lst = ti.l0 > P.lmin ? ti.l0 : P.lmin;
            if (l >= lst && l < a.bl) {
              const double yr = y[2 * bb], yi = y[2 * bb + 1];
              P.dst[(int64_t)b * P.ds + (int64_t)l * l + l + ti.m] = weighted(P, make_double2(yr, yi), l);
            }
          }
        }
      }
    }
  }

  // producer: on abort, wait (bounded) for its own copies still in flight: the
  // last one of every stage
  __syncthreads();
  if (warp == 0 && lane == 0 && *abort_flag) {
    const long long t0 = clock64();
    for (int i = max(0, issuedR - kRST); i < issuedR; ++i)
      while (!bar_try(&fullR[i % kRST], (i / kRST) & 1) && clock64() - t0 < kWaitCycles) {
      }
    for (int i = max(0, issuedX - kXST); i < issuedX; ++i)
      while (!bar_try(&fullX[i % kXST], (i / kXST) & 1) && clock64() - t0 < kWaitCycles) {
      }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMC) : "memory");
}

// ---------------------------------------------------------------------------
// host side: sliced-table cache, tile lists, launches
// ---------------------------------------------------------------------------

struct TileList {
  int2 *d_tiles = nullptr;
  int ntiles = 0;
  int64_t *d_xoff = nullptr;
  int64_t x_elems = 0;
  int64_t work_entries = 0;  // table entries streamed per launch (all tiles)
};

// Which table a contraction reads, and how: rows of the panels are t (l -> t)
// or l (t -> l), from D[t][l] or Q[l][t]; two of the four read it transposed.
// TK_W and TK_WT: the quadrature operators W_+ and W_- of a recomputed table's
// grid, and their transposes.
enum TableKind { TK_L2T_D = 0, TK_T2L_Q = 1, TK_L2T_Q = 2, TK_T2L_D = 3, TK_W = 4, TK_WT = 5 };
MxMode kind_mode(int kind) {
  if (kind >= TK_W) return MX_QUAD;
  return kind == TK_T2L_Q || kind == TK_T2L_D ? MX_T2L : MX_L2T;
}
bool kind_of_q(int kind) { return kind == TK_T2L_Q || kind == TK_L2T_Q; }
bool kind_transposed(int kind) { return kind == TK_L2T_Q || kind == TK_T2L_D || kind == TK_WT; }

struct SlicedTable {
  int bl = 0, nt = 0, an = 0, mlo = 0, nm = 0;
  int mode = MX_L2T;
  uint8_t *panels = nullptr;   // 7 digit slices
  uint8_t *panels8 = nullptr;  // the eighth, built when an FP64 contraction first needs it
  int16_t *eA = nullptr;
  int64_t *d_pan_off = nullptr, *d_e_off = nullptr;
  size_t bytes = 0, bytes8 = 0;  // of everything; of panels8
  int users = 0;                 // calls between looking the panels up and their last launch
  bool forward7 = false;         // the split-precision forward contractions read panels
  bool captured = false;         // a graph holds the panels' addresses
  std::map<std::tuple<int, int, int, int>, TileList> lists;  // (n, mlo, mhi, lmin)
  void release() {
    cudaFree(panels);
    cudaFree(panels8);
    cudaFree(eA);
    cudaFree(d_pan_off);
    cudaFree(d_e_off);
    for (auto &l : lists) {
      cudaFree(l.second.d_tiles);
      cudaFree(l.second.d_xoff);
    }
  }
};

std::mutex g_mx_mu;
using TableKey = std::tuple<int, int, int, int>;  // (bl, an, ss, kind)
std::map<TableKey, std::unique_ptr<SlicedTable>> g_sliced;
// Optional panels that did not fit when last wanted: asked for again after
// kAskAgain, or (given back by an allocation that needed the room) not before the
// plans are released.
struct Refusal {
  std::chrono::steady_clock::time_point when;
  bool given_back;
};
constexpr std::chrono::milliseconds kAskAgain{500};
std::map<TableKey, Refusal> g_refused;
size_t g_mx_bytes = 0;
int *g_err = nullptr;

void refuse(const TableKey &key, bool given_back) {
  g_refused[key] = Refusal{std::chrono::steady_clock::now(), given_back};
}

bool capturing(cudaStream_t st) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  S2G_CUDA(cudaStreamIsCapturing(st, &cap));
  return cap != cudaStreamCaptureStatusNone;
}

// Frees the optional panels that nothing uses (caller holds g_mx_mu): the eighth
// slices, and all slices of a table that the split-precision forward contractions do
// not read.  Not those that a call is about to launch with or a graph holds.  False
// when there were none.
bool give_back_panels() {
  std::vector<TableKey> keys;
  for (auto &kv : g_sliced) {
    const SlicedTable &s = *kv.second;
    if (s.panels8 && s.users == 0 && !s.captured) keys.push_back(kv.first);
  }
  if (keys.empty()) return false;
  if (cudaDeviceSynchronize() != cudaSuccess) {  // launches that still read them
    cudaGetLastError();
    return false;
  }
  for (const TableKey &key : keys) {
    SlicedTable &s = *g_sliced[key];
    if (s.forward7) {
      cudaFree(s.panels8);
      s.panels8 = nullptr;
      s.bytes -= s.bytes8;
      g_mx_bytes -= s.bytes8;
      s.bytes8 = 0;
    } else {
      g_mx_bytes -= s.bytes;
      s.release();
      g_sliced.erase(key);
    }
    refuse(key, true);
  }
  return true;
}

// Caller holds g_mx_mu; optional: no room is made for it.
template <class T>
T *dev_alloc(size_t n, size_t *acc, bool optional = false) {
  void *p = nullptr;
  const size_t bytes = sizeof(T) * (n ? n : 1);
  cudaError_t e = cudaMalloc(&p, bytes);
  if (e == cudaErrorMemoryAllocation && !optional && give_back_panels()) {
    cudaGetLastError();
    e = cudaMalloc(&p, bytes);
  }
  S2G_CUDA(e);
  *acc += bytes;
  return (T *)p;
}

// Device memory that must stay free beside optional panels: a third of it, or
// S2LET_GPU_PANEL_RESERVE_GB.
size_t panel_reserve(size_t total) {
  const char *e = getenv("S2LET_GPU_PANEL_RESERVE_GB");
  return e && e[0] ? (size_t)(atof(e) * 1073741824.0) : total / 3;
}
// Whether `need` bytes of optional panels leave that much free.  What the
// stream-ordered pool holds without using it (the scratch of earlier calls) counts
// as free, and is released when it is wanted.
bool panels_fit(size_t need) {
  size_t fr = 0, tot = 0;
  S2G_CUDA(cudaMemGetInfo(&fr, &tot));
  const size_t want = need + panel_reserve(tot);
  if (fr >= want) return true;
  int dev = 0;
  S2G_CUDA(cudaGetDevice(&dev));
  cudaMemPool_t pool;
  S2G_CUDA(cudaDeviceGetDefaultMemPool(&pool, dev));
  uint64_t held = 0, used = 0;
  S2G_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held));
  S2G_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used));
  if (fr + (size_t)(held - used) < want) return false;
  S2G_CUDA(cudaMemPoolTrimTo(pool, 0));
  S2G_CUDA(cudaMemGetInfo(&fr, &tot));
  return fr >= want;
}

// Panels of one table and kind (caller holds g_mx_mu).  The split-precision
// forward contractions cannot do without theirs; the others (with the eighth
// digit) are optional: the FP64 and double-float kernels take over (nullptr)
// when table copies are switched off (s2let_gpu_set_split_tables), when a third of
// the device memory would not stay free (panels_fit), or when a stream capture
// meets a table that no earlier call has built.  A refusal is looked at again
// kAskAgain later.
SlicedTable *sliced(const WignerTable &tb, int kind, bool eighth, cudaStream_t st) {
  const int mode = kind_mode(kind);
  // the quadrature operators belong to the grid: one block per parity
  const bool quad = mode == MX_QUAD;
  const int nm = quad ? 2 : tb.nm, tmlo = quad ? 0 : tb.mlo;
  const TableKey key = std::make_tuple(tb.bl, quad ? -1 : tb.an, tb.ss, kind);
  if (eighth && !get_split_tables()) return nullptr;
  auto it = g_sliced.find(key);
  if (it != g_sliced.end() && (!eighth || it->second->panels8)) return it->second.get();
  if (eighth) {
    if (capturing(st)) return nullptr;
    const auto no = g_refused.find(key);
    if (no != g_refused.end() &&
        (no->second.given_back || std::chrono::steady_clock::now() - no->second.when < kAskAgain))
      return nullptr;
  }
  const bool fresh = it == g_sliced.end();
  std::vector<int64_t> po(nm), eo(nm);
  int64_t ptot = 0, etot = 0;
  for (int mi = 0; mi < nm; ++mi) {
    const Geom g = geom(tb.bl, tb.nt, tb.an, tmlo + mi, mode);
    po[mi] = ptot;
    eo[mi] = etot;
    ptot += (int64_t)g.nrt * g.nkc * kS * kPanelA;
    etot += (int64_t)g.nrt * kPM;
  }
  if (eighth) {
    if (!panels_fit((size_t)(ptot / kS) * (fresh ? kSmax : 1))) {
      refuse(key, false);
      return nullptr;
    }
  }
  std::unique_ptr<SlicedTable> made;
  SlicedTable *s = fresh ? nullptr : it->second.get();
  size_t by = 0, by8 = 0;
  if (fresh) {
    made = std::make_unique<SlicedTable>();
    s = made.get();
    s->bl = tb.bl;
    s->nt = tb.nt;
    s->an = tb.an;
    s->mlo = tmlo;
    s->nm = nm;
    s->mode = mode;
  }
  uint8_t *p8 = nullptr;
  try {
    if (fresh) {
      s->panels = dev_alloc<uint8_t>((size_t)ptot, &by, eighth);
      s->eA = dev_alloc<int16_t>((size_t)etot, &by, eighth);
      s->d_pan_off = dev_alloc<int64_t>(nm, &by, eighth);
      s->d_e_off = dev_alloc<int64_t>(nm, &by, eighth);
      S2G_CUDA(cudaMemcpyAsync(s->d_pan_off, po.data(), sizeof(int64_t) * nm, cudaMemcpyHostToDevice, st));
      S2G_CUDA(cudaMemcpyAsync(s->d_e_off, eo.data(), sizeof(int64_t) * nm, cudaMemcpyHostToDevice, st));
    }
    if (eighth) p8 = dev_alloc<uint8_t>((size_t)(ptot / kS), &by8, true);
    const dim3 grid(nm, (std::max(tb.bl, tb.nt) + kPM - 1) / kPM);
    int64_t *d_woff = nullptr;  // the operators' blocks from W_+
    if (quad) {
      const int64_t woff[2] = {0, (int64_t)(((intptr_t)tb.W[1] - (intptr_t)tb.W[0]) / (intptr_t)sizeof(double))};
      S2G_CUDA(cudaMallocAsync((void **)&d_woff, sizeof woff, st));
      S2G_CUDA(cudaMemcpyAsync(d_woff, woff, sizeof woff, cudaMemcpyHostToDevice, st));
    }
    k_slice_table<<<grid, 128, 0, st>>>(quad ? tb.W[0] : (kind_of_q(kind) ? tb.Q : tb.D), quad ? d_woff : tb.d_off,
                                        tb.bl, tb.nt, tb.an, tmlo, mode, kind_transposed(kind) ? 1 : 0,
                                        fresh ? s->panels : nullptr, p8, s->d_pan_off, s->eA, s->d_e_off);
    S2G_LAUNCHED();
    if (d_woff) cudaFreeAsync(d_woff, st);
    S2G_CUDA(cudaStreamSynchronize(st));
  } catch (const Error &e) {
    if (fresh) s->release();
    cudaFree(p8);
    if (!eighth || e.code != ERR_NOMEM) throw;
    cudaGetLastError();
    refuse(key, false);
    return nullptr;
  }
  if (p8) {
    s->panels8 = p8;
    s->bytes8 = by8;
    g_refused.erase(key);
  }
  s->bytes += by + by8;
  g_mx_bytes += by + by8;
  if (fresh) g_sliced.emplace(key, std::move(made));
  return s;
}

// tiles of one problem (caller holds g_mx_mu); nullptr when a stream capture
// meets an optional one (see sliced)
const TileList *tile_list(SlicedTable &s, int n, int mlo, int mhi, int lmin, bool optional, cudaStream_t st) {
  auto key = std::make_tuple(n, mlo, mhi, lmin);
  auto it = s.lists.find(key);
  if (it != s.lists.end()) return &it->second;
  if (optional && capturing(st)) return nullptr;
  TileList L;
  std::vector<int2> tiles;
  std::vector<int64_t> xoff(mhi - mlo + 1);
  int64_t xe = 0, work = 0;
  for (int m = mlo; m <= mhi; ++m) {
    const Geom g = geom(s.bl, s.nt, s.an, m, s.mode);
    xoff[m - mlo] = xe;
    xe += (int64_t)g.nkc * 16 * kPK;  // per digit slice and 16 columns
    if (g.nl <= 0) continue;
    const int lst = g.l0 > lmin ? g.l0 : lmin;
    int rt0 = 0, kc0 = 0;
    if (s.mode == MX_T2L) {
      if (lst >= s.bl) continue;
      rt0 = (lst - g.l0) / kPM;
    } else if (s.mode == MX_L2T) {
      kc0 = lst >= s.bl ? g.nkc : (lst - g.l0) / kPK;
    }
    for (int rt = rt0; rt < g.nrt; ++rt) {
      tiles.push_back(make_int2(m - mlo, rt));
      work += (int64_t)(g.nkc - kc0) * kPK * kPM;
    }
  }
  size_t by = 0;
  L.ntiles = (int)tiles.size();
  L.d_tiles = dev_alloc<int2>(tiles.size(), &by);
  L.d_xoff = dev_alloc<int64_t>(xoff.size(), &by);
  L.x_elems = xe;
  L.work_entries = work;
  if (!tiles.empty())
    S2G_CUDA(cudaMemcpyAsync(L.d_tiles, tiles.data(), sizeof(int2) * tiles.size(), cudaMemcpyHostToDevice, st));
  S2G_CUDA(cudaMemcpyAsync(L.d_xoff, xoff.data(), sizeof(int64_t) * xoff.size(), cudaMemcpyHostToDevice, st));
  S2G_CUDA(cudaStreamSynchronize(st));
  g_mx_bytes += by;
  s.bytes += by;
  return &s.lists.emplace(key, L).first->second;
}

int num_sms() {
  static const int n = [] {
    int dev = 0, v = 0;
    S2G_CUDA(cudaGetDevice(&dev));
    S2G_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
    return v;
  }();
  return n;
}

int *error_flag() {
  if (!g_err) {
    S2G_CUDA(cudaMalloc(&g_err, sizeof(int)));
    S2G_CUDA(cudaMemset(g_err, 0, sizeof(int)));
  }
  return g_err;
}

struct Problem {
  int kind;     // TableKind
  bool eighth;  // 8 digit slices
  const WignerTable *tb;
  int n, mlo, mhi;
  int nparts;
  Part part[kMaxParts];
  int nb;
};

// a problem's table panels and tiles
struct Prepared {
  SlicedTable *s = nullptr;
  const TileList *L = nullptr;
  int *err = nullptr;
  int lmin = 0;
};

// False (nothing launched) when an optional problem's coefficient panels do
// not fit in device memory.
template <int NC, int S>
bool run_mixed(const Problem &p, const Prepared &pr, cudaStream_t st, int gpl_max) {
  using C = Cfg<NC, S>;
  static const bool attr = [] {  // once per instantiation (thread-safe static initialisation)
    S2G_CUDA(cudaFuncSetAttribute(k_contract_mx<NC, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)C::kSmemBytes));
    return true;
  }();
  (void)attr;
  const int mode = kind_mode(p.kind);
  const SlicedTable *s = pr.s;
  const TileList *L = pr.L;
  int *err = pr.err;
  const int lmin = pr.lmin;
  const int nmp = p.mhi - p.mlo + 1;
  const int mpp = NC / (2 * p.nparts);  // maps per part per launch
  int nkcmax = 0;
  for (int pm = 0; pm < nmp; ++pm) nkcmax = std::max(nkcmax, geom(p.tb->bl, p.tb->nt, p.tb->an, p.mlo + pm, mode).nkc);
  const size_t slice_smem = sizeof(double2) * kMG * (size_t)sv_idx(nkcmax * kPK);
  constexpr int kSliceSmemMax = 232448 - 1024;  // the opt-in maximum less the static arrays
  S2G_REQUIRE(slice_smem <= (size_t)kSliceSmemMax, ERR_INVALID,
              "coefficient slicing: K too large for shared-memory staging");
  static const bool attr_x = [] {
    S2G_CUDA(cudaFuncSetAttribute(k_slice_x<NC, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSliceSmemMax));
    return true;
  }();
  (void)attr_x;
  const int ngroups = (p.nb + mpp - 1) / mpp;
  // map groups run up to gpl_max at a time in one launch (their tiles
  // interleaved, the table read once from HBM and again from L2)
  const int gpl = ngroups < gpl_max ? ngroups : gpl_max;
  // coefficient panels: the tile list's offsets count one slice of 16 columns
  const int64_t x_elems = L->x_elems * (NC / 16 * S);
  const int64_t *xoff = L->d_xoff;
  Scratch scratch(st);
  uint16_t *xpan;
  int *eX;
  if (p.eighth) {
    xpan = scratch.try_get<uint16_t>(x_elems * gpl);
    eX = xpan ? scratch.try_get<int>((int64_t)nmp * NC * gpl) : nullptr;
    if (!eX) return false;
  } else {
    xpan = scratch.get<uint16_t>(x_elems * gpl);
    eX = scratch.get<int>((int64_t)nmp * NC * gpl);
  }
  const double entries = (double)L->work_entries;
  for (int g0 = 0; g0 < ngroups; g0 += gpl) {
    const int ng = ngroups - g0 < gpl ? ngroups - g0 : gpl;
    double fl = 0, by = 0;
    for (int g = g0; g < g0 + ng; ++g) {
      const int b0 = g * mpp;
      const int nbg = p.nb - b0 < mpp ? p.nb - b0 : mpp;
      double xby = 0;
      if (timing_enabled()) {
        fl += 4.0 * entries * nbg * p.nparts;
        by += entries * S + (double)x_elems * 2.0 + 16.0 * nbg * p.nparts * (double)p.tb->nt * nmp;
        xby = (double)x_elems * 2.0 * (1.0 + 8.0 / (2.0 * S));  // panels written + FP64 values read
      }
      XArgs xa{};
      xa.mode = mode;
      xa.bl = p.tb->bl;
      xa.nt = p.tb->nt;
      xa.an = p.tb->an;
      xa.mlo = p.mlo;
      xa.lmin = lmin;
      xa.nparts = p.nparts;
      for (int i = 0; i < p.nparts; ++i) xa.part[i] = p.part[i];
      xa.nb = p.nb;
      xa.b0 = b0;
      xa.mpp = mpp;
      xa.xoff = xoff;
      xa.xpan = xpan + (int64_t)(g - g0) * x_elems;
      xa.eX = eX + (int64_t)(g - g0) * nmp * NC;
      xa.nmp = nmp;
      xa.nkcmax = nkcmax;
      xa.kst = sv_idx(nkcmax * kPK);
      KTimer kx(mode == MX_QUAD ? KC_QUAD : KC_SLICE, st, 0.0, xby);
      k_slice_x<NC, S><<<dim3((nmp + kMG - 1) / kMG, NC / 2), kSliceThreads, slice_smem, st>>>(xa);
      S2G_LAUNCHED();
    }
    if (L->ntiles == 0) continue;
    KTimer kt(mode == MX_QUAD ? KC_QUAD : KC_MIXED, st, fl, by);
    MxArgs ma{};
    ma.mode = mode;
    ma.panels = s->panels;
    ma.panels8 = s->panels8;
    ma.pan_off = s->d_pan_off;
    ma.eA = s->eA;
    ma.e_off = s->d_e_off;
    ma.bl = p.tb->bl;
    ma.nt = p.tb->nt;
    ma.an = p.tb->an;
    ma.tmlo = p.tb->mlo;
    ma.n = p.n;
    ma.mlo = p.mlo;
    ma.lmin = lmin;
    ma.xpan = xpan;
    ma.xoff = xoff;
    ma.eX = eX;
    ma.tiles = L->d_tiles;
    ma.ntiles = L->ntiles;
    ma.nparts = p.nparts;
    for (int i = 0; i < p.nparts; ++i) ma.part[i] = p.part[i];
    ma.nb = p.nb;
    ma.mpp = mpp;
    ma.b0 = g0 * mpp;
    ma.ngroups = ng;
    ma.xg = x_elems;
    ma.eXg = nmp * NC;
    ma.err = err;
    const int nwork = L->ntiles * ng;
    const int grid = nwork < num_sms() ? nwork : num_sms();
    k_contract_mx<NC, S><<<grid, C::kThreads, C::kSmemBytes, st>>>(ma);
    S2G_LAUNCHED();
  }
  return true;
}

// Columns per table pass (2 (re, im) x maps x parts) and map groups per launch.
// Built-in: the smallest of 16 / 32 / 64 columns that holds the whole batch
// (larger batches loop over map groups), 4 groups per launch.  With tuning
// on, the candidates below are timed per (band-limit bucket, column bucket,
// direction) and the fastest kept.
template <int S>
bool run_shapes(const Problem &p, const Prepared &pr, cudaStream_t st) {
  struct Shape {
    int nc, gpl;
  };
  static const Shape kCand[7] = {{16, 1}, {16, 4}, {32, 1}, {32, 4}, {64, 1}, {64, 2}, {64, 4}};
  const int cols = 2 * p.nb * p.nparts;
  const int def = cols <= 16 ? 1 : (cols <= 32 ? 3 : 6);
  static_assert(2 * kMaxParts <= 16, "the narrowest candidate holds a map of every part");
  const auto run = [&](const Shape &sh) {
    if (sh.nc == 16) return run_mixed<16, S>(p, pr, st, sh.gpl);
    if (sh.nc == 32) return run_mixed<32, S>(p, pr, st, sh.gpl);
    return run_mixed<64, S>(p, pr, st, sh.gpl);
  };
  const int c = tuned(TF_MIXED, tune_bucket(p.tb->bl), tune_bucket(cols), p.kind + (S == kSmax ? 4 : 0), 7, def, st,
                      [&](int i) { run(kCand[i]); });
  return run(kCand[c]);
}

// false when the problem's optional table panels are not to be had
bool run_problem(const Problem &p, cudaStream_t st) {
  Prepared pr;
  pr.lmin = p.part[0].lmin;
  for (int i = 1; i < p.nparts; ++i) pr.lmin = std::min(pr.lmin, p.part[i].lmin);
  struct User {  // keeps the panels until the launches are in the stream
    SlicedTable *s = nullptr;
    ~User() {
      if (!s) return;
      std::lock_guard<std::mutex> lk(g_mx_mu);
      --s->users;
    }
  } user;
  {
    std::lock_guard<std::mutex> lk(g_mx_mu);
    pr.s = sliced(*p.tb, p.kind, p.eighth, st);
    if (!pr.s) return false;
    ++pr.s->users;  // before anything else is allocated
    user.s = pr.s;
    if (!p.eighth) pr.s->forward7 = true;
    pr.L = tile_list(*pr.s, p.n, p.mlo, p.mhi, pr.lmin, p.eighth, st);
    if (!pr.L) return false;
    pr.err = error_flag();
    if (capturing(st)) pr.s->captured = true;
  }
  return p.eighth ? run_shapes<kSmax>(p, pr, st) : run_shapes<kS>(p, pr, st);
}

Part part_of(const L2T &a) {
  Part P{};
  P.src = a.x;
  P.ss = a.xs;
  P.x_half = a.x_half ? 1 : 0;
  P.w = a.w;
  P.wscale = a.wscale;
  P.wconj = a.wconj ? 1 : 0;
  P.wkind = a.wkind;
  P.lmin = a.lmin;
  P.dst = a.out;
  P.ds = a.os;
  P.dw = a.ow;
  P.d_mlo = a.omlo;
  return P;
}

Part part_of(const T2L &a) {
  Part P{};
  P.src = a.in;
  P.ss = a.is;
  P.sw = a.iw;
  P.s_mlo = a.imlo;
  P.w = a.w;
  P.wscale = a.wscale;
  P.wconj = a.wconj ? 1 : 0;
  P.wkind = a.wkind;
  P.lmin = a.lmin;
  P.dst = a.y;
  P.ds = a.ys;
  return P;
}

template <class A>
bool same_problem(const A &x, const A &y) {
  return x.tb == y.tb && x.n == y.n && x.use_q == y.use_q && x.mlo == y.mlo && x.mhi == y.mhi && x.nb == y.nb;
}

}  // namespace

namespace {
// The split-precision mode's forward contractions take 7 slices (8 below
// band-limit 128, where double-float would be the alternative); the FP64 mode
// and the adjoints of both modes 8 (accuracy: mixed.h).  Reductions longer than
// 1365, where classes 0-2 could leave the exact range, stay on the FP64 kernels.
// Measured against a 64-bit reference, errors equal the FP64 kernels' to 1 % at L =
// 128 to 1024 (7.6e-13 / 7.5e-13 of f_wav at L = 1024), and px2wav + wav2px of 2 maps
// at L = 1024, N = 4 contracts in 13.0 ms against 64.9 on the FP64 pipe.
constexpr int kMaxK8 = 1365;

template <class A>
bool contract_mixed(const A *a, int nparts, int kind, cudaStream_t st) {
  if (nparts < 1 || nparts > kMaxParts) return false;
  if (a[0].tb->bl < kMinBl8 || a[0].nb <= 0 || a[0].mhi < a[0].mlo) return false;
  for (int i = 1; i < nparts; ++i)
    if (!same_problem(a[0], a[i])) return false;
  Problem p{};
  p.kind = kind;
  p.eighth = t_precision == 0 || kind_transposed(kind) || a[0].tb->bl < kMinBl;
  if (p.eighth && std::max(a[0].tb->bl, a[0].tb->nt) > kMaxK8) return false;
  p.tb = a[0].tb;
  p.n = a[0].n;
  p.mlo = a[0].mlo;
  p.mhi = a[0].mhi;
  p.nb = a[0].nb;
  p.nparts = nparts;
  for (int i = 0; i < nparts; ++i) p.part[i] = part_of(a[i]);
  return run_problem(p, st);
}
}  // namespace

bool contract_l2t_mixed(const L2T *a, int nparts, cudaStream_t st) {
  return contract_mixed(a, nparts, a[0].use_q ? TK_L2T_Q : TK_L2T_D, st);
}
bool contract_t2l_mixed(const T2L *a, int nparts, cudaStream_t st) {
  return contract_mixed(a, nparts, a[0].use_q ? TK_T2L_Q : TK_T2L_D, st);
}

bool quadrature_mixed(const WignerTable &tb, bool trans, const QuadIO *io, int n, int mlo, int mhi, int64_t is, int iw,
                      int i_mlo, int64_t os, int ow, int o_mlo, int nb, cudaStream_t st) {
  if (n < 1 || n > kMaxParts || nb <= 0 || mhi < mlo) return false;
  if (tb.bl < kMinBl8 || std::max(tb.bl, tb.nt) > kMaxK8) return false;
  Problem p{};
  p.kind = trans ? TK_WT : TK_W;
  p.eighth = true;
  p.tb = &tb;
  p.n = tb.an & 1;
  p.mlo = mlo;
  p.mhi = mhi;
  p.nb = nb;
  p.nparts = n;
  for (int i = 0; i < n; ++i) {
    Part &P = p.part[i];
    P.src = io[i].in;
    P.ss = is;
    P.sw = iw;
    P.s_mlo = i_mlo;
    P.wscale = 1.0;
    P.dst = io[i].out;
    P.ds = os;
    P.dw = ow;
    P.d_mlo = o_mlo;
  }
  return run_problem(p, st);
}

void release_sliced_tables() {
  std::lock_guard<std::mutex> lk(g_mx_mu);
  for (auto &kv : g_sliced) kv.second->release();
  g_sliced.clear();
  g_refused.clear();
  g_mx_bytes = 0;
}

size_t optional_panel_bytes() {
  std::lock_guard<std::mutex> lk(g_mx_mu);
  size_t n = 0;
  for (auto &kv : g_sliced) {
    const SlicedTable &s = *kv.second;
    if (s.panels8 && !s.captured) n += s.forward7 ? s.bytes8 : s.bytes;
  }
  return n;
}

int refused_tables() {
  std::lock_guard<std::mutex> lk(g_mx_mu);
  return (int)g_refused.size();
}

cudaError_t device_malloc(void **p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  std::lock_guard<std::mutex> lk(g_mx_mu);
  return give_back_panels() ? cudaMalloc(p, bytes) : e;
}

cudaError_t device_malloc_async(void **p, size_t bytes, cudaStream_t st) {
  const cudaError_t e = cudaMallocAsync(p, bytes, st);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  if (capturing(st)) return e;
  std::lock_guard<std::mutex> lk(g_mx_mu);
  return give_back_panels() ? cudaMallocAsync(p, bytes, st) : e;
}

size_t sliced_table_bytes() {
  std::lock_guard<std::mutex> lk(g_mx_mu);
  return g_mx_bytes;
}

int mixed_error_flag_read_and_clear() {
  std::lock_guard<std::mutex> lk(g_mx_mu);
  if (!g_err) return 0;
  int v = 0;
  S2G_CUDA(cudaMemcpy(&v, g_err, sizeof(int), cudaMemcpyDeviceToHost));
  if (v) S2G_CUDA(cudaMemset(g_err, 0, sizeof(int)));
  return v;
}

}  // namespace s2g
