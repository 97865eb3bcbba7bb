// Legendre/Wigner contractions on the tcgen05 tensor cores by digit slicing.
//
// Every FP64 operand row (a table row, a coefficient column) is written as
// 2^e * sum_{i<S} d_i 2^{-6-7i} with integer digits |d_i| <= 64 held exactly in
// bf16.  The digit products with i + j < S (28 for S = 7, 36 for S = 8) are
// accumulated in FP32 by tcgen05.mma, each class c = i + j by itself: at most c + 1
// products of magnitude <= 2^12 per term, in units of 2^(-12-7c).
//
// What is lost, in units of max|row| max|column| (the powers of two above them):
//  - values: an entry keeps 48 (S = 7) or 55 (S = 8) bits below its row's or column's
//    power of two, so one that is 2^-k of the largest keeps 55 - k: as good as FP64
//    normwise, not entry by entry; per term 2^-56 for S = 8.
//  - products with i + j >= S: below 6 2^-49 (S = 7), 7 2^-56 (S = 8) per term, of
//    either sign.
//  - the FP32 sums: exact below 2^24.  Classes 0 to 2 are for K <= 1365, class 3 for
//    K <= 1024.  The others could pass 2^24 only if the low digits of row and column
//    agreed in sign and were near 64 over most of the range (class 3 at K = 1365: on
//    average 3072 of 4096 per product); the digits below the leading one of Wigner
//    functions are equidistributed, and their sums stay near 2^17.  If it happened, a
//    rounding would cost 2^-43 K at most, where the roundings of an FP64 sum are bounded
//    by 2^-53 K^2 in all (2^-42.6 K at K = 1365).
// S = 7 (split precision): the epilogue combines the classes in double-float
// (measured 2.5e-12 normwise on adversarial synthetic rows; the oracle tolerance of
// the path is 1e-10).  S = 8 (FP64 mode, adjoints): combined in integers and rounded
// once.  A column that holds an infinity or a NaN gives NaN.
#pragma once

#include <cuda_runtime.h>

#include "kernels.h"

namespace s2g {

// True when the contraction ran on the tensor cores; false when the problem is
// outside the kernel's domain (small band-limit, a reduction too long for FP64
// results, no room for the optional table panels) and the caller must run the
// FP64 or double-float kernel.
// nparts <= kMaxParts problems that differ only in their coefficients, weights,
// lmin and outputs (scales sharing one band-limit and n) share one pass over
// the table.
bool contract_l2t_mixed(const L2T *a, int nparts, cudaStream_t st);
bool contract_t2l_mixed(const T2L *a, int nparts, cudaStream_t st);

// The quadrature operator W_eps(m) (trans: its transpose) of a recomputed table's
// grid on the ring spectra of n <= kMaxParts problems, m in [mlo, mhi]: in eight
// digit slices; false as above.
struct QuadIO {
  const double2 *in;
  double2 *out;
};
bool quadrature_mixed(const WignerTable &tb, bool trans, const QuadIO *io, int n, int mlo, int mhi, int64_t is, int iw,
                      int i_mlo, int64_t os, int ow, int o_mlo, int nb, cudaStream_t st);

void release_sliced_tables();
size_t sliced_table_bytes();
// bytes of optional panels that an allocation may take back (device_malloc)
size_t optional_panel_bytes();
// tables whose optional panels were last refused for want of memory
int refused_tables();
// Reads and clears the device flag raised by a split-precision launch whose
// bounded wait expired (1: pipeline wait, 2: MMA drain); 0 when none did.
int mixed_error_flag_read_and_clear();

// Contraction precision of the calling host thread (0 FP64, 1 split precision).
extern thread_local int t_precision;

}  // namespace s2g
