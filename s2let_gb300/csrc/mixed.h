// Legendre/Wigner contractions on the tcgen05 tensor cores by digit slicing.
//
// Every FP64 operand row (a table row, a coefficient column) is written as
// 2^e * sum_{i<S} d_i 2^{-6-7i} with integer digits |d_i| <= 64 held exactly in
// bf16.  The digit products with i + j < S (28 for S = 7, 36 for S = 8) are
// accumulated in FP32 by tcgen05.mma; a class c = i + j sums at most c + 1
// products of magnitude <= 2^12 over K <= 1024 terms, so classes 0..2 are exact
// integers and the rounding of the others sits below 2^-45 of the result.
// S = 7 (split precision): the epilogue combines the classes in double-float;
// truncation error about 2^-41 of max|row| * max|column| per term (measured
// 2.5e-12 normwise on adversarial synthetic rows; the oracle tolerance of the
// path is 1e-10).  S = 8 (FP64 mode, adjoints): combined in integers and rounded
// once, 2^-56 of max|row| * max|column| per term, no more than the rounding of
// an FP64 sum.  A column that holds an infinity or a NaN gives NaN.
#pragma once

#include <cuda_runtime.h>

#include "kernels.h"

namespace s2g {

// True when the contraction ran on the tensor cores; false when the problem is
// outside the kernel's domain (small band-limit, a reduction too long for FP64
// results, no room for the optional table panels) and the caller must run the
// FP64 or double-float kernel.
// nparts (1 or 2) problems that differ only in their coefficients, weights,
// lmin and outputs (scales sharing one band-limit and n) share one pass over
// the table.
bool contract_l2t_mixed(const L2T *a, int nparts, cudaStream_t st);
bool contract_t2l_mixed(const T2L *a, int nparts, cudaStream_t st);

// The quadrature operator W_eps(m) (trans: its transpose) of a recomputed table's
// grid on the ring spectra of n <= kMaxParts problems, m in [mlo, mhi]: in eight
// digit slices, with FP64 rounding error in both modes; false as above.
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
