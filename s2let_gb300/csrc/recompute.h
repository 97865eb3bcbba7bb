// Contractions against recomputed (checkpointed) Wigner tables (WignerTable::rc):
// the same operators as contract_l2t / contract_t2l with the table values
// regenerated in the kernels instead of read from memory.
#pragma once

#include <cuda_runtime.h>

#include "kernels.h"

namespace s2g {

// n problems; those on one table (scales of a band-limit, directions n and -n)
// share the regenerated values and the quadrature's launches
void contract_l2t_rc(const L2T *p, int n, cudaStream_t st);
void contract_t2l_rc(const T2L *p, int n, cudaStream_t st);

// the rescaled recursion of a recomputed table (WignerTable::rec), on the device
RcRec *build_rec(int bl, int an, int mlo, int nm, const int64_t *d_roff, int64_t n);

}  // namespace s2g
