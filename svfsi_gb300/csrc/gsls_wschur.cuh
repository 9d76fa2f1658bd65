// CGRAD_SCHUR on the row partition (gsls_wschur.cu).
#pragma once

#include "gsls_internal.cuh"

namespace gsls {

// Schur CG scalar block (CGRAD_SCHUR, CGRAD.f:51-123)
struct SchurScal {
  double err, errO, eps, dot, iNorm2;
  int done, suc, itr, mItr;
};
static_assert(sizeof(SchurScal) <= kScalRed, "scalar block");

// Lays out the operands of the Schur products (mG 3x1, Gt 1x3, mL per CSR
// block) for the kernel; *fits false when the partition does not fit.
template <class VT>
int wschur_pack(gsls_lhs *lhs, const VT *mG, const VT *Gt, const VT *mL, bool *fits);
// P in: right-hand side, out: solution; scalars in *out (done 4: a wait ran out)
template <class VT, class XT>
int wschur_run(gsls_lhs *lhs, const gsls_sub_ls *ls, XT *P, SchurScal *out);

}  // namespace gsls
