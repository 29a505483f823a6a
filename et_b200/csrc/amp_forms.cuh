// Packed doubles <-> full (v,o,v,o) arrays together with their exchanged form X_aibj -> X_ajbi.
#pragma once

#include "common.cuh"

namespace ccsd {

// For each of nvec packed vectors p (stride n_t2) the symmetric full array S (stride (o v)^2) and
// U_aibj = c1 S_aibj + c2 S_ajbi; either output may be null.  acc_s / acc_u: add instead of overwrite.
// squareup (reordering.F90:4174) and construct_u_aibj (omega_ccsd.F90:881) with c1 = 2, c2 = -1.
void square_forms(Exec &ex, const double *p, int64_t no, int64_t nv, int64_t nvec, double c1, double c2, double *S,
                  double *U, bool acc_s, bool acc_u);

// p[(M, m)] (+)= Z[M, m] + Z[m, M] over M > m, Z[M, M] on the diagonal, for
// Z_aibj = F_aibj + c1 X_aibj + c2 X_ajbi (F or X may be null): eT's symmetric_sum,
// scale_diagonal(1/2) and packin (omega_ccsd.F90:87-102) with the exchange terms of omega_ccsd_c2_d2
// joined (symmetrize_and_pack, packed_array_utilities_r.F90:586).
void sym_pack(Exec &ex, const double *F, const double *X, int64_t no, int64_t nv, int64_t nvec, double c1, double c2,
              double *p, bool accumulate);

}  // namespace ccsd
