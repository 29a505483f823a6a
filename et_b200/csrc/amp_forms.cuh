// Packed doubles <-> full (v,o,v,o) arrays together with their exchanged form X_aibj -> X_ajbi.
#pragma once

#include <cuda_bf16.h>

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

// The amplitudes of the A2 ladder (omega_ccsd.F90:113-480) for nvec packed vectors (stride n_t2):
//   t+_cd,ij = (1 - d_cd/2)(1 - d_ij/2)(t_cidj + t_cjdi) over c >= d, i >= j,   t-_cd,ij = t_cidj - t_cjdi
// over c > d, i > j, as K-major columns: column vec n_ij + ij at stride ldp / ldm, cd fastest.
void build_tpm(Exec &ex, const double *t2, int64_t no, int64_t nv, int64_t nvec, double *tp, int64_t ldp, double *tm,
               int64_t ldm);
// the same as np bf16 planes (plane strides plane_p / plane_m) of rows vec n_ij + ij, K positions cd; the
// K positions beyond the pairs and the rows beyond nvec n_ij (up to rows_p / rows_m) are cleared
void build_tpm_planes(Exec &ex, const double *t2, int64_t no, int64_t nv, int64_t nvec, int np, __nv_bfloat16 *tp,
                      int64_t rows_p, int64_t ldp, __nv_bfloat16 *tm, int64_t rows_m, int64_t ldm);

// Omega_aibj += w+ + w-, Omega_ajbi += w+ - w- (add_double_packed_plus_minus, omega_ccsd.F90:440-458) for
// a in [a0, a1), b <= a, i >= j and nvec vectors: w+ column vec n_ij + ij at stride ldwp, row
// a(a+1)/2 + b minus that of (a0, 0); w- over a > b, i > j likewise.
void add_omega_pm(Exec &ex, double *om2, const double *wp, const double *wm, int64_t no, int64_t nv, int64_t nvec,
                  int64_t a0, int64_t a1, int64_t ldwp, int64_t ldwm);

}  // namespace ccsd
