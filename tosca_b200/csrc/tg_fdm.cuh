// Direct solve of the pressure operator on a tensor-product mesh by fast
// diagonalisation (see tg_fdm.cu).
#pragma once

#include "tg_internal.cuh"

namespace tg {

struct Fdm;   // opaque

// the factors of the face coefficients (device arrays):
// aE = kx_i my_j mz_k, aN = mx_i ky_j mz_k, aT = mx_i my_j kz_k
struct FdmOp { const double *kx, *mx, *ky, *my, *kz, *mz; };
// true if the factors reproduce the coefficients to rounding (1e-13), so that
// the operator may be evaluated from them
bool fdm_factors(const Fdm *F, FdmOp *op);

// face coefficients as for mg_create (tg_mg.cuh); on a mesh of planes t, whose
// spacings are the factors, else null. nullptr when the operator does not separate
// or a direction is outside the solver's range; the caller then uses the
// multigrid.
Fdm *fdm_create(tg_ctx *C, const Tensor *t, const double *aE, const double *aN, const double *aT,
                int nx, int ny, int nz, int pi, int pj, int pk);
void fdm_destroy(Fdm *F);

// z with L z = r' up to a constant, L the singular operator without the pin
// and r' = r with its pinned entry (natural index 0) replaced by -sum(r)
// (d_sum[0]); the caller subtracts z[0]. r and z are distinct.
void fdm_apply(tg_ctx *C, Fdm *F, const double *r, const double *d_sum, double *z);

}  // namespace tg
