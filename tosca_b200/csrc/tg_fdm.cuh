// Direct solve of the pressure operator on a tensor-product mesh by fast
// diagonalisation (see tg_fdm.cu).
#pragma once

#include "tg_internal.cuh"

namespace tg {

struct Fdm;   // opaque

// face coefficients as for mg_create (tg_mg.cuh). nullptr when the operator
// does not separate or a direction is outside the solver's range; the caller
// then uses the multigrid.
Fdm *fdm_create(tg_ctx *C, const double *aE, const double *aN, const double *aT,
                int nx, int ny, int nz, int pi, int pj, int pk);
void fdm_destroy(Fdm *F);

// z with L z = r' up to a constant, L the singular operator without the pin
// and r' = r with its pinned entry (natural index 0) replaced by -sum(r)
// (d_sum[0]); the caller subtracts z[0]. r and z are distinct.
void fdm_apply(tg_ctx *C, Fdm *F, const double *r, const double *d_sum, double *z);

}  // namespace tg
