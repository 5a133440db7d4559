// Explicit time update of one face value, shared by the momentum kernels.
#pragma once

#include "tg_internal.cuh"

namespace tg {

// Explicit time update of one face value u with right-hand side r (UeqnFE,
// ueqn_solvers.c:1411-1442: U = r dt + U_o; UeqnRK4, ueqn_solvers.c:1446-1504,
// stage st: Utmp = U_o + b_st dt r (st = 0) or Utmp + b_st dt r, U = U_o +
// a_{st+1} dt r, after the last stage U = Utmp + b_3 dt r), in the order of
// the reference's VecScale / VecAXPY / VecWAXPY calls.
struct RkArgs {
    double cb, ca;      // b_st dt (FE: dt), a_{st+1} dt
    int first, last, fe;
};
__device__ __forceinline__ void rk_point(double *uc, double *ut, const double *uo, double r, const RkArgs &a)
{
    if (a.fe) { *uc = r * a.cb + *uo; return; }
    if (a.last) { *uc = a.cb * r + *ut; return; }
    const double o = *uo;
    if (a.first) *ut = a.cb * r + o;
    else *ut = *ut + a.cb * r;
    *uc = a.ca * r + o;
}

// resetNonResolvedCellFaces (inline.h:1674-1835) on the + faces of an interior
// cell: the face of the last interior cell of a non-periodic direction keeps
// its right-hand side only for outflow or on a zeroGradient patch
__device__ __forceinline__ void mask_last_faces(const Grid &g, const State &s, const Params &p, int k, int j, int i, int c, R3<double> &o)
{
    if (!g.pi && i == g.mx - 2 && !(p.bc[TG_IRIGHT] == TG_BC_ZERO_GRADIENT || s.ucont_o.x[c] > 0)) o.x = 0.0;
    if (!g.pj && j == g.my - 2 && !(p.bc[TG_JRIGHT] == TG_BC_ZERO_GRADIENT || s.ucont_o.y[c] > 0)) o.y = 0.0;
    if (!g.pk && k == g.mz - 2 && !(p.bc[TG_KRIGHT] == TG_BC_ZERO_GRADIENT || s.ucont_o.z[c] > 0)) o.z = 0.0;
}

}  // namespace tg
