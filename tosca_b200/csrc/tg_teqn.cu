// Temperature transport (SolveTEqn, teqn.c:259-276) with the explicit RK4
// scheme (TeqnRK4, teqn_solvers.c:759-818): FormT (teqn_solvers.c:6-594)
// evaluates per face the WENO3 convective flux -V^q weno3(T) and the diffusive
// flux (g^{q1} dT/dcsi + g^{q2} dT/deta + g^{q3} dT/dzeta) ajc kappa_eff, the
// cell budget times aj forms the right-hand side. kappa_eff = nu/Pr without
// LES; with Smagorinsky the molecular part is dropped and kappa_eff = nu_t/Pr_t
// with the stability-corrected Pr_t = 1/(1 + 2 l/delta), delta = (1/ajc)^(1/3),
// l = min(delta, 7.6 nu_t/delta sqrt(tRef/|g dT/deta|)) in stable
// stratification (teqn_solvers.c:180-195). Boundary ghosts follow
// UpdateTemperatureBCs (boundary.c:2052-2616) for zeroGradient, fixedValue,
// fixedGradient, periodic and (zero-gradient) thetaWallFunction patches; the
// thetaWallFunction's heat flux (UpdateWallModelsT, boundary.c:3858-4178)
// replaces the diffusive flux of the jLeft wall faces. FP64 in every
// precision mode.
#include <algorithm>
#include <cmath>

#include "tg_internal.cuh"
#include "tg_mo.cuh"

namespace tg {

namespace {

inline dim3 gint(const Grid &g) { return grid3(g.mx - 2, g.my - 2, g.mz - 2); }
inline int nblk(int64_t n) { int64_t b = (n + 255) / 256; return (int)(b < 148 * 16 ? b : 148 * 16); }

// weno3, inline.h:5147-5180, with the weights in one division:
// w0 = alpha0 / (alpha0 + alpha1) with alpha_q = d_q / (eps + beta_q)^2 is
// d0 s1^2 / (d0 s1^2 + d1 s0^2), s_q = eps + beta_q (same value up to
// rounding; a double division or library pow call costs tens of instructions)
__device__ __forceinline__ double weno3(double f0, double f1, double f2, double f3, double wavespeed)
{
    double fL, fC, fR;
    if (wavespeed > 0) { fL = f0; fC = f1; fR = f2; }
    else { fL = f3; fC = f2; fR = f1; }
    const double d0 = 2. / 3., d1 = 1. / 3., eps = 1.e-6;
    const double s0 = eps + (fC - fR) * (fC - fR), s1 = eps + (fL - fC) * (fL - fC);
    const double A = d0 * (s1 * s1), B = d1 * (s0 * s0);
    const double u0 = (fC * 0.5 + fR * 0.5), u1 = (-fL * 0.5 + fC * 1.5);
    return (A * u0 + B * u1) / (A + B);
}

// kappa_eff at a face (teqn_solvers.c:164-214); dtde: the face's eta
// derivative. With Smagorinsky, nu_t / Pr_t with Pr_t = 1 / (1 + 2 l/delta)
// and, in stable stratification, l/delta = min(1, 7.6 nu_t sqrt(tRef/|g
// dT/deta|) / delta^2), delta = (1/ajc)^(1/3): evaluated as nu_t (1 + 2
// l/delta) with rd2 = 1/delta^2 from the mesh (k_t_width: no cube root per face
// and stage) and one reciprocal square root
__device__ __forceinline__ double kappa_eff(const Params &p, double nut, double dtde, double rd2, double sqt)
{
    if (!p.les) return p.nu / p.prandtl;
    const double gradTdotG = dtde * (-9.81);
    double ratio = 1.0;                                    // l / delta
    if (gradTdotG < 0.) ratio = fmin(1.0, 7.6 * nut * rd2 * (sqt * rsqrt(-gradTdotG)));
    return nut * (1.0 + 2.0 * ratio);
}

// 4-cell stencil ends of a face (getFace2Cell4Stencil*, inline.h:2190-2380)
__device__ __forceinline__ void stencil4(int i, int m, int per, int &L, int &R)
{
    if (i == 0 || i == m - 2) {
        if (per && i == m - 2) { R = m + 2; L = i - 1; }
        else if (per && i == 0) { L = -3; R = i + 2; }
        else if (i == 0) { L = i; R = i + 2; }
        else { L = i - 1; R = i + 1; }
    } else { L = i - 1; R = i + 2; }
}

// pass 1: the flux at the faces of the interior cells, convective plus diffusive
// (mode 0), convective (1) or diffusive (2). A block takes 32 x 8 columns of
// interior cells and marches along k; a thread forms the i, j and k faces on its
// cell's + side, and a cell next to a non-periodic 0 boundary also the face on
// its - side (face 0; face 0 of a periodic direction is read from face m-2 by
// the budget and is not formed). T and nut are read from a ring of six planes in
// shared memory with one cell below and two above in i and j; plane k + 4 is
// copied while plane k is worked on, one barrier per plane. Bound by instruction
// issue and by the latency of the divisions: a launch takes three to five times what
// its 64 (planes) to 160 (curvilinear) bytes per cell do. A step of 192 x 96 x 96
// (curvilinear) takes 3.43 ms and one of 128 x 128 x 64 0.875; with blocks of
// 32 x 4 x 2 cells that stage 35 x 7 x 5 points each, 3.52 and 0.890.
// The WENO points of the boundary faces, which may lie outside the tile (periodic
// i = mx + 2 and i = -3), are read from global memory.
//
// AX: a mesh of planes: the metric tensor of a face is its normal component
// squared, and with aj a product of spacings (tg_tensor.cu, t), so no metric is
// read; the cross terms are left out with the derivatives they multiply;
// kappa_eff still reads the eta derivative of every face (the stability
// correction of Pr_t). Elsewhere the products of the metric tensor with the face
// Jacobian are SetCoeffMatrix's arrays (9 values per cell, the face metrics 30).
// rd2: 1/delta^2 of the i, j and k faces (k_t_width), on a
// mesh of planes a product of factors as well.
constexpr int TBX = 32, TBY = 8, TBN = TBX * TBY;
constexpr int TTX = TBX + 3, TTY = TBY + 3, TTN = TTX * TTY, TRING = 6;

template <bool AX, int mode>
__global__ void __launch_bounds__(TBN, 4) k_t_face_fluxes(const __grid_constant__ Grid g, const __grid_constant__ Metrics m, const __grid_constant__ Tensor t,
                                                          const __grid_constant__ State s, const __grid_constant__ Params p, V3f<double> rd2, V3f<double> fl,
                                                          int nbi, int nbj, int kc)
{
    __shared__ double ring[TRING * 2 * TTN];         // per plane T, then nut
    const int mx = g.mx, my = g.my, mz = g.mz, pl = mx * my;
    const int br = blockIdx.x / nbi;
    const int i0 = 1 + (blockIdx.x % nbi) * TBX, j0 = 1 + (br % nbj) * TBY, k0 = 1 + (br / nbj) * kc, k1 = min(k0 + kc - 1, mz - 2);
    // what this thread copies of every plane: elements tid and tid + TBN of the
    // tile (DMDA i0 - 1 + x, j0 - 1 + y; points outside the domain are never used
    // and read the plane's first element)
    const int tid = threadIdx.y * TBX + threadIdx.x;
    static_assert(TTN <= 2 * TBN, "two elements per thread");
    int off[2];
    #pragma unroll
    for (int q = 0; q < 2; q++) {
        const int e = tid + q * TBN, ti = i0 - 1 + e % TTX, tj = j0 - 1 + e / TTX;
        off[q] = ti < mx && tj < my ? tj * mx + ti : 0;
    }
    const bool les = p.les, two = tid < TTN - TBN;
    // plane q into a slot of the ring
    auto load = [&](int q, double *d) {
        if (q <= mz - 1) {
            const int o = q * pl;
            d += tid;
            cp_async8(d, s.tmprt + o + off[0]);
            if (mode != 1 && les) cp_async8(d + TTN, s.nut + o + off[0]);
            if (two) {
                cp_async8(d + TBN, s.tmprt + o + off[1]);
                if (mode != 1 && les) cp_async8(d + TBN + TTN, s.nut + o + off[1]);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    #pragma unroll
    for (int q = 0; q < 5; q++) load(k0 - 1 + q, ring + q * 2 * TTN);
    const int i = i0 + threadIdx.x, j = j0 + threadIdx.y;
    const bool on = i <= mx - 2 && j <= my - 2;
    const int t0 = (threadIdx.y + 1) * TTX + threadIdx.x + 1;
    int slot = 0;                                    // of plane k - 1
    const bool npi = !g.pi, npj = !g.pj, npk = !g.pk;
    const int ni = (i == 1 && npi) ? 2 : 1, nj = (j == 1 && npj) ? 2 : 1;
    auto TG = [&](int kk, int jj, int ii) { return s.tmprt[g.id(kk, jj, ii)]; };
    const double sqt = sqrt(p.t_ref);
    // the column's factors of 1/delta^2 (q) and of the diffusion (w) at the faces E, N, T
    const bool ax = AX && on;
    const double qE = ax && les ? t.rqyf[i] * t.rqz[j] : 0.0, qN = ax && les ? t.rqy[i] * t.rqzf[j] : 0.0, qT = ax && les ? t.rqy[i] * t.rqz[j] : 0.0;
    const double wE = ax ? t.dz[j] * t.rdyf[i] : 0.0, wN = ax ? t.dy[i] * t.rdzf[j] : 0.0, wT = ax ? t.dy[i] * t.dz[j] : 0.0;
    // plane k + 2 is there when all but the newest copy have arrived
    for (int k = k0; k <= k1; k++, slot = slot == TRING - 1 ? 0 : slot + 1) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        auto plane = [&](int d) { const int q = slot + d; return ring + (q >= TRING ? q - TRING : q) * (2 * TTN); };
        load(k + 4, plane(5));
        if (!on) continue;
        const double *const Pm = plane(0) + t0, *const P0 = plane(1) + t0, *const P1 = plane(2) + t0, *const P2 = plane(3) + t0;
        auto T = [&](int dk, int dj, int di) { return (dk < 0 ? Pm : dk == 0 ? P0 : P1)[dj * TTX + di]; };
        auto NUT = [&](int dj, int di) { return P0[TTN + dj * TTX + di]; };
        const double rqx = AX && les ? t.rqx[k] : 0.0, dx = AX ? t.dx[k] : 0.0;
        // A derivative along a face is central except, on a face of the boundary, at
        // the two ends of its direction when either is not periodic.

        // ---- i face fi = i + e (Compute_dscalar_i, inline.h:3210-3247)
        auto iface = [&](int fi, int e) {
            const int f = g.lin(k, j, fi);
            const double dtdc = T(0, 0, e + 1) - T(0, 0, e);
            double dtde = (T(0, 1, e + 1) + T(0, 1, e) - T(0, -1, e + 1) - T(0, -1, e)) * 0.25, dtdz = 0.0, o = 0.0;
            if (!AX) dtdz = (T(1, 0, e + 1) + T(1, 0, e) - T(-1, 0, e + 1) - T(-1, 0, e)) * 0.25;
            const double uc = mode != 2 ? s.ucont.x[f] : 0.0;
            if (fi == 0 || fi == mx - 2) {
                if (npj || npi) {
                    if (j == my - 2)   dtde = (T(0, 0, e + 1) + T(0, 0, e) - T(0, -1, e + 1) - T(0, -1, e)) * 0.5;
                    else if (j == 1)   dtde = (T(0, 1, e + 1) + T(0, 1, e) - T(0, 0, e + 1) - T(0, 0, e)) * 0.5;
                }
                if (!AX && (npk || npi)) {
                    if (k == mz - 2)   dtdz = (T(0, 0, e + 1) + T(0, 0, e) - T(-1, 0, e + 1) - T(-1, 0, e)) * 0.5;
                    else if (k == 1)   dtdz = (T(1, 0, e + 1) + T(1, 0, e) - T(0, 0, e + 1) - T(0, 0, e)) * 0.5;
                }
                if (mode != 2) {
                    int iL, iR;
                    stencil4(fi, mx, g.pi, iL, iR);
                    o = -uc * weno3(TG(k, j, iL), T(0, 0, e), T(0, 0, e + 1), TG(k, j, iR), uc);
                }
            } else if (mode != 2) o = -uc * weno3(T(0, 0, e - 1), T(0, 0, e), T(0, 0, e + 1), T(0, 0, e + 2), uc);
            if (mode == 1) { fl.x[f] = o; return; }
            const double wd = !les ? 0.0 : AX ? rqx * (e == 0 ? qE : t.rqyf[0] * t.rqz[j]) : rd2.x[f];
            const double ke = kappa_eff(p, les ? 0.5 * (NUT(0, e) + NUT(0, e + 1)) : 0.0, dtde, wd, sqt);
            if (AX) {
                fl.x[f] = o + (dx * (e == 0 ? wE : t.dz[j] * t.rdyf[0]) * dtdc) * ke;
            } else {
                double a = 0.0, b = 0.0, c = 0.0;
                if (e == 0) { a = m.g11[f]; b = m.g12[f]; c = m.g13[f]; }
                else {                       // face 0 has its own metrics
                    const R3<double> n = ld3(m.icsi, f);
                    const double w = m.iaj[f];
                    a = dot3(ld3(m.icsi, f), n) * w; b = dot3(ld3(m.ieta, f), n) * w; c = dot3(ld3(m.izet, f), n) * w;
                }
                fl.x[f] = o + (a * dtdc + b * dtde + c * dtdz) * ke;
            }
        };
        // ---- j face fj = j + e (Compute_dscalar_j, inline.h:3252-3289)
        auto jface = [&](int fj, int e) {
            const int f = g.lin(k, fj, i);
            const double dtde = T(0, e + 1, 0) - T(0, e, 0);
            double dtdc = 0.0, dtdz = 0.0, o = 0.0;
            if (!AX) {
                dtdc = (T(0, e + 1, 1) + T(0, e, 1) - T(0, e + 1, -1) - T(0, e, -1)) * 0.25;
                dtdz = (T(1, e + 1, 0) + T(1, e, 0) - T(-1, e + 1, 0) - T(-1, e, 0)) * 0.25;
            }
            const double uc = mode != 2 ? s.ucont.y[f] : 0.0;
            if (fj == 0 || fj == my - 2) {
                if (!AX && (npi || npj)) {
                    if (i == mx - 2)   dtdc = (T(0, e + 1, 0) + T(0, e, 0) - T(0, e + 1, -1) - T(0, e, -1)) * 0.5;
                    else if (i == 1)   dtdc = (T(0, e + 1, 1) + T(0, e, 1) - T(0, e + 1, 0) - T(0, e, 0)) * 0.5;
                }
                if (!AX && (npk || npj)) {
                    if (k == mz - 2)   dtdz = (T(0, e + 1, 0) + T(0, e, 0) - T(-1, e + 1, 0) - T(-1, e, 0)) * 0.5;
                    else if (k == 1)   dtdz = (T(1, e + 1, 0) + T(1, e, 0) - T(0, e + 1, 0) - T(0, e, 0)) * 0.5;
                }
                if (mode != 2) {
                    int jL, jR;
                    stencil4(fj, my, g.pj, jL, jR);
                    o = -uc * weno3(TG(k, jL, i), T(0, e, 0), T(0, e + 1, 0), TG(k, jR, i), uc);
                }
            } else if (mode != 2) o = -uc * weno3(T(0, e - 1, 0), T(0, e, 0), T(0, e + 1, 0), T(0, e + 2, 0), uc);
            if (mode == 1) { fl.y[f] = o; return; }
            const double wd = !les ? 0.0 : AX ? rqx * (e == 0 ? qN : t.rqy[i] * t.rqzf[0]) : rd2.y[f];
            double ke = kappa_eff(p, les ? 0.5 * (NUT(e, 0) + NUT(e + 1, 0)) : 0.0, dtde, wd, sqt);
            double v0 = 0.0;
            if (p.t_wall && fj == 0) {
                // thetaWallFunction (teqn_solvers.c:337-352): the modelled flux
                // -qWall . jEta, qWall = (0, 0, q), replaces the diffusive one
                const R3<double> et = ld3(m.jeta, f);
                v0 = -1.0 * (0.0 * et.x + 0.0 * et.y + s.qwall[k * mx + i] * et.z);
                ke = 0.0;
            }
            if (AX) {
                fl.y[f] = o + (v0 + (dx * (e == 0 ? wN : t.dy[i] * t.rdzf[0]) * dtde) * ke);
            } else {
                double a = 0.0, b = 0.0, c = 0.0;
                if (e == 0) { a = m.g21[f]; b = m.g22[f]; c = m.g23[f]; }
                else {                       // face 0 has its own metrics
                    const R3<double> n = ld3(m.jeta, f);
                    const double w = m.jaj[f];
                    a = dot3(ld3(m.jcsi, f), n) * w; b = dot3(ld3(m.jeta, f), n) * w; c = dot3(ld3(m.jzet, f), n) * w;
                }
                fl.y[f] = o + (v0 + (a * dtdc + b * dtde + c * dtdz) * ke);
            }
        };
        // ---- k face fk = k + e (Compute_dscalar_k, inline.h:3294-3331). A and B: the
        // planes of its two cells, Z and C: those before and after
        auto kface = [&](int fk, int e, const double *Z, const double *A, const double *B, const double *C) {
            const int f = g.lin(fk, j, i);
            double dtdc = 0.0, dtde = (B[TTX] + A[TTX] - B[-TTX] - A[-TTX]) * 0.25, o = 0.0;
            if (!AX) dtdc = (B[1] + A[1] - B[-1] - A[-1]) * 0.25;
            const double dtdz = B[0] - A[0], uc = mode != 2 ? s.ucont.z[f] : 0.0;
            if (fk == 0 || fk == mz - 2) {
                if (!AX && (npi || npk)) {
                    if (i == mx - 2)   dtdc = (B[0] + A[0] - B[-1] - A[-1]) * 0.5;
                    else if (i == 1)   dtdc = (B[1] + A[1] - B[0] - A[0]) * 0.5;
                }
                if (npj || npk) {
                    if (j == my - 2)   dtde = (B[0] + A[0] - B[-TTX] - A[-TTX]) * 0.5;
                    else if (j == 1)   dtde = (B[TTX] + A[TTX] - B[0] - A[0]) * 0.5;
                }
                if (mode != 2) {
                    int kL, kR;
                    stencil4(fk, mz, g.pk, kL, kR);
                    o = -uc * weno3(TG(kL, j, i), A[0], B[0], TG(kR, j, i), uc);
                }
            } else if (mode != 2) o = -uc * weno3(Z[0], A[0], B[0], C[0], uc);
            if (mode == 1) { fl.z[f] = o; return; }
            const double wd = !les ? 0.0 : AX ? t.rqxf[fk] * qT : rd2.z[f];
            const double ke = kappa_eff(p, les ? 0.5 * (A[TTN] + B[TTN]) : 0.0, dtde, wd, sqt);
            if (AX) {
                fl.z[f] = o + (wT * t.rdxf[fk] * dtdz) * ke;
            } else {
                double a = 0.0, b = 0.0, c = 0.0;
                if (e == 0) { a = m.g31[f]; b = m.g32[f]; c = m.g33[f]; }
                else {                       // face 0 has its own metrics
                    const R3<double> n = ld3(m.kzet, f);
                    const double w = m.kaj[f];
                    a = dot3(ld3(m.kcsi, f), n) * w; b = dot3(ld3(m.keta, f), n) * w; c = dot3(ld3(m.kzet, f), n) * w;
                }
                fl.z[f] = o + (a * dtdc + b * dtde + c * dtdz) * ke;
            }
        };
#pragma unroll 1
        for (int e = 0; e > -ni; e--) iface(i + e, e);
#pragma unroll 1
        for (int e = 0; e > -nj; e--) jface(j + e, e);
        kface(k, 0, Pm, P0, P1, P2);
        if (k == 1 && npk) kface(0, -1, Pm, Pm, P0, P1);      // its outer points are not in the ring
    }
}

// FormT pass 1 on the context's stream
template <int mode>
void t_face_fluxes(tg_ctx *C)
{
    const Grid g = C->g;
    const int nbi = (g.mx - 2 + TBX - 1) / TBX, nbj = (g.my - 2 + TBY - 1) / TBY, nk = g.mz - 2;
    // planes per block: every chunk costs about three planes of start-up, every
    // started wave of four blocks per SM a chunk
    int kc = nk;
    int64_t best = INT64_MAX;
    for (int ch = 1; ch <= std::max(1, nk / 2); ch++) {
        const int c = (nk + ch - 1) / ch;
        const int64_t waves = ((int64_t)nbi * nbj * ((nk + c - 1) / c) + 4 * 148 - 1) / (4 * 148), cost = waves * (c + 3);
        if (cost < best) { best = cost; kc = c; }
    }
    const dim3 gr(nbi * nbj * ((nk + kc - 1) / kc)), bl(TBX, TBY);
    State &s = C->s;
    if (C->axis_aligned)
        TG_PROF(C, "teqn_face_fluxes", (k_t_face_fluxes<true, mode><<<gr, bl, 0, C->stream>>>(g, C->m, C->ts, s, C->prm, s.trd2, s.tflux, nbi, nbj, kc)));
    else
        TG_PROF(C, "teqn_face_fluxes", (k_t_face_fluxes<false, mode><<<gr, bl, 0, C->stream>>>(g, C->m, C->ts, s, C->prm, s.trd2, s.tflux, nbi, nbj, kc)));
}

// pass 2 (teqn_solvers.c:520-566): the flux budget of interior cell c times aj,
// face 0 of a periodic direction read from face m-2 (resetFacePeriodicFluxesVector)
__device__ __forceinline__ double t_budget(const Grid &g, const V3f<double> &fl, int k, int j, int i, int c)
{
    const int pl = g.mx * g.my;
    const int iw = (i == 1 && g.pi) ? c + g.mx - 3 : c - 1;
    const int js = (j == 1 && g.pj) ? c + (g.my - 3) * g.mx : c - g.mx;
    const int kb = (k == 1 && g.pk) ? c + (g.mz - 3) * pl : c - pl;
    return fl.x[c] - fl.x[iw] + fl.y[c] - fl.y[js] + fl.z[c] - fl.z[kb];
}
__global__ void k_t_rhs(Grid g, Metrics m, V3f<double> fl, double *rhs)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1, k = blockIdx.z * blockDim.z + threadIdx.z + 1;
    if (i > g.mx - 2 || j > g.my - 2 || k > g.mz - 2) return;
    const int c = g.lin(k, j, i);
    rhs[c] = t_budget(g, fl, k, j, i, c) * m.aj[c];
}

// pass 2 with the RK4 bookkeeping after stage st: Ttmp (+)= dt b Rhs, next stage
// T = T_o + a dt Rhs, last T = Ttmp. The right-hand side is zero off the
// interior, so T keeps its T_o there but for the periodic ghosts, which a cell
// writes with its own value (resetCellPeriodicFluxes). 80 bytes per cell where
// the budget, the update of every point and the ghost copies moved 152 in up to
// five launches.
__global__ void k_t_rk(Grid g, Metrics m, V3f<double> fl, double *t, const double *to, double *ttmp, double cb, double ca, int first, int last)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1, k = blockIdx.z * blockDim.z + threadIdx.z + 1;
    if (i > g.mx - 2 || j > g.my - 2 || k > g.mz - 2) return;
    const int c = g.lin(k, j, i);
    const double r = t_budget(g, fl, k, j, i, c) * m.aj[c], o = (first || !last) ? to[c] : 0.0;
    const double tt = (first ? o : ttmp[c]) + cb * r;
    double v = tt;
    if (!last) { ttmp[c] = tt; v = ca * r + o; }
    t[c] = v;
    auto image = [](int l, int mm, int per) { return !per ? l : l == 1 ? mm - 1 : l == mm - 2 ? 0 : l; };
    const int gi = image(i, g.mx, g.pi), gj = image(j, g.my, g.pj), gk = image(k, g.mz, g.pk);
    if (gi == i && gj == j && gk == k) return;
    for (int b = 1; b < 8; b++) {
        if (((b & 1) && gi == i) || ((b & 2) && gj == j) || ((b & 4) && gk == k)) continue;
        t[g.lin((b & 4) ? gk : k, (b & 2) ? gj : j, (b & 1) ? gi : i)] = v;
    }
}

// 1/delta^2 = ajc^(2/3) of every face of an interior cell
__global__ void k_t_width(Grid g, Metrics m, V3f<double> rd2)
{
    const int64_t n = g.size();
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const double a = cbrt(m.iaj[q]), b = cbrt(m.jaj[q]), c = cbrt(m.kaj[q]);
        rd2.x[q] = a * a; rd2.y[q] = b * b; rd2.z[q] = c * c;
    }
}

// TeqnABBE steps 3-5 (teqn_solvers.c:835-880): bT = 3/2 Conv - 1/2 Conv_o
// (Conv on the first step), b = dt bT (zero off the interior) + T_o, and the
// guess x = b
__global__ void k_t_abbe_b(int64_t n, double *b, double *x, const double *conv, const double *conv_o, const double *to,
                           double dt, int ab2)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        double bt = 0.0;
        if (ab2) { bt = bt + 1.5 * conv[q]; bt = bt + -0.5 * conv_o[q]; }
        else bt = bt + 1.0 * conv[q];
        const double v = bt * dt + 1.0 * to[q];
        b[q] = v;
        x[q] = v;
    }
}

// SNESFuncEvalT tail (teqn_solvers.c:688-711): F = dt FormT(T) (zero off the
// interior) - T + T_o, or with BDF2 - 3/2 T + 2 T_o - 1/2 T_oo
__global__ void k_t_snes_f(int64_t n, double *F, const double *rhs, const double *t, const double *to, const double *too,
                           double dt, int bdf2)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        double r = rhs[q] * dt;
        if (bdf2) { r = r + (-3.0 / 2.0) * t[q]; r = r + 2.0 * to[q]; r = r + (-1.0 / 2.0) * too[q]; }
        else { r = r + -1.0 * t[q]; r = r + 1.0 * to[q]; }
        F[q] = r;
    }
}

// ABBEMatVec tail (teqn_solvers.c:930-943): Av = v - dt D(v), D(v) zero off the interior
__global__ void k_t_abbe_av(int64_t n, double *Av, const double *v, const double *d, double dt)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
        Av[q] = v[q] + -1.0 * (d[q] * dt);
}

// UpdateTemperatureBCs (boundary.c:2052-2616) on the face ghosts of one patch
// pair (blockIdx.z: 0 i, 1 j, 2 k), from the interior next to them: no ghost is
// read, so the three directions share a launch
__global__ void k_t_bcs(Grid g, Metrics m, Params p, double *t, const double *series_st, const double *d_it, double it_start)
{
    const int dir = blockIdx.z;
    const int a = blockIdx.x * blockDim.x + threadIdx.x + 1, b = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int na = dir == 0 ? g.my : g.mx, nb = dir == 2 ? g.my : g.mz;
    if (a > na - 2 || b > nb - 2) return;
    const int mdir = dir == 0 ? g.mx : (dir == 1 ? g.my : g.mz);
    auto at = [&](int l) { return dir == 0 ? g.lin(b, a, l) : (dir == 1 ? g.lin(b, l, a) : g.lin(l, b, a)); };
    const V3f<double> &S = dir == 0 ? m.csi : (dir == 1 ? m.eta : m.zet);
    for (int side = 0; side < 2; side++) {
        const int patch = 2 * dir + side;
        const int ci = side == 0 ? 1 : mdir - 2, gh = side == 0 ? 0 : mdir - 1;
        const int c = at(ci), q = at(gh);
        const int type = p.t_bc[patch];
        if (type == TG_TBC_WALL_FUNCTION && patch == TG_JLEFT && p.t_wall == TG_TWALL_SURFACE_SERIES && series_st &&
            d_it[0] != it_start)
            t[q] = 2.0 * series_st[0] - t[c];        // -4 after the first step, boundary.c:2392-2408
        else if (type == TG_TBC_ZERO_GRADIENT || type == TG_TBC_WALL_FUNCTION) t[q] = t[c];
        else if (type == TG_TBC_FIXED_VALUE) t[q] = p.t_bc_value[patch];
        else if (type == TG_TBC_FIXED_GRADIENT) {
            const double area = sqrt(S.x[c] * S.x[c] + S.y[c] * S.y[c] + S.z[c] * S.z[c]);
            const double d = (1.0 / m.aj[c]) / area;
            t[q] = d * p.t_bc_value[patch] + t[c];
        } else {
            t[q] = t[at(side == 0 ? mdir - 2 : 1)];   // periodic: the opposite interior cell
        }
    }
}

// ---- UpdateWallModelsT, jLeft thetaWallFunction (boundary.c:3858-4178) ----
// wall-parallel velocity magnitude and wall distance 0.5 / (aj |eta|) of the
// wall cell (k, 1, i)
__device__ __forceinline__ void twall_cell(Grid g, Metrics m, State s, int k, int i, double &upm, double &dist)
{
    const int c = g.lin(k, 1, i);
    R3<double> n;
    const R3<double> et = ld3(m.eta, c);
    calc_normal(ld3(m.csi, c), et, ld3(m.zet, c), 1, n);
    const R3<double> U = ld3(s.ucat, c);
    const R3<double> Up = U - dot3(U, n) * n;
    upm = sqrt(dot3(Up, Up));
    dist = 0.5 / m.aj[c] / sqrt(dot3(et, et));
}

// -4: the surface temperature at the clock time of the step, t_start + (it -
// it_start) dt + dt (clock.c:366), interpolated in the series as
// findInterpolationWeights does (inline.h:5873-5940: the two nearest points,
// points within a relative 1e-5 of the nearer one's distance skipped,
// extrapolating beyond the ends); one thread, out[0]
__global__ void k_twall_series(const double *tv, const double *vv, int n, const double *d_it, double it_start, double t_start,
                               double dt, double *out)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    if (n < 2 || !tv || !vv) { out[0] = 0.0; return; }     // no series: not launched by the host
    const double pval = t_start + (d_it[0] - it_start) * dt + dt;
    const double eqTol = 1e-5;
    int i1 = 0, i2 = 1;
    for (int q = 0; q < n; q++) {
        const double dq = fabs(tv[q] - pval);
        const double tol1 = fabs(dq - fabs(tv[i2] - pval)) / dq;
        if (dq < fabs(tv[i1] - pval) && tol1 > eqTol) { i2 = i1; i1 = q; }
        const double tol2 = fabs(dq - fabs(tv[i1] - pval)) / dq;
        if (dq < fabs(tv[i2] - pval) && q != i1 && tol2 > eqTol) i2 = q;
    }
    if (tv[i2] < tv[i1]) { const int t = i1; i1 = i2; i2 = t; }
    const double idx = (double)(i2 - i1) / (tv[i2] - tv[i1]) * (pval - tv[i1]) + (double)i1;
    const double w0 = ((double)i2 - idx) / (double)(i2 - i1), w1 = (idx - (double)i1) / (double)(i2 - i1);
    out[0] = w0 * vv[i1] + w1 * vv[i2];
}

// -3, first call: surfaceTheta = the wall value 0.5 (T(j=1) + T(j=0))
__global__ void k_twall_seed(Grid g, State s)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, k = blockIdx.y * blockDim.y + threadIdx.y + 1;
    if (i > g.mx - 2 || k > g.mz - 2) return;
    s.surf_theta[k * g.mx + i] = 0.5 * (s.tmprt[g.lin(k, 1, i)] + s.tmprt[g.lin(k, 0, i)]);
}

// -3 localized: surfaceTheta += heatingRate dt, then qWallShumann per cell
__global__ void k_twall_local(Grid g, Metrics m, State s, Params p, const double *sts)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, k = blockIdx.y * blockDim.y + threadIdx.y + 1;
    if (i > g.mx - 2 || k > g.mz - 2) return;
    const int w = k * g.mx + i;
    double upm, dist;
    twall_cell(g, m, s, k, i, upm, dist);
    double st;
    if (sts) st = sts[0];
    else { st = s.surf_theta[w] + p.tw_heating * p.dt; s.surf_theta[w] = st; }
    s.qwall[w] = mo::qwall(upm, dist, p.tw_z0, p.tw_gamma_m, p.tw_gamma_h, p.tw_alpha_h, p.tw_theta_ref,
                           s.tmprt[g.lin(k, 1, i)] - st, p.tw_kappa);
}

// -3 averaged: surfaceTheta += heatingRate dt, the sums of T(j=1) - surfaceTheta,
// |U_par| and the wall distance, and in the last block qWallShumann once from
// the plane means, the result into every wall cell (a separate launch whose one
// thread walked the 148 partials took 17 us)
__global__ void __launch_bounds__(256) k_twall_sums(Grid g, Metrics m, State s, Params p, double *part, const double *sts, unsigned *count, double *sc)
{
    const int nI = g.mx - 2, nK = g.mz - 2;
    double sT = 0.0, sU = 0.0, sD = 0.0;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nI * nK; t += gridDim.x * blockDim.x) {
        const int i = t % nI + 1, k = t / nI + 1, w = k * g.mx + i;
        double upm, dist;
        twall_cell(g, m, s, k, i, upm, dist);
        double st;
        if (sts) st = sts[0];
        else { st = s.surf_theta[w] + p.tw_heating * p.dt; s.surf_theta[w] = st; }
        sT += (s.tmprt[g.lin(k, 1, i)] - st);
        sU += upm;
        sD += dist;
    }
    double v[3] = {sT, sU, sD};
    block_reduce<256>(v, RedSum{}, RedSum{}, RedSum{});
    if (threadIdx.x == 0)
        for (int q = 0; q < 3; q++) part[3 * blockIdx.x + q] = v[q];
    if (!last_block(count)) return;
    sum_partials<256>(part, v);
    __shared__ double qw;
    if (threadIdx.x == 0) {
        const double n = (double)nI * (double)nK;
        sc[0] = v[0] / n; sc[1] = v[1] / n; sc[2] = v[2] / n;
        qw = mo::qwall(v[1] / n, v[2] / n, p.tw_z0, p.tw_gamma_m, p.tw_gamma_h, p.tw_alpha_h, p.tw_theta_ref, v[0] / n, p.tw_kappa);
        sc[3] = qw;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nI * nK; t += blockDim.x) s.qwall[(t / nI + 1) * g.mx + t % nI + 1] = qw;
}

// -2 (fixed): the prescribed flux into every wall cell
__global__ void k_twall_fill(Grid g, Params p, double *sc, State s)
{
    const int nI = g.mx - 2, nK = g.mz - 2, t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) sc[3] = p.tw_qwall;
    if (t < nI * nK) s.qwall[(t / nI + 1) * g.mx + t % nI + 1] = p.tw_qwall;
}

}  // namespace

// SolveTEqn with TeqnABBE (teqn_solvers.c:821-945): AB2 convection,
// backward-Euler diffusion A T = b, A v = v - dt D(v) (ABBEMatVec: D is FormT
// with formMode 2 of v, periodic ghosts reset, zero off the interior; the
// boundary ghosts of v stay those of the Krylov vector, and kappa_eff follows
// v's vertical gradient, so A is not linear in v for LES, as in the reference)
// by GMRES (kspIMEX: PCNONE, restart -kspGMRESRestartT, relTolT / absTolT,
// 1000 iterations, the b as initial guess). Returns the GMRES status.
static int solve_t_abbe(tg_ctx *C)
{
    const Grid g = C->g;
    const int64_t G = g.size();
    State &s = C->s;
    const double dt = C->prm.dt;
    if (!C->tgm) C->tgm = gmres_alloc(C, G, C->cfg.t_gmres_restart > 0 ? C->cfg.t_gmres_restart : 30);
    // Steps 1-2: periodic ghosts, convective right-hand side at T^n
    reset_cell_periodic_s(C, s.tmprt);
    t_face_fluxes<1>(C);
    TG_PROF(C, "teqn_rhs", k_t_rhs<<<gint(g), block3(), 0, C->stream>>>(g, C->m, s.tflux, C->tconv));
    // Steps 3-4: b (in Ttmp) and the guess; as in the reference the solution
    // goes into RhsConv_o, whose AB2 history this kernel consumes first
    double *b = s.ttmp, *x = C->tconv_o;
    TG_PROF(C, "teqn_abbe_b", k_t_abbe_b<<<nblk(G), 256, 0, C->stream>>>(G, b, x, C->tconv, C->tconv_o, s.tmprt_o, dt,
                                                                         C->it > C->cfg.it_start ? 1 : 0));
    // Step 5: GMRES on ABBEMatVec
    auto A = [&](const double *v, double *Av) {
        TG_CUDA(cudaMemcpyAsync(s.tmprt, v, sizeof(double) * G, cudaMemcpyDeviceToDevice, C->stream));
        reset_cell_periodic_s(C, s.tmprt);
        t_face_fluxes<2>(C);
        TG_PROF(C, "teqn_rhs", k_t_rhs<<<gint(g), block3(), 0, C->stream>>>(g, C->m, s.tflux, s.trhs));
        TG_PROF(C, "teqn_abbe_av", k_t_abbe_av<<<nblk(G), 256, 0, C->stream>>>(G, Av, v, s.trhs, dt));
    };
    int its = 0;
    double res = 0.0;
    const int rc = gmres_solve(C, *C->tgm, A, b, x, C->cfg.t_rtol, C->cfg.t_atol, its, res);
    // Steps 6-7: T = solution, RhsConv_o = RhsConv
    TG_CUDA(cudaMemcpyAsync(s.tmprt, x, sizeof(double) * G, cudaMemcpyDeviceToDevice, C->stream));
    TG_CUDA(cudaMemcpyAsync(C->tconv_o, C->tconv, sizeof(double) * G, cudaMemcpyDeviceToDevice, C->stream));
    C->t_its = its;
    return rc;
}

// SolveTEqn with TeqnSNES (teqn_solvers.c:596-712; bT = 0 without
// hyperviscosity or controller): the root of SNESFuncEvalT from T_o by the
// Newton-Krylov solver of the Crank-Nicolson momentum step (jfnk_solve; the
// reference uses SNESNEWTONTR with MATMFFD products: converged tightly, the
// root does not depend on the path), -absTolT / -relTolT, 20 Newton steps
static int solve_t_snes(tg_ctx *C)
{
    const Grid g = C->g;
    const int64_t G = g.size();
    State &s = C->s;
    const double dt = C->prm.dt;
    const int bdf2 = (C->cfg.t_ddt_scheme == TG_TDDT_BDF2 && C->it > C->cfg.it_start) ? 1 : 0;
    if (!C->tsn) C->tsn = jfnk_alloc(C, G, C->cfg.t_gmres_restart > 0 ? C->cfg.t_gmres_restart : 30);
    double *T = jfnk_u(C->tsn);
    TG_CUDA(cudaMemcpyAsync(T, s.tmprt_o, sizeof(double) * G, cudaMemcpyDeviceToDevice, C->stream));
    auto Feval = [&](const double *t, double *F) {
        TG_CUDA(cudaMemcpyAsync(s.tmprt, t, sizeof(double) * G, cudaMemcpyDeviceToDevice, C->stream));
        reset_cell_periodic_s(C, s.tmprt);
        t_face_fluxes<0>(C);
        TG_PROF(C, "teqn_rhs", k_t_rhs<<<gint(g), block3(), 0, C->stream>>>(g, C->m, s.tflux, s.trhs));
        TG_PROF(C, "teqn_snes_f", k_t_snes_f<<<nblk(G), 256, 0, C->stream>>>(G, F, s.trhs, t, s.tmprt_o,
                                                                           bdf2 ? C->tmprt_oo : s.tmprt_o, dt, bdf2));
    };
    int newton = 0, linear = 0;
    double fn = 0.0;
    const int rc = jfnk_solve(C, *C->tsn, Feval, C->cfg.t_atol, C->cfg.t_rtol, 20, newton, linear, fn);
    TG_CUDA(cudaMemcpyAsync(s.tmprt, T, sizeof(double) * G, cudaMemcpyDeviceToDevice, C->stream));
    C->t_its = linear;
    return rc;
}

// SolveTEqn (teqn.c:259-276) with TeqnRK4 (teqn_solvers.c:714-818),
// TeqnABBE or TeqnSNES; returns the implicit solve's status (0 for RK4)
int solve_t(tg_ctx *C)
{
    const Grid g = C->g;
    State &s = C->s;
    const double dt = C->prm.dt;
    if (C->cfg.t_ddt_scheme == TG_TDDT_BE || C->cfg.t_ddt_scheme == TG_TDDT_BDF2) {
        const int rc = solve_t_snes(C);
        reset_cell_periodic_s(C, s.tmprt);
        return rc;
    }
    if (C->cfg.t_ddt_scheme == TG_TDDT_ABBE) {
        const int rc = solve_t_abbe(C);
        reset_cell_periodic_s(C, s.tmprt);
        return rc;
    }
    const double b[4] = {1.0 / 6.0, 1.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0};
    const double a[4] = {0.0, 0.5, 0.5, 1.0};
    // FormExplicitRhsT's periodic ghosts: copied before the first stage, then
    // written by each stage's update
    reset_cell_periodic_s(C, s.tmprt);
    for (int st = 0; st < 4; st++) {
        t_face_fluxes<0>(C);
        TG_PROF(C, "teqn_rk_update", k_t_rk<<<gint(g), block3(), 0, C->stream>>>(g, C->m, s.tflux, s.tmprt, s.tmprt_o, s.ttmp,
                                                                               dt * b[st], st < 3 ? a[st + 1] * dt : 0.0, st == 0, st == 3));
    }
    return 0;
}

// UpdateWallModelsT (boundary.c:3858-4178), jLeft thetaWallFunction: the
// wall heat flux qWall of the wall cells for the temperature step that
// follows and the velocity wall function of the next step. -2: the
// prescribed flux. -3: surfaceTheta is seeded from the wall value on the
// first call and rises by heatingRate * dt on every call; qWallShumann once
// from the plane means ("averaged") or per cell ("localized")
// -4: the surface temperature of the step into its device slot (nullptr
// when the series is not set yet: the steps refuse to run then, and the ghost
// update at initialisation, on the first step's clock, is zero-gradient)
static const double *series_surface(tg_ctx *C)
{
    if (C->prm.t_wall != TG_TWALL_SURFACE_SERIES || C->series_n < 2 || !C->series_t || !C->series_v) return nullptr;
    double *out = C->d_scal + SC_TWALL + 4;
    k_twall_series<<<1, 32, 0, C->stream>>>(C->series_t, C->series_v, C->series_n, C->d_scal + SC_IT, (double)C->cfg.it_start,
                                            C->cfg.t_start, C->prm.dt, out);
    TG_CUDA(cudaGetLastError());
    return out;
}

const char *theta_wall_missing(const tg_ctx *C)
{
    if (C->prm.t_wall == TG_TWALL_SURFACE_SERIES && C->series_n < 2)
        return "thetaWallFunction -4 needs its surface temperature series (tg_set_surface_temperature)";
    return nullptr;
}

void update_wall_models_t(tg_ctx *C)
{
    if (!C->prm.les || !C->prm.t_wall) return;
    const Grid g = C->g;
    const dim3 b2(32, 8), grid((g.mx - 2 + 31) / 32, (g.mz - 2 + 7) / 8);
    if (C->prm.t_wall == TG_TWALL_FIXED_FLUX) {
        TG_PROF(C, "twall_fill", k_twall_fill<<<((g.mx - 2) * (g.mz - 2) + 255) / 256, 256, 0, C->stream>>>(g, C->prm, C->d_scal + SC_TWALL, C->s));
        return;
    }
    const double *sts = series_surface(C);
    if (C->prm.t_wall == TG_TWALL_SURFACE_SERIES && !sts)     // the entry points refuse this case before any launch
        throw CudaError{cudaErrorInvalidValue, "thetaWallFunction -4 without its surface temperature series"};
    if (!sts && !C->surf_set) {
        k_twall_seed<<<grid, b2, 0, C->stream>>>(g, C->s);
        C->surf_set = true;
    }
    if (C->prm.t_wall_localized) {
        TG_PROF(C, "twall_local", k_twall_local<<<grid, b2, 0, C->stream>>>(g, C->m, C->s, C->prm, sts));
        return;
    }
    const int nb = 148;
    TG_PROF(C, "twall_sums", k_twall_sums<<<nb, 256, 0, C->stream>>>(g, C->m, C->s, C->prm, C->d_red, sts, C->d_count + 1, C->d_scal + SC_TWALL));
}

void update_temperature_bcs(tg_ctx *C)
{
    const Grid g = C->g;
    const dim3 b2(32, 8);
    const dim3 gr((std::max(g.mx, g.my) - 2 + 31) / 32, (std::max(g.my, g.mz) - 2 + 7) / 8, 3);
    const double *sts = series_surface(C);
    TG_PROF(C, "teqn_bcs", k_t_bcs<<<gr, b2, 0, C->stream>>>(g, C->m, C->prm, C->s.tmprt, sts, C->d_scal + SC_IT, (double)C->cfg.it_start));
}

void refresh_teqn_mesh(tg_ctx *C)
{
    if (!C->prm.teqn || !C->prm.les) return;
    k_t_width<<<nblk(C->g.size()), 256, 0, C->stream>>>(C->g, C->m, C->s.trd2);
    TG_CUDA(cudaGetLastError());
}

}  // namespace tg
