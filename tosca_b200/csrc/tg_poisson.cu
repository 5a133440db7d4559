// Pressure Poisson solve for TOSCA's pinned 19-point operator (peqn.c:703-1501)
// replacing the HYPRE BoomerAMG-GMRES solve (peqn.c:3856-3929).
//
// Unknowns live in a compact interior layout c = (kc*ny + jc)*nx + ic
// (ic = i-1, ...). The operator is applied matrix-free from the nine face
// metric-tensor arrays g11..g33 at the east/north/top face of each cell; the
// 19 coefficients of a row are rebuilt in registers with the reference's
// one-sided rules and its |v| > 1e-10 insertion filter, so the product equals
// the assembled matrix. On orthogonal grids (all cross terms zero) a 7-point
// kernel reads three coefficient arrays only.
//
// Solved system: L phi = -b with L = -A (positive semidefinite away from the
// pinned row), row (1,1,1) the identity (peqn.c:883-887). Symmetric operators
// use preconditioned CG on the reduced system (the pinned unknown stays zero);
// others use right-preconditioned BiCGStab.
//
// Preconditioner: on a mesh of planes the direct solve of tg_fdm.cu, elsewhere
// the geometric multigrid V-cycle of tg_mg.cu on the 7-point part of the
// operator; both are applied in the grounded form z = P M P^T r (P shifts
// so that z at the pinned cell is zero), which is the inverse structure of the
// pinned operator. In the mixed-precision mode the multigrid stores and
// computes in FP32; the direct solve, residuals, inner products and the
// solution stay FP64.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "tg_internal.cuh"
#include "tg_fdm.cuh"
#include "tg_mg.cuh"

namespace tg {

struct PoissonCtx {
    int nx, ny, nz, pi, pj, pk;
    int64_t n;
    int pin;                     // compact index of the pinned cell (0)
    bool ortho;
    double *gE1, *gE2, *gE3, *gN1, *gN2, *gN3, *gT1, *gT2, *gT3;  // fine face tensors (compact)
    double *x, *b, *r, *z, *p, *q, *rhat, *v, *s, *t, *aj;
    double *xprev, *xprev2;      // the two previous steps' solutions (extrapolated initial guess)
    double *part;                // reduction partials (4 per block)
    int nblocks;
    MG *mg;                      // multigrid preconditioner (host object), where fdm does not apply
    Fdm *fdm;                    // direct solve on a mesh of planes, else null
    FdmOp op;                    // its factors, used for the operator if op_exact
    bool op_exact;
    unsigned *count;             // arrival counter of last_block
};

namespace {

constexpr int RB = 256;   // reduction block size

struct Cg {   // compact grid indexing with periodic wrap
    int nx, ny, nz, pi, pj, pk;
    __device__ __forceinline__ int wi(int i) const { if (i < 0) i += nx; else if (i >= nx) i -= nx; return i; }
    __device__ __forceinline__ int wj(int j) const { if (j < 0) j += ny; else if (j >= ny) j -= ny; return j; }
    __device__ __forceinline__ int wk(int k) const { if (k < 0) k += nz; else if (k >= nz) k -= nz; return k; }
    __device__ __forceinline__ int id(int k, int j, int i) const { return (wk(k) * ny + wj(j)) * nx + wi(i); }
};

// ------------------------------------------------------------ setup kernels
// planes: the normal coefficients from the spacings that the projection reads
// (k_pressure_project). The metrics give the same up to the rounding of the
// coordinates, but a projection that differs from the operator it was solved with
// leaves that much divergence.
__global__ void k_gather_g(Grid g, Metrics m, Tensor t, bool planes, PoissonCtx P)
{
    int ic = blockIdx.x * blockDim.x + threadIdx.x, jc = blockIdx.y * blockDim.y + threadIdx.y, kc = blockIdx.z * blockDim.z + threadIdx.z;
    if (ic >= P.nx || jc >= P.ny || kc >= P.nz) return;
    int c = (kc * P.ny + jc) * P.nx + ic;
    int d = g.lin(kc + 1, jc + 1, ic + 1);
    P.gE1[c] = m.g11[d]; P.gE2[c] = m.g12[d]; P.gE3[c] = m.g13[d];
    P.gN1[c] = m.g21[d]; P.gN2[c] = m.g22[d]; P.gN3[c] = m.g23[d];
    P.gT1[c] = m.g31[d]; P.gT2[c] = m.g32[d]; P.gT3[c] = m.g33[d];
    P.aj[c] = m.aj[d];
    if (planes) {
        const double dx = t.dx[kc + 1], dy = t.dy[ic + 1], dz = t.dz[jc + 1];
        P.gE1[c] = dx * dz * t.rdyf[ic + 1]; P.gN2[c] = dx * dy * t.rdzf[jc + 1]; P.gT3[c] = dy * dz * t.rdxf[kc + 1];
    }
}

// --------------------------------------------------------- fine operators
// 7-point: (L x)_c = sum_f a_f (x_c - x_nb); pinned row = identity
__global__ void k_apply7(PoissonCtx P, const double *__restrict__ x, double *__restrict__ y)
{
    int ic = blockIdx.x * blockDim.x + threadIdx.x, jc = blockIdx.y * blockDim.y + threadIdx.y, kc = blockIdx.z * blockDim.z + threadIdx.z;
    if (ic >= P.nx || jc >= P.ny || kc >= P.nz) return;
    const int nx = P.nx, pl = P.nx * P.ny;
    int c = (kc * P.ny + jc) * nx + ic;
    if (c == P.pin) { y[c] = x[c]; return; }
    // neighbours by offset; a periodic seam wraps to the opposite end
    const int e = ic < nx - 1 ? c + 1 : c + 1 - nx, w = ic > 0 ? c - 1 : c - 1 + nx;
    const int n = jc < P.ny - 1 ? c + nx : c + nx - pl, s = jc > 0 ? c - nx : c - nx + pl;
    const int t = kc < P.nz - 1 ? c + pl : c + pl - pl * P.nz, b = kc > 0 ? c - pl : c - pl + pl * P.nz;
    double xc = x[c], acc = 0.0;
    if (ic < nx - 1 || P.pi)   acc += P.gE1[c] * (xc - x[e]);
    if (ic > 0 || P.pi)        acc += P.gE1[w] * (xc - x[w]);
    if (jc < P.ny - 1 || P.pj) acc += P.gN2[c] * (xc - x[n]);
    if (jc > 0 || P.pj)        acc += P.gN2[s] * (xc - x[s]);
    if (kc < P.nz - 1 || P.pk) acc += P.gT3[c] * (xc - x[t]);
    if (kc > 0 || P.pk)        acc += P.gT3[b] * (xc - x[b]);
    y[c] = acc;
}

enum { CP, EP, WP, NP, SP, TP, BP, NE, SE, NW, SW, TN, BN, TS, BS, TE, BE, TW, BW, NST };

// 19 coefficients of one row of SetCoeffMatrix (peqn.c:889-1388). The derivative
// of a face value along a tangential direction is
//     hi (x_+ + ..) + own (x_0 + ..) - lo (x_- + ..)
// with weights of the cell's position in that direction: 1/4, 0, 1/4 inside,
// 0, 1/2, 1/2 at the last cell and 1/2, -1/2, 0 at the first (the last wins in
// a direction of one cell). Weights instead of the reference's branches: every
// lane of a warp runs the same 90 products where rows that meet a domain end
// used to run the interior and the end branches one after the other.
struct CrossW {
    double hi, own, lo;
    __device__ __forceinline__ CrossW(int l, int n)
    {
        const bool last = l == n - 1, first = l == 0 && !last;
        hi = last ? 0.0 : first ? 0.5 : 0.25;
        own = last ? 0.5 : first ? -0.5 : 0.0;
        lo = first ? 0.0 : last ? 0.5 : 0.25;
    }
};
__device__ __forceinline__ void row19(const PoissonCtx &P, const Cg &q, int ic, int jc, int kc, double (&vol)[NST])
{
    #pragma unroll
    for (int m = 0; m < NST; m++) vol[m] = 0.0;
    const int nx = P.nx, ny = P.ny, nz = P.nz, c = (kc * ny + jc) * nx + ic;
    const CrossW wi(ic, nx), wj(jc, ny), wk(kc, nz);
    // tangential term t of a face whose other cell is `nb`: `pi`/`mi` the + and -
    // neighbours of this cell along the tangent, `pn`/`mn` those of `nb`
    auto cross = [&](double t, const CrossW &w, int nb, int pi, int pn, int mi, int mn) {
        vol[CP] += t * w.own; vol[nb] += t * w.own;
        vol[pi] += t * w.hi; vol[pn] += t * w.hi;
        vol[mi] -= t * w.lo; vol[mn] -= t * w.lo;
    };
    // face f of this cell (on: it carries a flux; sg: +1 for its + side)
    auto face = [&](bool on, const double *gn, const double *gt1, const double *gt2, int f, double sg, int nb, const CrossW &w1, int p1, int pn1,
                    int m1, int mn1, const CrossW &w2, int p2, int pn2, int m2, int mn2) {
        if (!on) return;
        const double a = gn[f];
        vol[CP] -= a; vol[nb] += a;
        cross(sg * gt1[f], w1, nb, p1, pn1, m1, mn1);
        cross(sg * gt2[f], w2, nb, p2, pn2, m2, mn2);
    };
    face(ic < nx - 1 || P.pi, P.gE1, P.gE2, P.gE3, c, 1.0, EP, wj, NP, NE, SP, SE, wk, TP, TE, BP, BE);
    face(ic > 0 || P.pi, P.gE1, P.gE2, P.gE3, q.id(kc, jc, ic - 1), -1.0, WP, wj, NP, NW, SP, SW, wk, TP, TW, BP, BW);
    face(jc < ny - 1 || P.pj, P.gN2, P.gN1, P.gN3, c, 1.0, NP, wi, EP, NE, WP, NW, wk, TP, TN, BP, BN);
    face(jc > 0 || P.pj, P.gN2, P.gN1, P.gN3, q.id(kc, jc - 1, ic), -1.0, SP, wi, EP, SE, WP, SW, wk, TP, TS, BP, BS);
    face(kc < nz - 1 || P.pk, P.gT3, P.gT1, P.gT2, c, 1.0, TP, wi, EP, TE, WP, TW, wj, NP, TN, SP, TS);
    face(kc > 0 || P.pk, P.gT3, P.gT1, P.gT2, q.id(kc - 1, jc, ic), -1.0, BP, wi, EP, BE, WP, BW, wj, NP, BN, SP, BS);
}

// 19-point: y = -(A x) on non-pinned rows (entries |v| <= 1e-10 dropped as
// at peqn.c:1410-1418), y = x on the pinned row
// Bound by the latency of its 55 loads: those of x do not wait for the coefficient's
// threshold, and 80 registers hold them at three blocks per SM. A step of
// 192 x 96 x 96 took 3.47 ms with loads under the threshold, 3.39 ms this way.
__global__ void __launch_bounds__(256, 3) k_apply19(PoissonCtx P, const double *__restrict__ x, double *__restrict__ y)
{
    int ic = blockIdx.x * blockDim.x + threadIdx.x, jc = blockIdx.y * blockDim.y + threadIdx.y, kc = blockIdx.z * blockDim.z + threadIdx.z;
    if (ic >= P.nx || jc >= P.ny || kc >= P.nz) return;
    Cg q{P.nx, P.ny, P.nz, P.pi, P.pj, P.pk};
    int c = (kc * P.ny + jc) * P.nx + ic;
    if (c == P.pin) { y[c] = x[c]; return; }
    double vol[NST];
    row19(P, q, ic, jc, kc, vol);
    // the wrapped row and plane offsets once; a neighbour outside the domain has a
    // zero coefficient (its face carries no flux and its tangential weight is zero)
    // and reads the cell itself
    const int pl = P.nx * P.ny;
    const int ie = ic < P.nx - 1 ? 1 : P.pi ? 1 - P.nx : 0, iw = ic > 0 ? -1 : P.pi ? P.nx - 1 : 0;
    const int jn = jc < P.ny - 1 ? P.nx : P.pj ? P.nx - pl : 0, js = jc > 0 ? -P.nx : P.pj ? pl - P.nx : 0;
    const int kt = kc < P.nz - 1 ? pl : P.pk ? pl - pl * P.nz : 0, kb = kc > 0 ? -pl : P.pk ? pl * P.nz - pl : 0;
    double acc = vol[CP] * x[c];
    auto add = [&](int m, int o) { const double xv = x[c + o], t = acc + vol[m] * xv; acc = fabs(vol[m]) > 1.e-10 ? t : acc; };
    add(EP, ie); add(WP, iw); add(NP, jn); add(SP, js); add(TP, kt); add(BP, kb);
    add(NE, jn + ie); add(SE, js + ie); add(NW, jn + iw); add(SW, js + iw);
    add(TN, kt + jn); add(BN, kb + jn); add(TS, kt + js); add(BS, kb + js);
    add(TE, kt + ie); add(BE, kb + ie); add(TW, kt + iw); add(BW, kb + iw);
    y[c] = -acc;
}

// ------------------------------------------------------ vector kernels
// The vectors are separate cudaMalloc allocations (256-byte aligned), so the
// grid-stride loops below move two doubles per access (double2, 16-byte
// loads and stores); an odd last element is taken by thread 0 of block 0
// after its loop.
__device__ __forceinline__ const double2 *v2(const double *a) { return reinterpret_cast<const double2 *>(a); }
__device__ __forceinline__ double2 *v2(double *a) { return reinterpret_cast<double2 *>(a); }
__device__ __forceinline__ bool odd_tail(int64_t n) { return (n & 1) && blockIdx.x == 0 && threadIdx.x == 0; }
#define TG_PAIRS(t, n2) for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < (n2); t += (int64_t)gridDim.x * blockDim.x)

// partial sums: slot 0 = a.b, slot 1 = sum(a), slot 2 = max |a * w|
__device__ __forceinline__ void dot_acc(double av, double bv, double wv, double (&v)[3])
{
    v[0] += av * bv;
    v[1] += av;
    v[2] = fmax(v[2], fabs(av * wv));
}
__device__ __forceinline__ void dot_store(double (&v)[3], double *part)
{
    block_reduce<RB>(v, RedSum{}, RedSum{}, RedMax{});
    if (threadIdx.x == 0) { part[3 * blockIdx.x] = v[0]; part[3 * blockIdx.x + 1] = v[1]; part[3 * blockIdx.x + 2] = v[2]; }
}
// sh: constant subtracted from b (the preconditioned residual is used up to
// its value at the pinned cell), or null
__global__ void __launch_bounds__(RB) k_dot_partial(int64_t n, const double *a, const double *b, const double *sh, const double *w, double *part)
{
    double v[3] = {0.0, 0.0, 0.0};
    const double b0 = sh ? sh[0] : 0.0;
    const int64_t n2 = n >> 1;
    TG_PAIRS(t, n2) {
        const double2 av = v2(a)[t], bv = v2(b)[t];
        const double2 wv = w ? v2(w)[t] : double2{0.0, 0.0};
        dot_acc(av.x, bv.x - b0, wv.x, v);
        dot_acc(av.y, bv.y - b0, wv.y, v);
    }
    if (odd_tail(n)) dot_acc(a[n - 1], b[n - 1] - b0, w ? w[n - 1] : 0.0, v);
    dot_store(v, part);
}
// final: out[0..2] = totals
__global__ void __launch_bounds__(RB) k_dot_final(const double *part, int nb, double *out)
{
    double v[3] = {0.0, 0.0, 0.0};
    for (int b = threadIdx.x; b < nb; b += blockDim.x) { v[0] += part[3 * b]; v[1] += part[3 * b + 1]; v[2] = fmax(v[2], part[3 * b + 2]); }
    block_reduce<RB>(v, RedSum{}, RedSum{}, RedMax{});
    if (threadIdx.x == 0) { out[0] = v[0]; out[1] = v[1]; out[2] = v[2]; }
}

// y = b - y (residual from y = L x)
__global__ void k_resid(int64_t n, const double *b, double *y)
{
    const int64_t n2 = n >> 1;
    TG_PAIRS(t, n2) { const double2 bv = v2(b)[t], yv = v2(y)[t]; v2(y)[t] = double2{bv.x - yv.x, bv.y - yv.y}; }
    if (odd_tail(n)) y[n - 1] = b[n - 1] - y[n - 1];
}
__global__ void k_copy(int64_t n, const double *a, double *b)
{
    const int64_t n2 = n >> 1;
    TG_PAIRS(t, n2) v2(b)[t] = v2(a)[t];
    if (odd_tail(n)) b[n - 1] = a[n - 1];
}
__global__ void k_fill(int64_t n, double *a, double v)
{
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) a[t] = v;
}
__global__ void k_zero_at(double *z, int pin) { z[pin] = 0.0; }
// initial guess of the step's solve from the last three solutions (the
// reference starts from x_n): 3 x_n - 3 x_{n-1} + x_{n-2} (quadratic
// extrapolation), 2 x_n - x_{n-1} while only two are known, x_n with one;
// the history shifts (xprev2 <- xprev <- x_n). hist: device count of the
// solutions in the history, read here and advanced by k_hist_next
__global__ void k_extrapolate(int64_t n, double *x, double *xprev, double *xprev2, const double *hist, int order)
{
    const double h = fmin(hist[0], (double)order);
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const double xn = x[t], xp = xprev[t];
        if (h >= 2.0) x[t] = 3.0 * xn - 3.0 * xp + xprev2[t];
        else if (h >= 1.0) x[t] = 2.0 * xn - xp;
        xprev2[t] = xp;
        xprev[t] = xn;
    }
}
__global__ void k_hist_next(double *hist) { hist[0] = hist[0] + 1.0; }
inline int guess_order(const tg_ctx *C) { return C->cfg.poisson_guess < 0 ? 2 : C->cfg.poisson_guess; }
__global__ void k_negcopy(int64_t n, const double *a, double *b)
{
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) b[t] = -a[t];
}

// CG: alpha = rz / pq ; x += alpha p ; r -= alpha q, with the partials of
// k_dot_partial(r, r, w) formed in the same grid-stride order (same grid), so
// the totals equal those of a separate update and dot product
__global__ void __launch_bounds__(RB, 4) k_cg_update_rr(int64_t n, const double *rz, const double *pq, double *x, const double *p,
                                                     double *r, const double *q, const double *w, double *part)
{
    const double alpha = rz[0] / pq[0];
    double v[3] = {0.0, 0.0, 0.0};
    const int64_t n2 = n >> 1;
    TG_PAIRS(t, n2) {
        const double2 xv = v2(x)[t], pv = v2(p)[t], rv = v2(r)[t], qv = v2(q)[t];
        const double2 xn{xv.x + alpha * pv.x, xv.y + alpha * pv.y}, rn{rv.x - alpha * qv.x, rv.y - alpha * qv.y};
        v2(x)[t] = xn;
        v2(r)[t] = rn;
        const double2 wv = w ? v2(w)[t] : double2{0.0, 0.0};
        dot_acc(rn.x, rn.x, wv.x, v);
        dot_acc(rn.y, rn.y, wv.y, v);
    }
    if (odd_tail(n)) {
        x[n - 1] += alpha * p[n - 1];
        r[n - 1] -= alpha * q[n - 1];
        const double rv = r[n - 1];
        dot_acc(rv, rv, w ? w[n - 1] : 0.0, v);
    }
    dot_store(v, part);
}
__global__ void k_scalar_copy(const double *a, double *b, int n) { for (int t = 0; t < n; t++) b[t] = a[t]; }

// BiCGStab pieces (device scalars in sc: rho, alpha, omega, rho_old)
__global__ void k_bicg_p(int64_t n, const double *sc, double *p, const double *r, const double *v)
{
    // beta = (rho/rho_old) * (alpha/omega)
    double beta = (sc[0] / sc[3]) * (sc[1] / sc[2]);
    double omega = sc[2];
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        p[t] = r[t] + beta * (p[t] - omega * v[t]);
}
__global__ void k_bicg_s(int64_t n, const double *rho, const double *rhv, double *alpha_out, double *s, const double *r, const double *v)
{
    double alpha = rho[0] / rhv[0];
    if (blockIdx.x == 0 && threadIdx.x == 0) alpha_out[0] = alpha;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) s[t] = r[t] - alpha * v[t];
}
__global__ void k_bicg_x(int64_t n, const double *alpha, const double *ts, const double *tt, double *omega_out,
                         double *x, const double *phat, const double *shat, double *r, const double *s, const double *t_)
{
    double om = tt[0] > 0 ? ts[0] / tt[0] : 0.0;
    double al = alpha[0];
    if (blockIdx.x == 0 && threadIdx.x == 0) omega_out[0] = om;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        x[t] += al * phat[t] + om * shat[t];
        r[t] = s[t] - om * t_[t];
    }
}

// ---- loop control of the captured CG solve (device scalars: sc[50] iteration
// count, sc[51] first-direction flag, sc[52] converged flag, sc[53] BiCGStab
// restart after a failed true-residual check). The tests are
// those of krylov_solve; a non-finite residual also ends the loop.
__device__ inline bool cg_converged(const double *sc, double rtol, double divtol, double dt)
{
    const double bn = sqrt(sc[0]), rn = sqrt(sc[3]), rmax = sc[5] * dt;
    return bn == 0.0 || rn / bn <= rtol || (divtol > 0 && rmax <= divtol);
}
__global__ void k_cg_start(double *sc, double rtol, double divtol, double dt, int maxit, cudaGraphConditionalHandle h, int base)
{
    const double bn = sqrt(sc[0]), rn = sqrt(sc[3]);
    const bool conv = cg_converged(sc, rtol, divtol, dt);
    sc[base + ST_RES0] = bn > 0 ? rn / bn : rn;
    sc[50] = 0.0; sc[51] = 1.0; sc[52] = conv ? 1.0 : 0.0; sc[53] = 0.0;
    cudaGraphSetConditional(h, (!conv && maxit > 0 && isfinite(rn)) ? 1u : 0u);
}
__global__ void k_cg_next(double *sc, double rtol, double divtol, double dt, int maxit, cudaGraphConditionalHandle h)
{
    const double rn = sqrt(sc[3]);
    const int it = (int)sc[50] + 1;
    const bool conv = cg_converged(sc, rtol, divtol, dt);
    sc[50] = it; sc[51] = 0.0; sc[52] = conv ? 1.0 : 0.0;
    cudaGraphSetConditional(h, (!conv && it < maxit && isfinite(rn)) ? 1u : 0u);
}
// statistics of the solve, accumulated over the replayed solves in the
// ST_* slots from base
__global__ void k_cg_finish(double *sc, int base)
{
    const double bn = sqrt(sc[0]), rn = sqrt(sc[3]);
    sc[base + ST_IT] = sc[50];
    sc[base + ST_TOT] += sc[50];
    sc[base + ST_RES] = bn > 0 ? rn / bn : rn;
    if (!isfinite(rn)) sc[base + ST_NAN] = 1.0;
    else if (sc[52] == 0.0) sc[base + ST_NOCONV] += 1.0;
}
// CG direction: p = z - z[0] on the first pass through the loop (sc[51]), else
// p = z - z[0] + (rz_new / rz_old) p
__global__ void k_cg_dir(int64_t n, const double *sc, const double *z, double *p)
{
    const bool first = sc[51] != 0.0;
    const double beta = first ? 0.0 : sc[6] / sc[14], z0 = z[0];
    const int64_t n2 = n >> 1;
    TG_PAIRS(t, n2) {
        const double2 zv = v2(z)[t];
        double2 o{zv.x - z0, zv.y - z0};
        if (!first) { const double2 pv = v2(p)[t]; o = double2{o.x + beta * pv.x, o.y + beta * pv.y}; }
        v2(p)[t] = o;
    }
    if (odd_tail(n)) p[n - 1] = first ? z[n - 1] - z0 : z[n - 1] - z0 + beta * p[n - 1];
}

// ---------------------------------------------- solve with the direct solver
// The iteration with the direct solve as preconditioner. It reduces the
// residual to near rounding at once, so directions need no conjugation: each
// pass takes z = M r and the step length that CG's first iteration takes,
// alpha = (r, z) / (z, L z), and reads z where CG reads its direction p. The
// vector work of a solve is four kernels instead of 14 launches, each with its dot
// products finished by the last block to arrive (256 x 256 x 128: 0.61 ms before,
// 0.37 ms now, of 0.30 ms for their bytes). In k_direct_begin a warp takes a row of
// the compact grid, lanes along i, so that 3-D indices cost one division per row;
// the two that apply the operator march along k (op7_march).
struct Rows {
    int nx, ny, nrow, lane, row, step;
    __device__ __forceinline__ Rows(const PoissonCtx &P)
        : nx(P.nx), ny(P.ny), nrow(P.ny * P.nz), lane(threadIdx.x & 31),
          row((int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5)), step((int)((gridDim.x * blockDim.x) >> 5)) {}
};
// totals of N partials per block (sums; the last slot a maximum if MAX) into v of thread 0
template <int N, bool MAX>
__device__ __forceinline__ void total(const double *part, double (&v)[3])
{
    v[0] = v[1] = v[2] = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += RB) {
        #pragma unroll
        for (int q = 0; q < N; q++) {
            const double x = __ldcg(part + N * b + q);
            v[q] = (MAX && q == N - 1) ? fmax(v[q], x) : v[q] + x;
        }
    }
    __syncthreads();
    block_reduce<RB>(v, RedSum{}, RedSum{}, RedMax{});
}

// loop control, as k_cg_start / k_cg_next / k_cg_finish. CAP: the loop is a
// conditional node of a captured step.
struct Loop { double rtol, divtol, dt; int maxit, base; };
template <bool CAP>
__device__ void loop_go(double *sc, const Loop &L, int it, cudaGraphConditionalHandle h)
{
    if (!CAP) return;
    const double bn = sqrt(sc[0]), rn = sqrt(sc[3]);
    const bool conv = cg_converged(sc, L.rtol, L.divtol, L.dt);
    const bool go = !conv && it < L.maxit && isfinite(rn);
    sc[50] = it; sc[52] = conv ? 1.0 : 0.0;
    if (it == 0) sc[L.base + ST_RES0] = bn > 0 ? rn / bn : rn;
    if (!go) {
        sc[L.base + ST_IT] = it;
        sc[L.base + ST_TOT] += it;
        sc[L.base + ST_RES] = bn > 0 ? rn / bn : rn;
        if (!isfinite(rn)) sc[L.base + ST_NAN] = 1.0;
        else if (!conv) sc[L.base + ST_NOCONV] += 1.0;
    }
    cudaGraphSetConditional(h, go ? 1u : 0u);
}

// SetRHS (peqn.c:1942-2063) into the compact vector, negated (L = -A), the
// initial guess (k_extrapolate, k_hist_next) and |b|^2. keep[0] <- p(1,1,1), the
// gauge of the pressure after the update (phi is zero at the pinned cell).
__global__ void __launch_bounds__(RB) k_direct_begin(Grid g, State s, PoissonCtx P, double dt, double *hist, int order, double *sc, double *keep)
{
    const Rows R(P);
    const double h = fmin(hist[0], (double)order);
    double v[3] = {0.0, 0.0, 0.0};
    for (int row = R.row; row < R.nrow; row += R.step) {
        const int jc = row % R.ny, kc = row / R.ny, d0 = g.lin(kc + 1, jc + 1, 1), c0 = row * R.nx;
        #pragma unroll 4
        for (int i = R.lane; i < R.nx; i += 32) {
            const int c = c0 + i, d = d0 + i;
            double val = 0;
            val += s.ucont.x[d];
            val -= s.ucont.x[d - 1];
            val += s.ucont.y[d];
            val -= s.ucont.y[d - g.mx];
            val += s.ucont.z[d];
            val -= s.ucont.z[d - g.mx * g.my];
            val *= 1.0 / dt;
            const double b = c == P.pin ? 0.0 : -val;
            P.b[c] = b;
            v[0] += b * b;
            const double xn = P.x[c], xp = P.xprev[c];
            double x = xn;
            if (h >= 2.0) x = 3.0 * xn - 3.0 * xp + P.xprev2[c];
            else if (h >= 1.0) x = 2.0 * xn - xp;
            P.x[c] = c == P.pin ? 0.0 : x;
            P.xprev2[c] = xp;
            P.xprev[c] = xn;
        }
    }
    block_reduce<RB>(v, RedSum{}, RedSum{}, RedMax{});
    if (threadIdx.x == 0) P.part[blockIdx.x] = v[0];
    if (last_block(P.count)) {
        total<1, false>(P.part, v);
        if (threadIdx.x == 0) {
            sc[0] = v[0];
            hist[0] = hist[0] + 1.0;
            keep[0] = s.p[g.lin(1, 1, 1)];
        }
    }
}

// f(c, x_c, (L x)_c) of k_apply7 for every cell; FAC: coefficients from their
// factors, associated as the projection's (k_pressure_project): (area) / distance,
// so that the two are the same numbers. A block takes 32 x 8 columns (a warp per j) of kc cells along k and
// holds the column's cell, the one below and the one above in registers.
// Latency-bound: r = b - L x takes 77 us at 256 x 256 x 128 and the dot products 69, of
// 41 and 31 us for their bytes; rows of i per warp, whose loads wait for the stores
// of the cells before them and which fetch each x three times from L2, 137 and 89.
template <bool FAC, class F>
__device__ __forceinline__ void op7_march(const PoissonCtx &P, const double *x, int kc, F f)
{
    const int nx = P.nx, ny = P.ny, nz = P.nz, pl = nx * ny, nbi = (nx + 31) / 32, nbj = (ny + RB / 32 - 1) / (RB / 32), nt = nbi * nbj * ((nz + kc - 1) / kc);
    for (int t = blockIdx.x; t < nt; t += gridDim.x) {
        const int i = t % nbi * 32 + (threadIdx.x & 31), j = t / nbi % nbj * (RB / 32) + (threadIdx.x >> 5), k0 = t / (nbi * nbj) * kc, k1 = min(k0 + kc, nz);
        if (i >= nx || j >= ny) continue;
        // a face without a flux has a zero coefficient; its offset wraps inside the grid
        const int oE = i < nx - 1 ? 1 : 1 - nx, oW = i > 0 ? -1 : nx - 1, oN = j < ny - 1 ? nx : nx - pl, oS = j > 0 ? -nx : pl - nx;
        const bool hE = i < nx - 1 || P.pi, hW = i > 0 || P.pi, hN = j < ny - 1 || P.pj, hS = j > 0 || P.pj;
        double m = 0.0, my = 0.0, kE = 0.0, kW = 0.0, kN = 0.0, kS = 0.0;
        if (FAC) {
            m = P.op.mx[i]; my = P.op.my[j];
            kE = hE ? P.op.kx[i] : 0.0; kW = hW ? P.op.kx[i > 0 ? i - 1 : nx - 1] : 0.0;
            kN = hN ? P.op.ky[j] : 0.0; kS = hS ? P.op.ky[j > 0 ? j - 1 : ny - 1] : 0.0;
        }
        const double mmy = m * my;
        int c = (k0 * ny + j) * nx + i;
        double xb = __ldg(x + c + (k0 > 0 ? -pl : pl * nz - pl)), xc = __ldg(x + c);
        double gb = k0 > 0 || P.pk ? (FAC ? P.op.kz[k0 > 0 ? k0 - 1 : nz - 1] * mmy : __ldg(P.gT3 + c + (k0 > 0 ? -pl : pl * nz - pl))) : 0.0;
        #pragma unroll 2
        for (int k = k0; k < k1; k++, c += pl) {
            const bool top = k < nz - 1;
            const double xt = __ldg(x + (top ? c + pl : c + pl - pl * nz)), xe = __ldg(x + c + oE), xw = __ldg(x + c + oW), xn = __ldg(x + c + oN), xs = __ldg(x + c + oS);
            double acc = 0.0, gt = 0.0;
            if (FAC) {
                const double mz = __ldg(P.op.mz + k), e = my * mz;
                const double mmz = m * mz;
                if (top || P.pk) gt = __ldg(P.op.kz + k) * mmy;
                acc += (kE * e) * (xc - xe);
                acc += (kW * e) * (xc - xw);
                acc += (kN * mmz) * (xc - xn);
                acc += (kS * mmz) * (xc - xs);
                acc += gt * (xc - xt);
                acc += gb * (xc - xb);
            } else {
                if (top || P.pk) gt = __ldg(P.gT3 + c);
                acc += (hE ? __ldg(P.gE1 + c) : 0.0) * (xc - xe);
                acc += (hW ? __ldg(P.gE1 + c + oW) : 0.0) * (xc - xw);
                acc += (hN ? __ldg(P.gN2 + c) : 0.0) * (xc - xn);
                acc += (hS ? __ldg(P.gN2 + c + oS) : 0.0) * (xc - xs);
                acc += gt * (xc - xt);
                acc += gb * (xc - xb);
            }
            f(c, xc, acc);
            xb = xc; xc = xt; gb = gt;
        }
    }
}

// r = b - L x with |r|^2, sum r and max |r aj| (sc[3..5]), and the loop's start
template <bool FAC, bool CAP>
__global__ void __launch_bounds__(RB, 4) k_direct_resid(const __grid_constant__ PoissonCtx P, const double *w, int kc, double *sc, Loop L, cudaGraphConditionalHandle h)
{
    double v[3] = {0.0, 0.0, 0.0};
    op7_march<FAC>(P, P.x, kc, [&](int c, double x, double Lx) {
        const double r = __ldg(P.b + c) - (c == P.pin ? x : Lx);
        P.r[c] = r;
        dot_acc(r, r, w ? __ldg(w + c) : 0.0, v);
    });
    dot_store(v, P.part);
    if (last_block(P.count)) {
        total<3, true>(P.part, v);
        if (threadIdx.x == 0) {
            sc[3] = v[0]; sc[4] = v[1]; sc[5] = v[2];
            loop_go<CAP>(sc, L, 0, h);
        }
    }
}

// q = L z (zero at the pin) with (r, z - z_0) and (z - z_0, q) (sc[6], sc[9])
template <bool FAC>
__global__ void __launch_bounds__(RB, 4) k_direct_dots(const __grid_constant__ PoissonCtx P, int kc, double *sc)
{
    const double z0 = P.z[0];
    double v[3] = {0.0, 0.0, 0.0};
    op7_march<FAC>(P, P.z, kc, [&](int c, double zc, double Lz) {
        const double q = c == P.pin ? 0.0 : Lz, z = zc - z0;
        P.q[c] = q;
        v[0] += __ldg(P.r + c) * z;
        v[1] += z * q;
    });
    block_reduce<RB>(v, RedSum{}, RedSum{}, RedMax{});
    if (threadIdx.x == 0) { P.part[2 * blockIdx.x] = v[0]; P.part[2 * blockIdx.x + 1] = v[1]; }
    if (last_block(P.count)) {
        total<2, false>(P.part, v);
        if (threadIdx.x == 0) { sc[6] = v[0]; sc[9] = v[1]; }
    }
}

// x += alpha (z - z_0), r -= alpha q with the sums of k_direct_resid, and the
// loop's next pass
template <bool CAP>
__global__ void __launch_bounds__(RB) k_direct_update(PoissonCtx P, const double *w, double *sc, Loop L, cudaGraphConditionalHandle h)
{
    const double alpha = sc[6] / sc[9], z0 = P.z[0];
    double v[3] = {0.0, 0.0, 0.0};
    const int64_t n = P.n, n2 = n >> 1;
    TG_PAIRS(t, n2) {
        const double2 xv = v2(P.x)[t], zv = v2(P.z)[t], rv = v2(P.r)[t], qv = v2(P.q)[t];
        const double2 rn{rv.x - alpha * qv.x, rv.y - alpha * qv.y};
        v2(P.x)[t] = double2{xv.x + alpha * (zv.x - z0), xv.y + alpha * (zv.y - z0)};
        v2(P.r)[t] = rn;
        const double2 wv = w ? v2(w)[t] : double2{0.0, 0.0};
        dot_acc(rn.x, rn.x, wv.x, v);
        dot_acc(rn.y, rn.y, wv.y, v);
    }
    if (odd_tail(n)) {
        P.x[n - 1] += alpha * (P.z[n - 1] - z0);
        const double rn = P.r[n - 1] - alpha * P.q[n - 1];
        P.r[n - 1] = rn;
        dot_acc(rn, rn, w ? w[n - 1] : 0.0, v);
    }
    dot_store(v, P.part);
    if (last_block(P.count)) {
        total<3, true>(P.part, v);
        if (threadIdx.x == 0) {
            sc[3] = v[0]; sc[4] = v[1]; sc[5] = v[2];
            if (CAP) loop_go<CAP>(sc, L, (int)sc[50] + 1, h);
        }
    }
}

inline dim3 cgrid(int nx, int ny, int nz) { return grid3(nx, ny, nz); }
inline int vblocks(int64_t n) { int64_t b = (n + RB - 1) / RB; return (int)std::min<int64_t>(b, 148 * 8); }

}  // namespace

// ============================================================== host side
static void apply_op(tg_ctx *C, const double *x, double *y)
{
    PoissonCtx &P = *C->pois;
    if (P.ortho) TG_PROF(C, "pois_apply7", k_apply7<<<cgrid(P.nx, P.ny, P.nz), block3(), 0, C->stream>>>(P, x, y));
    else TG_PROF(C, "pois_apply19", k_apply19<<<cgrid(P.nx, P.ny, P.nz), block3(), 0, C->stream>>>(P, x, y));
}

// totals of (a.b, sum a, max|a w|) into out[0..2] (device); sh: see k_dot_partial
static void dot3v(tg_ctx *C, const double *a, const double *b, const double *w, double *out, const double *sh = nullptr)
{
    PoissonCtx &P = *C->pois;
    TG_PROF(C, "pois_dot", k_dot_partial<<<P.nblocks, RB, 0, C->stream>>>(P.n, a, b, sh, w, P.part));
    k_dot_final<<<1, RB, 0, C->stream>>>(P.part, P.nblocks, out);
}

// z = P M P^T r up to a constant (z[0], which the multigrid returns as zero);
// needs sum(r) at d_sum
static void precondition(tg_ctx *C, const double *r, double *z, const double *d_sum)
{
    if (C->pois->fdm) fdm_apply(C, C->pois->fdm, r, d_sum, z);
    else mg_apply(C, C->pois->mg, r, d_sum, z);
}

// SetRHS (peqn.c:1942-2063) into the compact vector, negated (L = -A)
__global__ void k_set_rhs(Grid g, State s, PoissonCtx P, double dt)
{
    int ic = blockIdx.x * blockDim.x + threadIdx.x, jc = blockIdx.y * blockDim.y + threadIdx.y, kc = blockIdx.z * blockDim.z + threadIdx.z;
    if (ic >= P.nx || jc >= P.ny || kc >= P.nz) return;
    int c = (kc * P.ny + jc) * P.nx + ic;
    if (c == P.pin) { P.b[c] = 0.0; return; }
    int d = g.lin(kc + 1, jc + 1, ic + 1);
    double val = 0;
    val += s.ucont.x[d];
    val -= s.ucont.x[d - 1];
    val += s.ucont.y[d];
    val -= s.ucont.y[d - g.mx];
    val += s.ucont.z[d];
    val -= s.ucont.z[d - g.mx * g.my];
    val *= 1.0 / dt;
    P.b[c] = -val;
}

// phiToPhi (peqn.c:1579-1636): compact solution into the DMDA interior
__global__ void k_phi_to_dmda(Grid g, State s, PoissonCtx P)
{
    int ic = blockIdx.x * blockDim.x + threadIdx.x, jc = blockIdx.y * blockDim.y + threadIdx.y, kc = blockIdx.z * blockDim.z + threadIdx.z;
    if (ic >= P.nx || jc >= P.ny || kc >= P.nz) return;
    s.phi[g.lin(kc + 1, jc + 1, ic + 1)] = P.x[(kc * P.ny + jc) * P.nx + ic];
}

void poisson_setup(tg_ctx *C)
{
    if (C->pois) poisson_destroy(C);
    const size_t mark = C->allocs.size();
    PoissonCtx *P = new PoissonCtx();
    C->pois = P;
    const Grid g = C->g;
    P->nx = g.mx - 2; P->ny = g.my - 2; P->nz = g.mz - 2;
    P->pi = g.pi; P->pj = g.pj; P->pk = g.pk;
    P->n = (int64_t)P->nx * P->ny * P->nz;
    P->pin = 0;
    P->ortho = C->orthogonal;
    const int64_t n = P->n;
    double **fine[] = {&P->gE1, &P->gE2, &P->gE3, &P->gN1, &P->gN2, &P->gN3, &P->gT1, &P->gT2, &P->gT3,
                       &P->x, &P->b, &P->r, &P->z, &P->p, &P->q, &P->rhat, &P->v, &P->s, &P->t, &P->aj, &P->xprev, &P->xprev2};
    for (double **f : fine) *f = dallocd(C, n);
    TG_CUDA(cudaMemsetAsync(C->d_scal + SC_PHIST, 0, sizeof(double), C->stream));   // empty guess history
    P->nblocks = vblocks(n);
    P->part = dallocd(C, 3 * (size_t)P->nblocks);
    P->count = (unsigned *)dalloc(C, sizeof(unsigned));
    k_gather_g<<<cgrid(P->nx, P->ny, P->nz), block3(), 0, C->stream>>>(g, C->m, C->ts, C->axis_aligned, *P);

    P->fdm = P->ortho ? fdm_create(C, C->axis_aligned ? &C->ts : nullptr, P->gE1, P->gN2, P->gT3, P->nx, P->ny, P->nz, P->pi, P->pj, P->pk) : nullptr;
    P->op_exact = P->fdm && fdm_factors(P->fdm, &P->op);
    P->mg = P->fdm ? nullptr : mg_create(C, C->cfg.precision == TG_PREC_MIXED, P->gE1, P->gN2, P->gT3,
                                         P->nx, P->ny, P->nz, P->pi, P->pj, P->pk);
    TG_CUDA(cudaGetLastError());
    C->pois_allocs.assign(C->allocs.begin() + mark, C->allocs.end());
    C->allocs.resize(mark);
}

void poisson_destroy(tg_ctx *C)
{
    if (C->pois && C->pois->mg) mg_destroy(C->pois->mg);
    if (C->pois && C->pois->fdm) fdm_destroy(C->pois->fdm);
    delete C->pois;
    C->pois = nullptr;
    if (C->pois_allocs.empty()) return;
    cudaStreamSynchronize(C->stream);
    for (void *p : C->pois_allocs) cudaFree(p);
    C->pois_allocs.clear();
}

// host read of device scalars [off, off+cnt)
static void read_scal(tg_ctx *C, int off, int cnt)
{
    TG_CUDA(cudaMemcpyAsync(C->h_scal + off, C->d_scal + off, sizeof(double) * cnt, cudaMemcpyDeviceToHost, C->stream));
    TG_CUDA(cudaStreamSynchronize(C->stream));
}

static Loop loop_of(tg_ctx *C, double rtol, double divtol, int maxit, int base) { return Loop{rtol, divtol, C->prm.dt, maxit, base}; }

// blocks and cells along k per block of op7_march: every chunk costs about two
// cells of start-up, every started wave of four blocks per SM a chunk
struct March {
    int kc, nb;
    explicit March(const PoissonCtx &P) : kc(P.nz)
    {
        const int64_t cols = (int64_t)((P.nx + 31) / 32) * ((P.ny + RB / 32 - 1) / (RB / 32));
        int64_t best = INT64_MAX;
        for (int ch = 1; ch <= P.nz; ch++) {
            const int c = (P.nz + ch - 1) / ch;
            const int64_t waves = (cols * ((P.nz + c - 1) / c) + 4 * 148 - 1) / (4 * 148), cost = waves * (c + 2);
            if (cost < best) { best = cost; kc = c; }
        }
        nb = (int)std::min<int64_t>(cols * ((P.nz + kc - 1) / kc), P.nblocks);
    }
};

// one pass of the direct solver's iteration; CAP: inside the captured loop
template <bool CAP>
static void direct_pass(tg_ctx *C, const Loop &L, cudaGraphConditionalHandle h)
{
    PoissonCtx &P = *C->pois;
    cudaStream_t s = C->stream;
    double *sc = C->d_scal;
    const March march(P);
    fdm_apply(C, P.fdm, P.r, sc + 4, P.z);
    if (P.op_exact) TG_PROF(C, "pois_dots", k_direct_dots<true><<<march.nb, RB, 0, s>>>(P, march.kc, sc));
    else TG_PROF(C, "pois_dots", k_direct_dots<false><<<march.nb, RB, 0, s>>>(P, march.kc, sc));
    TG_PROF(C, "pois_update", (k_direct_update<CAP><<<P.nblocks, RB, 0, s>>>(P, L.divtol > 0 ? P.aj : nullptr, sc, L, h)));
}
template <bool CAP>
static void direct_resid(tg_ctx *C, const Loop &L, cudaGraphConditionalHandle h)
{
    PoissonCtx &P = *C->pois;
    const double *w = L.divtol > 0 ? P.aj : nullptr;
    const March march(P);
    if (P.op_exact) TG_PROF(C, "pois_resid", (k_direct_resid<true, CAP><<<march.nb, RB, 0, C->stream>>>(P, w, march.kc, C->d_scal, L, h)));
    else TG_PROF(C, "pois_resid", (k_direct_resid<false, CAP><<<march.nb, RB, 0, C->stream>>>(P, w, march.kc, C->d_scal, L, h)));
}

// direct solve of L x = b from the current P.x (P.b and |b|^2 in sc[0] set by the caller)
static int direct_solve(tg_ctx *C, tg_stats *st, double rtol, double divtol, int maxit)
{
    const Loop L = loop_of(C, rtol, divtol, maxit, 0);
    double *hs = C->h_scal;
    direct_resid<false>(C, L, cudaGraphConditionalHandle{});
    read_scal(C, 0, 6);
    const double bn = std::sqrt(hs[0]);
    double rn = std::sqrt(hs[3]);
    if (st) st->poisson_initial_residual = bn > 0 ? rn / bn : rn;
    auto converged = [&]() { return bn == 0.0 || rn / bn <= rtol || (divtol > 0 && hs[5] * L.dt <= divtol); };
    int it = 0;
    while (!converged() && it < maxit && std::isfinite(rn)) {
        direct_pass<false>(C, L, cudaGraphConditionalHandle{});
        read_scal(C, 3, 3);
        rn = std::sqrt(hs[3]);
        it++;
    }
    TG_CUDA(cudaGetLastError());
    if (st) {
        st->poisson_iterations = it;
        st->poisson_total_iterations += it;
        st->poisson_final_residual = bn > 0 ? rn / bn : rn;
    }
    if (!std::isfinite(rn)) return 2;
    return converged() ? 0 : 1;
}

// Krylov solve of L x = b from the current P.x (P.b set by the caller):
// preconditioned CG on orthogonal grids (the iteration of direct_solve on a mesh
// of planes), BiCGStab otherwise. Stops at the relative residual rtol or, when
// divtol > 0, at dt * max|r aj| <= divtol.
static int krylov_solve(tg_ctx *C, tg_stats *st, double rtol, double divtol, int maxit)
{
    PoissonCtx &P = *C->pois;
    const int64_t n = P.n;
    cudaStream_t s = C->stream;
    const double dt = C->prm.dt;
    double *sc = C->d_scal;          // device scalar slots 0..7 used below
    double *hs = C->h_scal;

    dot3v(C, P.b, P.b, nullptr, sc + 0);
    if (P.fdm) return direct_solve(C, st, rtol, divtol, maxit);
    apply_op(C, P.x, P.r);
    k_resid<<<vblocks(n), RB, 0, s>>>(n, P.b, P.r);   // r = b - L x
    dot3v(C, P.r, P.r, divtol > 0 ? P.aj : nullptr, sc + 3);
    read_scal(C, 0, 6);
    const double bn = std::sqrt(hs[0]);
    double rn = std::sqrt(hs[3]);
    double rmax = hs[5] * dt;
    if (st) st->poisson_initial_residual = bn > 0 ? rn / bn : rn;
    int it = 0;
    auto converged = [&]() {
        if (bn == 0.0) return true;
        if (rn / bn <= rtol) return true;
        if (divtol > 0 && rmax <= divtol) return true;
        return false;
    };
    bool ok = converged();
    if (P.ortho) {
        // preconditioned CG on the reduced SPD system (r[pin] = 0, x[pin] = 0)
        precondition(C, P.r, P.z, sc + 4);
        dot3v(C, P.r, P.z, nullptr, sc + 6, P.z);            // rz at sc[6]
        k_fill<<<1, 32, 0, s>>>(1, sc + 51, 1.0);
        TG_PROF(C, "pois_cg_dir", k_cg_dir<<<vblocks(n), RB, 0, s>>>(n, sc, P.z, P.p));
        k_fill<<<1, 32, 0, s>>>(1, sc + 51, 0.0);
        while (!converged() && it < maxit) {
            apply_op(C, P.p, P.q);
            k_zero_at<<<1, 1, 0, s>>>(P.q, P.pin);
            dot3v(C, P.p, P.q, nullptr, sc + 9);             // pq at sc[9]
            // x += alpha p, r -= alpha q; rr, sum r, max|r aj|
            TG_PROF(C, "pois_cg_update", k_cg_update_rr<<<P.nblocks, RB, 0, s>>>(n, sc + 6, sc + 9, P.x, P.p, P.r, P.q, divtol > 0 ? P.aj : nullptr, P.part));
            k_dot_final<<<1, RB, 0, s>>>(P.part, P.nblocks, sc + 3);
            read_scal(C, 3, 3);
            rn = std::sqrt(hs[3]); rmax = hs[5] * dt;
            it++;
            if (converged()) { ok = true; break; }
            precondition(C, P.r, P.z, sc + 4);
            k_scalar_copy<<<1, 1, 0, s>>>(sc + 6, sc + 14, 1);   // rz_old
            dot3v(C, P.r, P.z, nullptr, sc + 6, P.z);            // rz_new
            TG_PROF(C, "pois_cg_dir", k_cg_dir<<<vblocks(n), RB, 0, s>>>(n, sc, P.z, P.p));
        }
    } else {
        // right-preconditioned BiCGStab on the full pinned system
        // scalars: sc[20]=rho sc[21]=alpha sc[22]=omega sc[23]=rho_old
        TG_PROF(C, "pois_copy", k_copy<<<vblocks(n), RB, 0, s>>>(n, P.r, P.rhat));
        double one[4] = {1.0, 1.0, 1.0, 1.0};
        TG_CUDA(cudaMemcpyAsync(sc + 20, one, sizeof(one), cudaMemcpyHostToDevice, s));
        TG_CUDA(cudaMemsetAsync(P.p, 0, sizeof(double) * n, s));
        TG_CUDA(cudaMemsetAsync(P.v, 0, sizeof(double) * n, s));
        double *phat = P.z, *shat = P.q;
        bool restart_pending = false;
        while (!converged() && it < maxit) {
            if ((it > 0 && (it % 50) == 0) || restart_pending) {
                // restart from the true residual (limits recursive drift)
                restart_pending = false;
                apply_op(C, P.x, P.r);
                TG_PROF(C, "pois_resid", k_resid<<<vblocks(n), RB, 0, s>>>(n, P.b, P.r));
                k_copy<<<vblocks(n), RB, 0, s>>>(n, P.r, P.rhat);
                TG_CUDA(cudaMemcpyAsync(sc + 20, one, sizeof(one), cudaMemcpyHostToDevice, s));
                TG_CUDA(cudaMemsetAsync(P.p, 0, sizeof(double) * n, s));
                TG_CUDA(cudaMemsetAsync(P.v, 0, sizeof(double) * n, s));
            }
            dot3v(C, P.rhat, P.r, nullptr, sc + 24);            // rho_new at sc[24]
            k_scalar_copy<<<1, 1, 0, s>>>(sc + 20, sc + 23, 1); // rho_old
            k_scalar_copy<<<1, 1, 0, s>>>(sc + 24, sc + 20, 1); // rho
            TG_PROF(C, "pois_bicg_p", k_bicg_p<<<vblocks(n), RB, 0, s>>>(n, sc + 20, P.p, P.r, P.v));
            dot3v(C, P.p, P.p, nullptr, sc + 27);               // sum(p) at sc[28]
            precondition(C, P.p, phat, sc + 28);
            apply_op(C, phat, P.v);
            dot3v(C, P.rhat, P.v, nullptr, sc + 30);            // rhat.v at sc[30]
            TG_PROF(C, "pois_bicg_s", k_bicg_s<<<vblocks(n), RB, 0, s>>>(n, sc + 20, sc + 30, sc + 21, P.s, P.r, P.v));
            dot3v(C, P.s, P.s, nullptr, sc + 33);               // sum(s) at sc[34]
            precondition(C, P.s, shat, sc + 34);
            apply_op(C, shat, P.t);
            dot3v(C, P.t, P.s, nullptr, sc + 36);               // t.s
            dot3v(C, P.t, P.t, nullptr, sc + 39);               // t.t
            TG_PROF(C, "pois_bicg_x", k_bicg_x<<<vblocks(n), RB, 0, s>>>(n, sc + 21, sc + 36, sc + 39, sc + 22, P.x, phat, shat, P.r, P.s, P.t));
            dot3v(C, P.r, P.r, divtol > 0 ? P.aj : nullptr, sc + 3);
            read_scal(C, 3, 3);
            rn = std::sqrt(hs[3]); rmax = hs[5] * dt;
            it++;
            if (!std::isfinite(rn)) break;
            if (converged()) {
                // the recursive residual drifts from b - L x: stop only when
                // the true residual meets the test, else restart from it
                apply_op(C, P.x, P.r);
                TG_PROF(C, "pois_resid", k_resid<<<vblocks(n), RB, 0, s>>>(n, P.b, P.r));
                dot3v(C, P.r, P.r, divtol > 0 ? P.aj : nullptr, sc + 3);
                read_scal(C, 3, 3);
                rn = std::sqrt(hs[3]); rmax = hs[5] * dt;
                if (!converged()) restart_pending = true;
            }
        }
        ok = converged();
        // true residual (reported; it may sit slightly above the recursive one at round-off level)
        apply_op(C, P.x, P.r);
        TG_PROF(C, "pois_resid", k_resid<<<vblocks(n), RB, 0, s>>>(n, P.b, P.r));
        dot3v(C, P.r, P.r, divtol > 0 ? P.aj : nullptr, sc + 3);
        read_scal(C, 3, 3);
        rn = std::sqrt(hs[3]); rmax = hs[5] * dt;
    }
    k_zero_at<<<1, 1, 0, s>>>(P.x, P.pin);
    TG_CUDA(cudaGetLastError());
    if (st) {
        st->poisson_iterations = it;
        st->poisson_total_iterations += it;
        st->poisson_final_residual = bn > 0 ? rn / bn : rn;
    }
    if (!std::isfinite(rn)) return 2;
    return ok ? 0 : 1;
}

static void direct_begin(tg_ctx *C)
{
    PoissonCtx &P = *C->pois;
    TG_PROF(C, "pois_begin", k_direct_begin<<<P.nblocks, RB, 0, C->stream>>>(C->g, C->s, P, C->prm.dt, C->d_scal + SC_PHIST, guess_order(C), C->d_scal, C->d_scal + SC_PREF));
}

// phi into the DMDA; on an axis-aligned mesh the pressure update that follows
// reads the compact solution itself
static void phi_to_dmda(tg_ctx *C)
{
    PoissonCtx &P = *C->pois;
    if (C->axis_aligned) return;
    TG_PROF(C, "pois_phi_to_dmda", k_phi_to_dmda<<<cgrid(P.nx, P.ny, P.nz), block3(), 0, C->stream>>>(C->g, C->s, P));
}

int poisson_solve(tg_ctx *C, tg_stats *st)
{
    PoissonCtx &P = *C->pois;
    const Grid g = C->g;
    cudaStream_t s = C->stream;
    const double rtol = C->cfg.poisson_rtol > 0 ? C->cfg.poisson_rtol : 1e-14;
    const int maxit = C->cfg.poisson_maxit > 0 ? C->cfg.poisson_maxit : 500;
    const dim3 cg3 = cgrid(P.nx, P.ny, P.nz);
    if (P.fdm) {
        direct_begin(C);
        const int rc = direct_solve(C, st, rtol, C->cfg.poisson_div_tol, maxit);
        phi_to_dmda(C);
        return rc;
    }
    TG_PROF(C, "pois_set_rhs", k_set_rhs<<<cg3, block3(), 0, s>>>(g, C->s, P, C->prm.dt));
    k_extrapolate<<<vblocks(P.n), RB, 0, s>>>(P.n, P.x, P.xprev, P.xprev2, C->d_scal + SC_PHIST, guess_order(C));
    k_hist_next<<<1, 1, 0, s>>>(C->d_scal + SC_PHIST);
    k_zero_at<<<1, 1, 0, s>>>(P.x, P.pin);            // warm start from the previous solutions
    int rc = krylov_solve(C, st, rtol, C->cfg.poisson_div_tol, maxit);
    phi_to_dmda(C);
    TG_CUDA(cudaGetLastError());
    return rc;
}

// ---------------------------------------------------- captured solves
// Conditional node of `type` appended to the graph being captured on
// C->stream; body() is captured into the node's body graph on the auxiliary
// stream `aux` (C->stream points there while body() runs).
template <class F>
static void capture_conditional(tg_ctx *C, cudaGraphConditionalHandle h, cudaGraphConditionalNodeType type,
                                cudaStream_t aux, F &&body)
{
    cudaStream_t s = C->stream;
    cudaStreamCaptureStatus cs;
    cudaGraph_t graph;
    const cudaGraphNode_t *deps = nullptr;
    size_t nd = 0;
    TG_CUDA(cudaStreamGetCaptureInfo(s, &cs, nullptr, &graph, &deps, &nd));
    cudaGraphNodeParams cp{};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = type;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    TG_CUDA(cudaGraphAddNode(&node, graph, deps, nd, &cp));
    cudaGraph_t bg = cp.conditional.phGraph_out[0];
    TG_CUDA(cudaStreamUpdateCaptureDependencies(s, &node, 1, cudaStreamSetCaptureDependencies));
    TG_CUDA(cudaStreamBeginCaptureToGraph(aux, bg, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    {
        struct Swap { tg_ctx *C; cudaStream_t keep; ~Swap() { C->stream = keep; } } sw{C, s};
        C->stream = aux;
        body();
    }
    cudaGraph_t done;
    TG_CUDA(cudaStreamEndCapture(aux, &done));
}

// conditional handle of the graph being captured on C->stream (no default
// value: a kernel sets it before the node runs)
static cudaGraphConditionalHandle capture_handle(tg_ctx *C)
{
    cudaStreamCaptureStatus cs;
    cudaGraph_t graph;
    TG_CUDA(cudaStreamGetCaptureInfo(C->stream, &cs, nullptr, &graph, nullptr, nullptr));
    if (cs != cudaStreamCaptureStatusActive) throw CudaError{cudaErrorStreamCaptureInvalidated, "capture_handle: stream not capturing"};
    cudaGraphConditionalHandle h;
    TG_CUDA(cudaGraphConditionalHandleCreate(&h, graph, 0, 0));
    return h;
}

// BiCGStab restarts from the true residual every 50 iterations, and after a
// true residual that missed the stopping test (sc[53] set); clears sc[53]
__global__ void k_bicg_restart_flag(double *sc, cudaGraphConditionalHandle h)
{
    const int it = (int)sc[50];
    const bool pending = sc[53] != 0.0;
    sc[53] = 0.0;
    cudaGraphSetConditional(h, ((it > 0 && (it % 50) == 0) || pending) ? 1u : 0u);
}
// the recursive residual met the stopping test: verify it on b - L x
__global__ void k_bicg_verify_flag(const double *sc, double rtol, double divtol, double dt, cudaGraphConditionalHandle h)
{
    cudaGraphSetConditional(h, cg_converged(sc, rtol, divtol, dt) ? 1u : 0u);
}
// after the verification: restart on the next pass if the true residual missed
__global__ void k_bicg_mark_restart(double *sc, double rtol, double divtol, double dt)
{
    sc[53] = cg_converged(sc, rtol, divtol, dt) ? 0.0 : 1.0;
}

// krylov_solve for a step being captured into a CUDA graph: the iterations
// form a conditional WHILE node whose condition a one-thread kernel sets from
// the device residuals, so the solve needs no host round trip per iteration.
// The CG body is krylov_solve's iteration rotated to start with the direction
// update (p = z on the first pass), the BiCGStab body is krylov_solve's with
// its restarts and its true-residual check as conditional IF nodes; both perform the same
// arithmetic in the same order. Statistics go to the ST_* slots from base.
// have_bb: |b|^2 is in sc[0] already (direct solver only).
static void krylov_capture(tg_ctx *C, double rtol, double divtol, int maxit, int base, bool have_bb = false)
{
    PoissonCtx &P = *C->pois;
    const int64_t n = P.n;
    cudaStream_t s = C->stream;
    const double dt = C->prm.dt;
    double *sc = C->d_scal;
    const int vb = vblocks(n);
    if (P.fdm) {
        if (!have_bb) dot3v(C, P.b, P.b, nullptr, sc + 0);
        const Loop L = loop_of(C, rtol, divtol, maxit, base);
        cudaGraphConditionalHandle h = capture_handle(C);
        direct_resid<true>(C, L, h);
        capture_conditional(C, h, cudaGraphCondTypeWhile, C->aux[0], [&]() { direct_pass<true>(C, L, h); });
        return;
    }
    dot3v(C, P.b, P.b, nullptr, sc + 0);
    apply_op(C, P.x, P.r);
    k_resid<<<vb, RB, 0, s>>>(n, P.b, P.r);
    dot3v(C, P.r, P.r, divtol > 0 ? P.aj : nullptr, sc + 3);
    if (P.ortho) {
        cudaGraphConditionalHandle h = capture_handle(C);
        k_cg_start<<<1, 1, 0, s>>>(sc, rtol, divtol, dt, maxit, h, base);
        capture_conditional(C, h, cudaGraphCondTypeWhile, C->aux[0], [&]() {
            cudaStream_t a = C->stream;
            precondition(C, P.r, P.z, sc + 4);
            k_scalar_copy<<<1, 1, 0, a>>>(sc + 6, sc + 14, 1);           // rz_old
            dot3v(C, P.r, P.z, nullptr, sc + 6, P.z);                     // rz
            k_cg_dir<<<vb, RB, 0, a>>>(n, sc, P.z, P.p);
            apply_op(C, P.p, P.q);
            k_zero_at<<<1, 1, 0, a>>>(P.q, P.pin);
            dot3v(C, P.p, P.q, nullptr, sc + 9);                          // pq
            k_cg_update_rr<<<P.nblocks, RB, 0, a>>>(n, sc + 6, sc + 9, P.x, P.p, P.r, P.q, divtol > 0 ? P.aj : nullptr, P.part);
            k_dot_final<<<1, RB, 0, a>>>(P.part, P.nblocks, sc + 3);      // rr, sum r, max|r aj|
            k_cg_next<<<1, 1, 0, a>>>(sc, rtol, divtol, dt, maxit, h);
        });
    } else {
        k_copy<<<vb, RB, 0, s>>>(n, P.r, P.rhat);
        k_fill<<<1, 32, 0, s>>>(4, sc + 20, 1.0);
        k_fill<<<vb, RB, 0, s>>>(n, P.p, 0.0);
        k_fill<<<vb, RB, 0, s>>>(n, P.v, 0.0);
        double *phat = P.z, *shat = P.q;
        cudaGraphConditionalHandle h = capture_handle(C);
        k_cg_start<<<1, 1, 0, s>>>(sc, rtol, divtol, dt, maxit, h, base);
        capture_conditional(C, h, cudaGraphCondTypeWhile, C->aux[0], [&]() {
            cudaStream_t a = C->stream;
            cudaGraphConditionalHandle hr = capture_handle(C);
            k_bicg_restart_flag<<<1, 1, 0, a>>>(sc, hr);
            capture_conditional(C, hr, cudaGraphCondTypeIf, C->aux[1], [&]() {
                cudaStream_t b = C->stream;
                apply_op(C, P.x, P.r);
                k_resid<<<vb, RB, 0, b>>>(n, P.b, P.r);
                k_copy<<<vb, RB, 0, b>>>(n, P.r, P.rhat);
                k_fill<<<1, 32, 0, b>>>(4, sc + 20, 1.0);
                k_fill<<<vb, RB, 0, b>>>(n, P.p, 0.0);
                k_fill<<<vb, RB, 0, b>>>(n, P.v, 0.0);
            });
            dot3v(C, P.rhat, P.r, nullptr, sc + 24);
            k_scalar_copy<<<1, 1, 0, a>>>(sc + 20, sc + 23, 1);
            k_scalar_copy<<<1, 1, 0, a>>>(sc + 24, sc + 20, 1);
            k_bicg_p<<<vb, RB, 0, a>>>(n, sc + 20, P.p, P.r, P.v);
            dot3v(C, P.p, P.p, nullptr, sc + 27);
            precondition(C, P.p, phat, sc + 28);
            apply_op(C, phat, P.v);
            dot3v(C, P.rhat, P.v, nullptr, sc + 30);
            k_bicg_s<<<vb, RB, 0, a>>>(n, sc + 20, sc + 30, sc + 21, P.s, P.r, P.v);
            dot3v(C, P.s, P.s, nullptr, sc + 33);
            precondition(C, P.s, shat, sc + 34);
            apply_op(C, shat, P.t);
            dot3v(C, P.t, P.s, nullptr, sc + 36);
            dot3v(C, P.t, P.t, nullptr, sc + 39);
            k_bicg_x<<<vb, RB, 0, a>>>(n, sc + 21, sc + 36, sc + 39, sc + 22, P.x, phat, shat, P.r, P.s, P.t);
            dot3v(C, P.r, P.r, divtol > 0 ? P.aj : nullptr, sc + 3);
            cudaGraphConditionalHandle hv = capture_handle(C);
            k_bicg_verify_flag<<<1, 1, 0, a>>>(sc, rtol, divtol, dt, hv);
            capture_conditional(C, hv, cudaGraphCondTypeIf, C->aux[1], [&]() {
                cudaStream_t b = C->stream;
                apply_op(C, P.x, P.r);
                k_resid<<<vb, RB, 0, b>>>(n, P.b, P.r);
                dot3v(C, P.r, P.r, divtol > 0 ? P.aj : nullptr, sc + 3);
                k_bicg_mark_restart<<<1, 1, 0, b>>>(sc, rtol, divtol, dt);
            });
            k_cg_next<<<1, 1, 0, a>>>(sc, rtol, divtol, dt, maxit, h);
        });
        // true residual (reported)
        apply_op(C, P.x, P.r);
        k_resid<<<vb, RB, 0, s>>>(n, P.b, P.r);
        dot3v(C, P.r, P.r, divtol > 0 ? P.aj : nullptr, sc + 3);
    }
    k_zero_at<<<1, 1, 0, s>>>(P.x, P.pin);
    k_cg_finish<<<1, 1, 0, s>>>(sc, base);
}

// poisson_solve for a step being captured into a CUDA graph
void poisson_solve_capture(tg_ctx *C)
{
    PoissonCtx &P = *C->pois;
    const Grid g = C->g;
    cudaStream_t s = C->stream;
    const double rtol = C->cfg.poisson_rtol > 0 ? C->cfg.poisson_rtol : 1e-14;
    const int maxit = C->cfg.poisson_maxit > 0 ? C->cfg.poisson_maxit : 500;
    const dim3 cg3 = cgrid(P.nx, P.ny, P.nz);
    if (P.fdm) {
        direct_begin(C);
    } else {
        k_set_rhs<<<cg3, block3(), 0, s>>>(g, C->s, P, C->prm.dt);
        k_extrapolate<<<vblocks(P.n), RB, 0, s>>>(P.n, P.x, P.xprev, P.xprev2, C->d_scal + SC_PHIST, guess_order(C));
        k_hist_next<<<1, 1, 0, s>>>(C->d_scal + SC_PHIST);
        k_zero_at<<<1, 1, 0, s>>>(P.x, P.pin);
    }
    krylov_capture(C, rtol, C->cfg.poisson_div_tol, maxit, SC_G, P.fdm != nullptr);
    phi_to_dmda(C);
    TG_CUDA(cudaGetLastError());
}

// poisson_solve_adjoint for a reversed step being captured into a CUDA graph
// (statistics in the SC_ADJ slots)
void poisson_solve_adjoint_capture(tg_ctx *C, const double *rhs, double *lam, double rtol)
{
    PoissonCtx &P = *C->pois;
    cudaStream_t s = C->stream;
    const int64_t n = P.n;
    TG_CUDA(cudaMemcpyAsync(P.v, P.x, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    k_negcopy<<<vblocks(n), RB, 0, s>>>(n, rhs, P.b);
    k_zero_at<<<1, 1, 0, s>>>(P.b, P.pin);
    TG_CUDA(cudaMemcpyAsync(P.x, lam, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    krylov_capture(C, rtol, 0.0, C->cfg.poisson_maxit > 0 ? C->cfg.poisson_maxit : 500, SC_ADJ);
    TG_CUDA(cudaMemcpyAsync(lam, P.x, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    TG_CUDA(cudaMemcpyAsync(P.x, P.v, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    TG_CUDA(cudaGetLastError());
}

// Adjoint pressure solve: lam = A^-T rhs for the pinned operator A of
// SetCoeffMatrix (rhs and lam compact, pinned entry of rhs ignored,
// lam[pin] = 0). On orthogonal grids the operator without the pinned row and
// column is symmetric, so this is the forward Krylov solve started from the
// value lam holds on entry (the caller's guess, adjoint_guess); the
// forward warm start P.x is kept. Returns 3 for the non-symmetric curvilinear
// operator.
int poisson_solve_adjoint(tg_ctx *C, const double *rhs, double *lam, double rtol, tg_stats *st)
{
    PoissonCtx &P = *C->pois;
    if (!P.ortho) return 3;
    cudaStream_t s = C->stream;
    const int64_t n = P.n;
    TG_CUDA(cudaMemcpyAsync(P.v, P.x, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    k_negcopy<<<vblocks(n), RB, 0, s>>>(n, rhs, P.b);       // the solver's operator is L = -A
    k_zero_at<<<1, 1, 0, s>>>(P.b, P.pin);
    TG_CUDA(cudaMemcpyAsync(P.x, lam, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    int rc = krylov_solve(C, st, rtol, 0.0, C->cfg.poisson_maxit > 0 ? C->cfg.poisson_maxit : 500);
    TG_CUDA(cudaMemcpyAsync(lam, P.x, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    TG_CUDA(cudaMemcpyAsync(P.x, P.v, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    return rc;
}

void adjoint_guess(tg_ctx *C, double *lam, double *lp, double *lp2, double *hist)
{
    PoissonCtx &P = *C->pois;
    cudaStream_t s = C->stream;
    k_extrapolate<<<vblocks(P.n), RB, 0, s>>>(P.n, lam, lp, lp2, hist, guess_order(C));
    k_hist_next<<<1, 1, 0, s>>>(hist);
    k_zero_at<<<1, 1, 0, s>>>(lam, P.pin);
    TG_CUDA(cudaGetLastError());
}

// compact Poisson solution vectors (the next solve extrapolates x, xprev, xprev2): snapshots
bool poisson_direct(const tg_ctx *C) { return C->pois->fdm != nullptr; }
double *poisson_x(tg_ctx *C) { return C->pois->x; }
double *poisson_xprev(tg_ctx *C) { return C->pois->xprev; }
double *poisson_xprev2(tg_ctx *C) { return C->pois->xprev2; }
int64_t poisson_n(tg_ctx *C) { return C->pois->n; }

}  // namespace tg
