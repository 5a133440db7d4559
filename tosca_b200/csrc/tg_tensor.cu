// Stage kernels on a mesh of planes (csi || y, eta || z, zet || x: the node
// coordinates are x(k), y(i), z(j)). Every metric of such a mesh is a product
// of one-dimensional spacings, so these kernels read six short arrays, which
// stay in the L1 cache, where the general kernels of tg_step.cu read 1 to 30
// metric values per cell from memory; the products that remain are those of
// the general formulas whose metric factors do not vanish, in FP64 in both
// precision modes (they read no metric copies that FP32 would shrink).
//
// Notation: at cell (k, j, i) dx = dx_k, dy = dy_i, dz = dz_j are the cell
// sizes and dxf, dyf, dzf the distances that the face metrics use across the
// k, i and j faces (mesh.c:1354-1930). Then
//     csi.y = dx dz, eta.z = dx dy, zet.x = dy dz, aj = 1/(dx dy dz),
// and at the i face icsi.y = dx dz, ieta.z = dx dyf, izet.x = dyf dz,
// iaj = 1/(dx dyf dz), the j and k faces likewise with dzf and dxf.
#include <algorithm>
#include <cmath>
#include <vector>

#include "tg_rk.cuh"

namespace tg {
namespace {

// ------------------------------------------------------------- detection
// largest relative deviation of the metric components from their products
// (cell metrics on all points, face metrics on the faces of interior rows)
__global__ void __launch_bounds__(256) k_tensor_check(Grid g, FaceMet<double> m, Tensor t, double *part)
{
    const int64_t n = g.size();
    double mm = 0.0;
    auto dev = [&](double a, double b) { mm = nanmax(mm, fabs(a / b - 1.0)); };
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(c % g.mx);
        const int64_t r = c / g.mx;
        const int j = (int)(r % g.my), k = (int)(r / g.my);
        const bool ii = i >= 1 && i <= g.mx - 2, jj = j >= 1 && j <= g.my - 2, kk = k >= 1 && k <= g.mz - 2;
        const double dx = t.dx[k], dy = t.dy[i], dz = t.dz[j];
        // cell metrics are mirrored into the face-adjacent ghosts
        if ((int)ii + (int)jj + (int)kk >= 2) {
            dev(m.csi.y[c], dx * dz); dev(m.eta.z[c], dx * dy); dev(m.zet.x[c], dy * dz);
            dev(m.aj[c] * (dx * dy * dz), 1.0);
        }
        if (kk && jj && i <= g.mx - 2) {
            const double d = t.dyf[i];
            dev(m.icsi.y[c], dx * dz); dev(m.ieta.z[c], dx * d); dev(m.izet.x[c], d * dz); dev(m.iaj[c] * (dx * d * dz), 1.0);
        }
        if (kk && ii && j <= g.my - 2) {
            const double d = t.dzf[j];
            dev(m.jcsi.y[c], dx * d); dev(m.jeta.z[c], dx * dy); dev(m.jzet.x[c], dy * d); dev(m.jaj[c] * (dx * dy * d), 1.0);
        }
        if (jj && ii && k <= g.mz - 2) {
            const double d = t.dxf[k];
            dev(m.kcsi.y[c], d * dz); dev(m.keta.z[c], d * dy); dev(m.kzet.x[c], dy * dz); dev(m.kaj[c] * (d * dy * dz), 1.0);
        }
    }
    double v[1] = {mm};
    block_reduce<256>(v, RedNanMax{});
    if (threadIdx.x == 0) part[blockIdx.x] = v[0];
}

// ------------------------------------------------ contravariantToCartesian
// ueqn.c:528-635 (k_contra_to_cart): the Cramer products reduce to one face
// area per component
__global__ void k_contra_tensor(Grid g, Tensor t, State s)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1, k = blockIdx.z * blockDim.z + threadIdx.z + 1;
    if (i > g.mx - 2 || j > g.my - 2 || k > g.mz - 2) return;
    const int c = g.lin(k, j, i);
    const double rx = t.rdx[k], ry = t.rdy[i], rz = t.rdz[j];
    s.ucat.x[c] = (0.5 * (s.ucont.z[c - g.mx * g.my] + s.ucont.z[c])) * (ry * rz);
    s.ucat.y[c] = (0.5 * (s.ucont.x[c - 1] + s.ucont.x[c])) * (rx * rz);
    s.ucat.z[c] = (0.5 * (s.ucont.y[c - g.mx] + s.ucont.y[c])) * (rx * ry);
}

// ------------------------------------------------------------ Smagorinsky
// k_smagorinsky (les.c:172-178, 2119-2514): nut = Cs^2 D^2 sqrt(2 S:S)
__global__ void k_smagorinsky_tensor(Grid g, Tensor t, State s, double cs)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1, k = blockIdx.z * blockDim.z + threadIdx.z + 1;
    if (i > g.mx - 2 || j > g.my - 2 || k > g.mz - 2) return;
    const int c = g.lin(k, j, i), pl = g.mx * g.my;
    // central, or one-sided next to a non-periodic boundary
    const bool ir = !g.pi && i == g.mx - 2, il = !g.pi && i == 1, jr = !g.pj && j == g.my - 2, jl = !g.pj && j == 1,
               kr = !g.pk && k == g.mz - 2, kl = !g.pk && k == 1;
    const int ip = ir ? c : c + 1, im = (il && !ir) ? c : c - 1;
    const int jp = jr ? c : c + g.mx, jm = (jl && !jr) ? c : c - g.mx;
    const int kp = kr ? c : c + pl, km = (kl && !kr) ? c : c - pl;
    const double hx = ((kr || kl) ? 1.0 : 0.5) * t.rdx[k], hy = ((ir || il) ? 1.0 : 0.5) * t.rdy[i], hz = ((jr || jl) ? 1.0 : 0.5) * t.rdz[j];
    const V3f<double> &u = s.ucat;
    const double dudx = hx * (u.x[kp] - u.x[km]), dvdx = hx * (u.y[kp] - u.y[km]), dwdx = hx * (u.z[kp] - u.z[km]);
    const double dudy = hy * (u.x[ip] - u.x[im]), dvdy = hy * (u.y[ip] - u.y[im]), dwdy = hy * (u.z[ip] - u.z[im]);
    const double dudz = hz * (u.x[jp] - u.x[jm]), dvdz = hz * (u.y[jp] - u.y[jm]), dwdz = hz * (u.z[jp] - u.z[jm]);
    const double sxy = dudy + dvdx, sxz = dudz + dwdx, syz = dvdz + dwdy;
    // 2 S:S = 2 (sum of squared diagonals) + (sum of squared doubled off-diagonals)
    const double q = 2.0 * (dudx * dudx + dvdy * dvdy + dwdz * dwdz) + (sxy * sxy + sxz * sxz + syz * syz);
    s.nut[c] = cs * (t.qx[k] * t.qy[i] * t.qz[j]) * sqrt(q);
}

// ------------------------------------------------------------------ GradP
// k_grad_p (peqn.c:3437-3773) at the + faces of interior cell c
__device__ __forceinline__ R3<double> grad_p_cell(const Grid &g, const Tensor &t, const double *p, int k, int j, int i, int c)
{
    const int pl = g.mx * g.my;
    const double dx = t.dx[k], dy = t.dy[i], dz = t.dz[j], pc = p[c];
    // the + neighbours lie inside the DMDA except across a periodic seam, where
    // index m + 1 wraps to 1
    const double pi = i == g.mx - 2 ? p[g.pi ? g.lin(k, j, 1) : c] : p[c + 1];
    const double pj = j == g.my - 2 ? p[g.pj ? g.lin(k, 1, i) : c] : p[c + g.mx];
    const double pk = k == g.mz - 2 ? p[g.pk ? g.lin(1, j, i) : c] : p[c + pl];
    return R3<double>{(pi - pc) * (dx * dz * t.rdyf[i]), (pj - pc) * (dx * dy * t.rdzf[j]), (pk - pc) * (dy * dz * t.rdxf[k])};
}
__global__ void k_grad_p_tensor(Grid g, Tensor t, State s)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1, k = blockIdx.z * blockDim.z + threadIdx.z + 1;
    if (i > g.mx - 2 || j > g.my - 2 || k > g.mz - 2) return;
    const int c = g.lin(k, j, i);
    st3(s.dp, c, grad_p_cell(g, t, s.p, k, j, i, c));
}

// ------------------------------------------------- FormU: cell budgets
// The budget of a cell outside the box of the lean kernel, with every boundary
// rule of the face fluxes (ueqn_solvers.c:173-778 with Compute_du_i,
// Compute_du_j, Compute_du_k, inline.h:2748-2931): one-sided cross derivatives
// at boundary faces along the domain edges, no viscous flux on slip patches,
// the wall stress in place of the eddy viscosity on the wall function's, and
// the periodic face 0 taken from the face m - 2 (resetFacePeriodicFluxesVector,
// inline.h:5357-5451).
template <int mode>
__device__ __forceinline__ R3<double> fp_boundary_cell(const Grid &g, const Tensor &t, const State &s, const Params &p, int k, int j, int i)
{
    const int mx = g.mx, my = g.my, mz = g.mz, pl = mx * my;
    const bool npi = !g.pi, npj = !g.pj, npk = !g.pk;
    auto U = [&](int q) { return ld3(s.ucat, q); };
    auto nuf = [&](int q, int e) { return p.les ? p.nu + 0.5 * (s.nut[q] + s.nut[e]) : p.nu; };
    auto slip = [&](int patch_, bool on) { return p.les && on && p.bc[patch_] == TG_BC_SLIP; };
    // derivative of the face value along a direction of stride st (cells at
    // index l of 1 .. m-2): central, or one-sided at a boundary face when either
    // direction is bounded; q and e are the two cells of the face
    auto cross = [&](int q, int e, int st, int l, int m, bool edge, bool np) {
        const R3<double> s0 = U(q) + U(e);
        if (edge && np && l == m - 2) return 0.5 * (s0 - (U(q - st) + U(e - st)));
        if (edge && np && l == 1) return 0.5 * ((U(q + st) + U(e + st)) - s0);
        return 0.25 * ((U(q + st) + U(e + st)) - (U(q - st) + U(e - st)));
    };
    auto conv = [&](int q, int e, double uc) { return mode == 2 ? R3<double>{0.0, 0.0, 0.0} : (-0.5 * uc) * (U(q) + U(e)); };
    // a periodic direction takes its face 0 from its face m - 2
    auto iface = [&](int fi) {
        if (fi == 0 && g.pi) fi = mx - 2;
        const int q = g.lin(k, j, fi), e = q + 1;
        const bool edge = fi == 0 || fi == mx - 2;
        R3<double> f = conv(q, e, s.ucont.x[q]);
        if (mode != 1) {
            const double n = (slip(TG_ILEFT, fi == 0) || slip(TG_IRIGHT, fi == mx - 2)) ? 0.0 : nuf(q, e);
            const double w = n * (t.dx[k] * t.dz[j] * t.rdyf[fi]);
            const R3<double> dc = U(e) - U(q);
            const double vx = cross(q, e, pl, k, mz, edge, npk || npi).y, vz = cross(q, e, mx, j, my, edge, npj || npi).y;
            f = f + R3<double>{w * dc.x + n * t.dz[j] * vx, 2.0 * w * dc.y, w * dc.z + n * t.dx[k] * vz};
        }
        return f;
    };
    auto jface = [&](int fj) {
        if (fj == 0 && g.pj) fj = my - 2;
        const int q = g.lin(k, fj, i), e = q + mx;
        const bool edge = fj == 0 || fj == my - 2;
        R3<double> f = conv(q, e, s.ucont.y[q]);
        if (mode != 1) {
            double n = nuf(q, e);
            // both j patches read the jLeft wall stress, ueqn_solvers.c:548-558
            if (p.les && ((p.bc[TG_JLEFT] == TG_BC_WALL_SHUMANN && fj == 0) || (p.bc[TG_JRIGHT] == TG_BC_WALL_SHUMANN && fj == my - 2))) {
                const int w = k * mx + i;
                f = f - R3<double>{s.twx[w], s.twy[w], s.twz[w]};
                n = p.nu;
            } else if (slip(TG_JLEFT, fj == 0) || slip(TG_JRIGHT, fj == my - 2)) n = 0.0;
            const double w = n * (t.dx[k] * t.dy[i] * t.rdzf[fj]);
            const R3<double> de = U(e) - U(q);
            const double wx = cross(q, e, pl, k, mz, edge, npk || npj).z, wy = cross(q, e, 1, i, mx, edge, npi || npj).z;
            f = f + R3<double>{w * de.x + n * t.dy[i] * wx, w * de.y + n * t.dx[k] * wy, 2.0 * w * de.z};
        }
        return f;
    };
    auto kface = [&](int fk) {
        if (fk == 0 && g.pk) fk = mz - 2;
        const int q = g.lin(fk, j, i), e = q + pl;
        const bool edge = fk == 0 || fk == mz - 2;
        R3<double> f = conv(q, e, s.ucont.z[q]);
        if (mode != 1) {
            const double n = (slip(TG_KLEFT, fk == 0) || slip(TG_KRIGHT, fk == mz - 2)) ? 0.0 : nuf(q, e);
            const double w = n * (t.dy[i] * t.dz[j] * t.rdxf[fk]);
            const R3<double> dk = U(e) - U(q);
            const double uy = cross(q, e, 1, i, mx, edge, npi || npk).x, uz = cross(q, e, mx, j, my, edge, npj || npk).x;
            f = f + R3<double>{2.0 * w * dk.x, w * dk.y + n * t.dz[j] * uy, w * dk.z + n * t.dy[i] * uz};
        }
        return f;
    };
    R3<double> f = iface(i) - iface(i - 1);
    f = f + (jface(j) - jface(j - 1));
    return f + (kface(k) - kface(k - 1));
}

// the boundary cells of block `blk` of boundary_blocks(): 32 x 8 cells of one of
// the six boundary planes; a cell on several planes belongs to the first
struct Box { int i0, i1, j0, j1, k0, k1; };   // cells of the lean kernel
inline __host__ __device__ void plane_blocks(const Grid &g, int patch, int &na, int &nb)
{
    const int dir = patch >> 1;
    na = ((dir == 0 ? g.my : g.mx) - 2 + 31) / 32;
    nb = ((dir == 2 ? g.my : g.mz) - 2 + 7) / 8;
}
inline int boundary_blocks(const Grid &g)
{
    int n = 0;
    for (int q = 0; q < 6; q++) { int na, nb; plane_blocks(g, q, na, nb); n += na * nb; }
    return n;
}
template <int mode>
__device__ void fp_boundary_block(const Grid &g, const Tensor &t, const State &s, const V3f<double> &fp, const Params &p, const Box &b, int blk)
{
    int patch = 0, na, nb;
    for (;; patch++) {
        plane_blocks(g, patch, na, nb);
        if (blk < na * nb) break;
        blk -= na * nb;
    }
    const int dir = patch >> 1, right = patch & 1;
    const int u = (blk % na) * 32 + threadIdx.x + 1, v = (blk / na) * 8 + threadIdx.y + 1;
    int i, j, k;
    if (dir == 0) { i = right ? g.mx - 2 : 1; j = u; k = v; }
    else if (dir == 1) { j = right ? g.my - 2 : 1; i = u; k = v; }
    else { k = right ? g.mz - 2 : 1; i = u; j = v; }
    if (i > g.mx - 2 || j > g.my - 2 || k > g.mz - 2) return;
    const bool oi = i < b.i0 || i > b.i1, oj = j < b.j0 || j > b.j1, ok = k < b.k0 || k > b.k1;
    if (!(dir == 0 ? oi : dir == 1 ? oj : ok) || (dir > 0 && oi) || (dir > 1 && oj)) return;
    st3(fp, g.lin(k, j, i), fp_boundary_cell<mode>(g, t, s, p, k, j, i));
}

// FormU passes 1 and 2 (ueqn_solvers.c:173-947) with central convection in one
// kernel: fp = sum of the convective and viscous fluxes of the six faces.
//
// The two-pass form (one thread per cell for its three + faces, the nine flux
// components through memory) took 494 + 127 us at 256 x 256 x 128, 1025 + 90
// instructions per cell: generic face rules, index arithmetic and 24 global
// loads per cell around 105 operations of flux. Here a face flux is about 26
// FP64 operations, so a thread forms five faces of its cell (the sixth is the
// top face of the cell below, which it handled before) and nothing but fp
// leaves the SM: 385 instructions per cell, 220 us and 27 for the boundary
// cells. Cells whose faces need a boundary rule (next to a non-periodic
// boundary, or the first of a periodic direction, whose face 0 is the face m-2)
// go to blocks of their own (the first of the grid: they run longest), which
// keeps those rules out of the others.
//
// A block takes 32 x 8 columns of KZ cells along k; Ucat and nut of its cells
// and one cell around them are copied asynchronously into shared memory.
constexpr int PX = 32, PY = 8, PTX = PX + 2, PTY = PY + 2;

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int mode, bool LES, int KZ>
__global__ void __launch_bounds__(PX * PY, 2) k_fp_tensor(Grid g, Tensor t, State s, V3f<double> fp, Params p, Box b, int nbnd, int nbi, int nbj)
{
    static_assert(PX == 32 && PY == 8, "blocks of boundary cells");
    if ((int)blockIdx.x < nbnd) { fp_boundary_block<mode>(g, t, s, fp, p, b, blockIdx.x); return; }
    constexpr int TN = PTX * PTY * (KZ + 2), J = PTX, K = PTX * PTY;
    extern __shared__ double sh[];
    double *U0 = sh, *U1 = sh + TN, *U2 = sh + 2 * TN, *N = sh + 3 * TN;
    const int mx = g.mx, my = g.my, mz = g.mz, pl = mx * my;
    const double nu = p.nu;
    const int blk = blockIdx.x - nbnd, bi = blk % nbi, br = blk / nbi;
    const int i0 = b.i0 + bi * PX, j0 = b.j0 + (br % nbj) * PY, k0 = b.k0 + (br / nbj) * KZ;
    const int lane = threadIdx.x, wid = threadIdx.y;
    // tile rows of 34: a lane each, the last two by lanes 0 and 1. Rows and
    // columns beyond the DMDA are not read by any cell of the block.
    for (int r = wid; r < PTY * (KZ + 2); r += PY) {
        const int ty = r % PTY, tz = r / PTY, gj = j0 - 1 + ty, gk = k0 - 1 + tz;
        if (gj >= my || gk >= mz) continue;
        const int q = r * PTX, row = (gk * my + gj) * mx + i0 - 1;
        auto put = [&](int tx) {
            if (i0 - 1 + tx >= mx) return;
            cp_async8(U0 + q + tx, s.ucat.x + row + tx);
            cp_async8(U1 + q + tx, s.ucat.y + row + tx);
            cp_async8(U2 + q + tx, s.ucat.z + row + tx);
            if (LES && mode != 1) cp_async8(N + q + tx, s.nut + row + tx);
        };
        put(lane);
        if (lane < 2) put(PX + lane);
    }
    cp_async_wait_all();
    __syncthreads();
    const int i = i0 + threadIdx.x, j = j0 + threadIdx.y;
    if (i > b.i1 || j > b.j1) return;
    const double dy = t.dy[i], dz = t.dz[j];
    const double ryE = t.rdyf[i], ryW = t.rdyf[i - 1], rzN = t.rdzf[j], rzS = t.rdzf[j - 1];
    int q = (PTY + threadIdx.y + 1) * PTX + threadIdx.x + 1;      // tile index of the current cell
    int c = g.lin(k0, j, i);
    const double qdz = 0.25 * dz, qdy = 0.25 * dy;
    auto nuf = [&](int a, int e) { return LES ? nu + 0.5 * (N[a] + N[e]) : nu; };
    // i face between tile points a and a + 1: uc its flux, I1 = iaj icsi^2,
    // 4 qdx = iaj icsi ieta (with d/deta of v), 4 qdz = iaj icsi izet
    auto iface = [&](int a, double uc, double I1, double qdx) {
        R3<double> f{0.0, 0.0, 0.0};
        const int e = a + 1;
        const double x0 = U0[a], x1 = U0[e], y0 = U1[a], y1 = U1[e], z0 = U2[a], z1 = U2[e];
        if (mode != 2) { const double h = -0.5 * uc; f.x = h * (x0 + x1); f.y = h * (y0 + y1); f.z = h * (z0 + z1); }
        if (mode != 1) {
            const double n = nuf(a, e), w = n * I1;
            const double vx = (U1[e + K] + U1[a + K]) - (U1[e - K] + U1[a - K]), vz = (U1[e + J] + U1[a + J]) - (U1[e - J] + U1[a - J]);
            f.x += w * (x1 - x0) + (n * qdz) * vx;
            f.y += (2.0 * w) * (y1 - y0);
            f.z += w * (z1 - z0) + (n * qdx) * vz;
        }
        return f;
    };
    // j face between a and a + J: J1 = jaj jeta^2; derivatives of w along x, y
    auto jface = [&](int a, double uc, double J1, double qdx) {
        R3<double> f{0.0, 0.0, 0.0};
        const int e = a + J;
        const double x0 = U0[a], x1 = U0[e], y0 = U1[a], y1 = U1[e], z0 = U2[a], z1 = U2[e];
        if (mode != 2) { const double h = -0.5 * uc; f.x = h * (x0 + x1); f.y = h * (y0 + y1); f.z = h * (z0 + z1); }
        if (mode != 1) {
            const double n = nuf(a, e), w = n * J1;
            const double wx = (U2[e + K] + U2[a + K]) - (U2[e - K] + U2[a - K]), wy = (U2[e + 1] + U2[a + 1]) - (U2[e - 1] + U2[a - 1]);
            f.x += w * (x1 - x0) + (n * qdy) * wx;
            f.y += w * (y1 - y0) + (n * qdx) * wy;
            f.z += (2.0 * w) * (z1 - z0);
        }
        return f;
    };
    // k face between a and a + K: K1 = kaj kzet^2; derivatives of u along y, z
    auto kface = [&](int a, double uc, double K1) {
        R3<double> f{0.0, 0.0, 0.0};
        const int e = a + K;
        const double x0 = U0[a], x1 = U0[e], y0 = U1[a], y1 = U1[e], z0 = U2[a], z1 = U2[e];
        if (mode != 2) { const double h = -0.5 * uc; f.x = h * (x0 + x1); f.y = h * (y0 + y1); f.z = h * (z0 + z1); }
        if (mode != 1) {
            const double n = nuf(a, e), w = n * K1;
            const double uy = (U0[e + 1] + U0[a + 1]) - (U0[e - 1] + U0[a - 1]), uz = (U0[e + J] + U0[a + J]) - (U0[e - J] + U0[a - J]);
            f.x += (2.0 * w) * (x1 - x0);
            f.y += w * (y1 - y0) + (n * qdz) * uy;
            f.z += w * (z1 - z0) + (n * qdy) * uz;
        }
        return f;
    };
    const double dydz = dy * dz;
    R3<double> bot = kface(q - K, s.ucont.z[c - pl], dydz * t.rdxf[k0 - 1]);
    #pragma unroll
    for (int kz = 0; kz < KZ; kz++, q += K, c += pl) {
        const int k = k0 + kz;
        if (k > b.k1) break;
        const double dx = t.dx[k], qdx = 0.25 * dx, dxdz = dx * dz, dxdy = dx * dy;
        const R3<double> top = kface(q, s.ucont.z[c], dydz * t.rdxf[k]);
        R3<double> f = top - bot;
        bot = top;
        f = f + (iface(q, s.ucont.x[c], dxdz * ryE, qdx) - iface(q - 1, s.ucont.x[c - 1], dxdz * ryW, qdx));
        f = f + (jface(q, s.ucont.y[c], dxdy * rzN, qdx) - jface(q - J, s.ucont.y[c - mx], dxdy * rzS, qdx));
        st3(fp, c, f);
    }
}

// ------------------------------------------------ stage fluxes from Ucont
// One explicit stage's fp straight from Ucont: the flux resets of
// ExplicitRhsU (resetNoPenetrationFluxes, resetFacePeriodicFluxes,
// inline.h:5262-5451), contravariantToCartesian, its periodic ghost copies and
// FormU passes 1 and 2 without the launches and the memory passes between them.
// Ucat is not written: no stage reads it from memory, and the step converts
// again after the projection.
//
// The resets are index rules here. Periodic directions are read through the
// wrap 0 -> m-2, m-1 -> 1 of cells and faces; wall faces are zero, set once
// before the first stage and again by each update (k_rhs_tensor); and the ghost
// cells of non-periodic directions come from Ucat, where they keep the values
// of the previous step's UpdateCartesianBCs as in the reference.
//
// A block marches its 32 x 8 columns through a chunk of planes. Ucont and nut of
// plane k+3 are copied asynchronously into a ring of four planes while plane k
// is worked on; each plane is converted once into a ring of four planes of
// Ucat. At 256 x 256 x 128 a launch takes 235 us (302 with two barriers per plane
// and ring slots from a modulus) against 90 + 220 + 27 for the conversion, the
// tile kernel and the boundary cells that it replaces, without their 10 launches
// of boundary kernels per stage, which is what bounds small grids (Taylor-Green
// 32^3 0.255 -> 0.167 ms a step). 462 instructions per cell; it is bound by the
// latency of its FP64 and shared-memory chains at two blocks per SM (43 % of
// issue slots, DRAM at 25 %). Three blocks (80 registers, 75 KB) took a step from
// 3.00 to 3.27 ms: what a thread overlaps is worth more than the warps.
__device__ __forceinline__ bool wall_patch(const Params &p, int q)
{
    const int t = p.bc[q];
    return t == TG_BC_NOSLIP || t == TG_BC_SLIP || t == TG_BC_WALL_SHUMANN;
}
// index of a cell or face of 1 .. m-2 in a periodic direction, others unchanged
__device__ __forceinline__ int wrap1(int l, int m, int per)
{
    if (per) { if (l < 1) l += m - 2; else if (l > m - 2) l -= m - 2; }
    return l;
}

// the stage's Ucont and Ucat at any point, for the cells along domain edges and
// the boundary planes. Components are numbered by direction: 0 the velocity
// along i (y), 1 along j (z), 2 along k (x).
struct StageField {
    const Grid &g;
    const Tensor &t;
    const State &s;
    const Params &p;
    __device__ __forceinline__ double v(int d, int k, int j, int i) const
    {
        i = wrap1(i, g.mx, g.pi); j = wrap1(j, g.my, g.pj); k = wrap1(k, g.mz, g.pk);
        const int l = d == 0 ? i : d == 1 ? j : k, m = d == 0 ? g.mx : d == 1 ? g.my : g.mz;
        if ((l == 0 && wall_patch(p, 2 * d)) || (l == m - 2 && wall_patch(p, 2 * d + 1))) return 0.0;
        return (d == 0 ? s.ucont.x : d == 1 ? s.ucont.y : s.ucont.z)[g.lin(k, j, i)];
    }
    __device__ __forceinline__ double u(int d, int k, int j, int i) const
    {
        i = wrap1(i, g.mx, g.pi); j = wrap1(j, g.my, g.pj); k = wrap1(k, g.mz, g.pk);
        if (i < 1 || i > g.mx - 2 || j < 1 || j > g.my - 2 || k < 1 || k > g.mz - 2)
            return (d == 0 ? s.ucat.y : d == 1 ? s.ucat.z : s.ucat.x)[g.lin(k, j, i)];
        const double r = d == 0 ? t.rdx[k] * t.rdz[j] : d == 1 ? t.rdx[k] * t.rdy[i] : t.rdy[i] * t.rdz[j];
        return (0.5 * (v(d, k - (d == 2), j - (d == 1), i - (d == 0)) + v(d, k, j, i))) * r;
    }
    __device__ __forceinline__ double nu(int k, int j, int i) const
    {
        return s.nut[g.lin(wrap1(k, g.mz, g.pk), wrap1(j, g.my, g.pj), wrap1(i, g.mx, g.pi))];
    }
};

// a cell is along a domain edge if two directions are at their first or last
// cell and one of them is bounded: only there do the cross derivatives change
__device__ __forceinline__ bool edge_cell(const Grid &g, int k, int j, int i)
{
    const bool bi = i == 1 || i == g.mx - 2, bj = j == 1 || j == g.my - 2, bk = k == 1 || k == g.mz - 2;
    return (bi && bj && !(g.pi && g.pj)) || (bi && bk && !(g.pi && g.pk)) || (bj && bk && !(g.pj && g.pk));
}
// 8 threads per cell of the 12 domain edges
inline int edge_threads(const Grid &g) { return 8 * 4 * (g.mx + g.my + g.mz - 6); }

// The budget of an edge cell, a thread per face and the sum by shuffles: one
// thread for all six faces is a chain of some 400 dependent accesses, 110 us at
// any grid size
__device__ void fp_edge_cell(const Grid &g, const Tensor &t, const State &s, const V3f<double> &fp, const Params &p, int e8)
{
    const int mx = g.mx, my = g.my, mz = g.mz;
    const int q = e8 & 7, d = q >> 1, lo = q & 1;
    int e = e8 >> 3, i = 1, j = 1, k = 1;
    bool on = q < 6;
    if (e < 4 * (mz - 2)) { k = 1 + (e >> 2); i = (e & 1) ? mx - 2 : 1; j = (e & 2) ? my - 2 : 1; }
    else if ((e -= 4 * (mz - 2)) < 4 * (my - 2)) { j = 1 + (e >> 2); i = (e & 1) ? mx - 2 : 1; k = (e & 2) ? mz - 2 : 1; }
    else if ((e -= 4 * (my - 2)) < 4 * (mx - 2)) { i = 1 + (e >> 2); j = (e & 1) ? my - 2 : 1; k = (e & 2) ? mz - 2 : 1; }
    else on = false;
    on = on && edge_cell(g, k, j, i);
    double F[3] = {0.0, 0.0, 0.0};          // by direction
    if (on) {
        const StageField f{g, t, s, p};
        // cells c and n of the face; a periodic face 0 is the face m-2
        int ck = k - (d == 2 && lo), cj = j - (d == 1 && lo), ci = i - (d == 0 && lo);
        if (ci == 0 && g.pi) ci = mx - 2;
        if (cj == 0 && g.pj) cj = my - 2;
        if (ck == 0 && g.pk) ck = mz - 2;
        const int nk = ck + (d == 2), nj = cj + (d == 1), ni = ci + (d == 0);
        const int l = d == 0 ? ci : d == 1 ? cj : ck, m = d == 0 ? mx : d == 1 ? my : mz;
        const bool edge = l == 0 || l == m - 2, npd = !(d == 0 ? g.pi : d == 1 ? g.pj : g.pk);
        double a[3], b[3];
        #pragma unroll
        for (int c = 0; c < 3; c++) { a[c] = f.u(c, ck, cj, ci); b[c] = f.u(c, nk, nj, ni); }
        const double h = -0.5 * f.v(d, ck, cj, ci);
        double n = p.les ? p.nu + 0.5 * (f.nu(ck, cj, ci) + f.nu(nk, nj, ni)) : p.nu;
        double tau[3] = {0.0, 0.0, 0.0};
        if (p.les && edge) {
            const int patch = 2 * d + (l != 0);
            if (d == 1 && p.bc[patch] == TG_BC_WALL_SHUMANN) {
                const int w = k * mx + i;
                tau[0] = s.twy[w]; tau[1] = s.twz[w]; tau[2] = s.twx[w];
                n = p.nu;
            } else if (p.bc[patch] == TG_BC_SLIP) n = 0.0;
        }
        const double size[3] = {t.dy[i], t.dz[j], t.dx[k]};
        const double rf = d == 0 ? t.rdyf[l] : d == 1 ? t.rdzf[l] : t.rdxf[l];
        const double area = size[d == 0 ? 1 : 0] * size[d == 2 ? 1 : 2], w = n * (area * rf);
        #pragma unroll
        for (int c = 0; c < 3; c++) {
            // viscous part of component c: w times its difference, and the
            // derivative along c of the face-normal component with the size of
            // the third direction as weight
            double x;
            if (c == d) x = w * (b[c] - a[c]);
            else {
                const int at = c == 0 ? i : c == 1 ? j : k, mc = c == 0 ? mx : c == 1 ? my : mz;
                const bool one = edge && (npd || !(c == 0 ? g.pi : c == 1 ? g.pj : g.pk));
                const int o1 = (one && at == mc - 2) ? 0 : 1, o0 = (one && at == 1 && at != mc - 2) ? 0 : -1;
                auto sum = [&](int o) {
                    return f.u(d, ck + (c == 2 ? o : 0), cj + (c == 1 ? o : 0), ci + (c == 0 ? o : 0)) +
                           f.u(d, nk + (c == 2 ? o : 0), nj + (c == 1 ? o : 0), ni + (c == 0 ? o : 0));
                };
                x = n * size[3 - c - d] * ((o1 - o0 == 1 ? 0.5 : 0.25) * (sum(o1) - sum(o0)));
            }
            F[c] = h * (a[c] + b[c]) + w * (b[c] - a[c]) + x - tau[c];
            if (lo) F[c] = -F[c];
        }
    }
    #pragma unroll
    for (int o = 4; o > 0; o >>= 1)
        #pragma unroll
        for (int c = 0; c < 3; c++) F[c] += __shfl_xor_sync(0xffffffffu, F[c], o, 8);
    if (on && q == 0) st3(fp, g.lin(k, j, i), R3<double>{F[2], F[0], F[1]});
}

// shared memory of k_stage_fp, in doubles: per plane of the Ucont ring X (35 x 10),
// Y (34 x 11), Z and nut (34 x 10); per plane of the Ucat ring three of 34 x 10
constexpr int SXW = PX + 3, SXN = SXW * PTY, SYN = PTX * (PTY + 1), SZN = PTX * PTY;
constexpr int OY = SXN, OZ = SXN + SYN, ON = OZ + SZN, SPL = ON + SZN, SUN = 3 * SZN;
constexpr int STAGE_SMEM = (4 * SPL + 4 * SUN + PTX + PTY + 2) * 8;

template <bool LES>
__global__ void __launch_bounds__(PX * PY, 2) k_stage_fp(const __grid_constant__ Grid g, const __grid_constant__ Tensor t, const __grid_constant__ State s,
                                                          V3f<double> fp, const __grid_constant__ Params p, int nedge, int nbi, int nbj, int kc)
{
    if ((int)blockIdx.x < nedge) { fp_edge_cell(g, t, s, fp, p, blockIdx.x * (PX * PY) + threadIdx.y * PX + threadIdx.x); return; }
    extern __shared__ double sh[];
    double *const raw = sh, *const uc = sh + 4 * SPL, *const sry = uc + 4 * SUN, *const srz = sry + PTX;
    const int mx = g.mx, my = g.my, mz = g.mz, pl = mx * my;
    const int blk = blockIdx.x - nedge, br = blk / nbi;
    const int i0 = 1 + (blk % nbi) * PX, j0 = 1 + (br % nbj) * PY, k0 = 1 + (br / nbj) * kc, k1 = min(k0 + kc - 1, mz - 2);
    const int tid = threadIdx.y * PX + threadIdx.x;
    // ---- what this thread copies of every plane: in-plane offsets of elements
    // tid and tid + 256 of each array. Elements outside the domain are never
    // used; they read the plane's first element.
    int dX[2], dY[2], dN[2];
    bool ghost[2];                 // a ghost of a non-periodic direction (or outside)
    auto inr = [](int l, int a, int b) { return l >= a && l <= b; };
    #pragma unroll
    for (int q = 0; q < 2; q++) {
        const int e = tid + q * (PX * PY);
        {
            const int j = wrap1(j0 - 1 + e / SXW, my, g.pj), f = wrap1(i0 - 2 + e % SXW, mx, g.pi);
            dX[q] = inr(j, 0, my - 1) && inr(f, 0, mx - 1) ? j * mx + f : 0;
        }
        {
            const int f = wrap1(j0 - 2 + e / PTX, my, g.pj), i = wrap1(i0 - 1 + e % PTX, mx, g.pi);
            dY[q] = inr(f, 0, my - 1) && inr(i, 0, mx - 1) ? f * mx + i : 0;
        }
        const int j = wrap1(j0 - 1 + e / PTX, my, g.pj), i = wrap1(i0 - 1 + e % PTX, mx, g.pi);
        dN[q] = inr(j, 0, my - 1) && inr(i, 0, mx - 1) ? j * mx + i : 0;
        ghost[q] = !(inr(j, 1, my - 2) && inr(i, 1, mx - 2));
    }
    if (tid < PTX) { const int i = wrap1(i0 - 1 + tid, mx, g.pi); sry[tid] = i <= mx - 1 ? t.rdy[i] : 0.0; }
    if (tid < PTY) { const int j = wrap1(j0 - 1 + tid, my, g.pj); srz[tid] = j <= my - 1 ? t.rdz[j] : 0.0; }
    // plane q of Ucont and nut into a slot of the ring
    auto load = [&](int q, double *d) {
        const int w = wrap1(q, mz, g.pk);
        if (w < 0 || w > mz - 1) return;
        const int o = w * pl;
        d += tid;
        cp_async8(d, s.ucont.x + o + dX[0]);
        cp_async8(d + OY, s.ucont.y + o + dY[0]);
        cp_async8(d + OZ, s.ucont.z + o + dN[0]);
        if (LES) cp_async8(d + ON, s.nut + o + dN[0]);
        d += PX * PY;
        if (tid < SYN - PX * PY) {
            cp_async8(d + OY, s.ucont.y + o + dY[1]);
            if (tid < SXN - PX * PY) cp_async8(d, s.ucont.x + o + dX[1]);
            if (tid < SZN - PX * PY) {
                cp_async8(d + OZ, s.ucont.z + o + dN[1]);
                if (LES) cp_async8(d + ON, s.nut + o + dN[1]);
            }
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    // Ucat of plane q from its Ucont d and the k faces of the plane below, zb
    auto convert = [&](int q, double rx, const double *d, const double *zb, double *u) {
        const int w = wrap1(q, mz, g.pk);
        if (w > mz - 1) return;
        const bool zghost = w < 1 || w > mz - 2;
        #pragma unroll
        for (int e2 = 0; e2 < 2; e2++) {
            const int e = tid + e2 * (PX * PY);
            if (e2 && tid >= SZN - PX * PY) break;
            if (zghost || ghost[e2]) {
                const int o = w * pl + dN[e2];
                u[e] = s.ucat.x[o]; u[SZN + e] = s.ucat.y[o]; u[2 * SZN + e] = s.ucat.z[o];
                continue;
            }
            const int r = e / PTX, c = e - r * PTX;
            const double ry = sry[c], rz = srz[r];
            const double *x = d + r * SXW + c, *y = d + OY + e;
            u[e] = (0.5 * (zb[OZ + e] + d[OZ + e])) * (ry * rz);
            u[SZN + e] = (0.5 * (x[0] + x[1])) * (rx * rz);
            u[2 * SZN + e] = (0.5 * (y[0] + y[PTX])) * (rx * ry);
        }
    };
    auto rdx = [&](int q) { return t.rdx[min(wrap1(q, mz, g.pk), mz - 1)]; };
    // planes k0-2 .. k0+1 in slots 0 .. 3; Ucat of k0-1, k0 and k0+1 in slots 1, 2, 3
    #pragma unroll
    for (int q = 0; q < 4; q++) load(k0 - 2 + q, raw + q * SPL);
    commit();
    cp_async_wait_all();
    __syncthreads();
    #pragma unroll
    for (int q = 1; q < 4; q++) convert(k0 - 2 + q, rdx(k0 - 2 + q), raw + q * SPL, raw + (q - 1) * SPL, uc + q * SUN);
    __syncthreads();
    const int i = i0 + threadIdx.x, j = j0 + threadIdx.y;
    const bool on = i <= mx - 2 && j <= my - 2;
    const double nu = p.nu, dy = on ? t.dy[i] : 0.0, dz = on ? t.dz[j] : 0.0, qdz = 0.25 * dz, qdy = 0.25 * dy, dydz = dy * dz;
    const double ryE = on ? t.rdyf[i] : 0.0, ryW = on ? t.rdyf[(i == 1 && g.pi) ? mx - 2 : i - 1] : 0.0;
    const double rzN = on ? t.rdzf[j] : 0.0, rzS = on ? t.rdzf[(j == 1 && g.pj) ? my - 2 : j - 1] : 0.0;
    // slip patches carry no viscous flux (with LES), the wall function's the wall stress
    const bool offW = LES && i == 1 && p.bc[TG_ILEFT] == TG_BC_SLIP, offE = LES && i == mx - 2 && p.bc[TG_IRIGHT] == TG_BC_SLIP;
    const bool offS = LES && j == 1 && p.bc[TG_JLEFT] == TG_BC_SLIP, offN = LES && j == my - 2 && p.bc[TG_JRIGHT] == TG_BC_SLIP;
    const bool wmS = LES && j == 1 && p.bc[TG_JLEFT] == TG_BC_WALL_SHUMANN, wmN = LES && j == my - 2 && p.bc[TG_JRIGHT] == TG_BC_WALL_SHUMANN;
    // edge_cell by parts: along this column, and at the first and last plane
    const bool bi = i == 1 || i == mx - 2, bj = j == 1 || j == my - 2;
    const bool edge = bi && bj && !(g.pi && g.pj), kedge = edge || (bi && !(g.pi && g.pk)) || (bj && !(g.pj && g.pk));
    const int a = (threadIdx.y + 1) * PTX + threadIdx.x + 1, ax = (threadIdx.y + 1) * SXW + threadIdx.x + 1;
    auto kface = [&](const double *lo, const double *hi, double n, double z, double K1) {
        const double x0 = lo[a], x1 = hi[a], y0 = lo[SZN + a], y1 = hi[SZN + a], z0 = lo[2 * SZN + a], z1 = hi[2 * SZN + a];
        const double h = -0.5 * z, w = n * K1;
        const double uy = (hi[a + 1] + lo[a + 1]) - (hi[a - 1] + lo[a - 1]), uz = (hi[a + PTX] + lo[a + PTX]) - (hi[a - PTX] + lo[a - PTX]);
        R3<double> f;
        f.x = h * (x0 + x1) + (2.0 * w) * (x1 - x0);
        f.y = h * (y0 + y1) + w * (y1 - y0) + (n * qdz) * uy;
        f.z = h * (z0 + z1) + w * (z1 - z0) + (n * qdy) * uz;
        return f;
    };
    R3<double> bot{0.0, 0.0, 0.0};
    if (on) {
        const double *rl = raw + SPL, *rh = raw + 2 * SPL;
        double n = LES ? nu + 0.5 * (rl[ON + a] + rh[ON + a]) : nu;
        if (LES && k0 == 1 && p.bc[TG_KLEFT] == TG_BC_SLIP) n = 0.0;
        bot = kface(uc + SUN, uc + 2 * SUN, n, rl[OZ + a], dydz * t.rdxf[(k0 == 1 && g.pk) ? mz - 2 : k0 - 1]);
    }
    __syncthreads();
    load(k0 + 2, raw);
    commit();
    // Plane k = k0 + t is in slots (t + 2) & 3; four planes per trip so that every
    // slot is a constant offset. One barrier per plane: Ucat of plane k+2 and the
    // copy of plane k+3 go to slots that plane k does not read.
    for (int kb = k0; kb <= k1; kb += 4) {
        #pragma unroll
        for (int ph = 0; ph < 4; ph++) {
            const int k = kb + ph;
            if (k > k1) break;
            const double dx = t.dx[k], rxf = t.rdxf[k], rx2 = rdx(k + 2);
            cp_async_wait_all();                                     // plane k+2 is there
            __syncthreads();
            if (k < k1) {
                convert(k + 2, rx2, raw + (ph & 3) * SPL, raw + ((ph + 3) & 3) * SPL, uc + (ph & 3) * SUN);
                if (k < k1 - 1) load(k + 3, raw + ((ph + 1) & 3) * SPL);
                commit();
            }
            if (!on) continue;
            const double *um = uc + ((ph + 1) & 3) * SUN, *u0 = uc + ((ph + 2) & 3) * SUN, *up = uc + ((ph + 3) & 3) * SUN;
            const double *r0 = raw + ((ph + 2) & 3) * SPL, *rp = raw + ((ph + 3) & 3) * SPL;
            const double *N = r0 + ON;
            const double qdx = 0.25 * dx, dxdz = dx * dz, dxdy = dx * dy;
            const double nc = LES ? N[a] : 0.0;
            double nt = LES ? nu + 0.5 * (nc + rp[ON + a]) : nu;
            if (LES && k == mz - 2 && p.bc[TG_KRIGHT] == TG_BC_SLIP) nt = 0.0;
            const R3<double> top = kface(u0, up, nt, r0[OZ + a], dydz * rxf);
            R3<double> f = top - bot;
            bot = top;
            const double *U0 = u0, *U1 = u0 + SZN, *U2 = u0 + 2 * SZN;
            // i face between tile points b and b + 1 (sg: + for the cell's + side)
            auto iface = [&](int b, double x, double n, double I1, double sg) {
                const int e = b + 1;
                const double x0 = U0[b], x1 = U0[e], y0 = U1[b], y1 = U1[e], z0 = U2[b], z1 = U2[e];
                const double h = -0.5 * x, w = n * I1;
                const double vx = (up[SZN + e] + up[SZN + b]) - (um[SZN + e] + um[SZN + b]), vz = (U1[e + PTX] + U1[b + PTX]) - (U1[e - PTX] + U1[b - PTX]);
                f.x += sg * (h * (x0 + x1) + w * (x1 - x0) + (n * qdz) * vx);
                f.y += sg * (h * (y0 + y1) + (2.0 * w) * (y1 - y0));
                f.z += sg * (h * (z0 + z1) + w * (z1 - z0) + (n * qdx) * vz);
            };
            auto jface = [&](int b, double y, double n, double J1, double sg) {
                const int e = b + PTX;
                const double x0 = U0[b], x1 = U0[e], y0 = U1[b], y1 = U1[e], z0 = U2[b], z1 = U2[e];
                const double h = -0.5 * y, w = n * J1;
                const double wx = (up[2 * SZN + e] + up[2 * SZN + b]) - (um[2 * SZN + e] + um[2 * SZN + b]), wy = (U2[e + 1] + U2[b + 1]) - (U2[e - 1] + U2[b - 1]);
                f.x += sg * (h * (x0 + x1) + w * (x1 - x0) + (n * qdy) * wx);
                f.y += sg * (h * (y0 + y1) + w * (y1 - y0) + (n * qdx) * wy);
                f.z += sg * (h * (z0 + z1) + (2.0 * w) * (z1 - z0));
            };
            const double *X = r0 + ax, *Y = r0 + OY + a;
            iface(a, X[1], offE ? 0.0 : LES ? nu + 0.5 * (nc + N[a + 1]) : nu, dxdz * ryE, 1.0);
            iface(a - 1, X[0], offW ? 0.0 : LES ? nu + 0.5 * (nc + N[a - 1]) : nu, dxdz * ryW, -1.0);
            jface(a, Y[PTX], offN ? 0.0 : wmN ? nu : LES ? nu + 0.5 * (nc + N[a + PTX]) : nu, dxdy * rzN, 1.0);
            jface(a - PTX, Y[0], offS ? 0.0 : wmS ? nu : LES ? nu + 0.5 * (nc + N[a - PTX]) : nu, dxdy * rzS, -1.0);
            if (wmS || wmN) {
                const int w = k * mx + i;
                const double sg = (wmS ? 1.0 : 0.0) - (wmN ? 1.0 : 0.0);
                f.x += sg * s.twx[w]; f.y += sg * s.twy[w]; f.z += sg * s.twz[w];
            }
            if (!((k == 1 || k == mz - 2) ? kedge : edge)) st3(fp, (k * my + j) * mx + i, f);
        }
    }
}

// Ucont and the ghosts of Ucat as SolveUEqn's tail leaves them (ueqn.c:413-437)
// after stages that read both through the index rules above: the no-penetration
// and periodic face resets on the boundary planes, and the periodic copies of
// Ucat into its ghost points (edges and corners included; the face ghosts and
// every interior cell are rewritten at the end of the step). One thread per
// point of the six boundary planes of the DMDA box.
__global__ void __launch_bounds__(256) k_stage_tail(const __grid_constant__ Grid g, const __grid_constant__ Tensor t, const __grid_constant__ State s,
                                                   const __grid_constant__ Params p)
{
    const int patch = blockIdx.z, dir = patch >> 1, right = patch & 1;
    const int a = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y * blockDim.y + threadIdx.y;
    int i, j, k;
    if (dir == 0) { if (a >= g.my || b >= g.mz) return; i = right ? g.mx - 1 : 0; j = a; k = b; }
    else if (dir == 1) { if (a >= g.mx - 2 || b >= g.mz) return; j = right ? g.my - 1 : 0; i = a + 1; k = b; }
    else { if (a >= g.mx - 2 || b >= g.my - 2) return; k = right ? g.mz - 1 : 0; i = a + 1; j = b + 1; }
    const int c = g.lin(k, j, i);
    // faces: plane 0 of a periodic direction takes plane m-2; then walls. Points
    // of the boundary planes themselves hold Ucont_o (their right-hand side is
    // zero), which no stage changed.
    const int fi = (i == 0 && g.pi) ? g.mx - 2 : i, fj = (j == 0 && g.pj) ? g.my - 2 : j, fk = (k == 0 && g.pk) ? g.mz - 2 : k;
    const int q = g.lin(fk, fj, fi);
    const bool shell = fi == 0 || fi == g.mx - 1 || fj == 0 || fj == g.my - 1 || fk == 0 || fk == g.mz - 1;
    const V3f<double> &u = shell ? s.ucont_o : s.ucont;
    auto wall = [&](int d, int l, int m, bool in) { return in && ((l == 0 && wall_patch(p, 2 * d)) || (l == m - 2 && wall_patch(p, 2 * d + 1))); };
    const bool ri = fi <= g.mx - 2, rj = fj <= g.my - 2, rk = fk <= g.mz - 2;
    const R3<double> v{wall(0, fi, g.mx, rj && rk) ? 0.0 : u.x[q], wall(1, fj, g.my, ri && rk) ? 0.0 : u.y[q], wall(2, fk, g.mz, ri && rj) ? 0.0 : u.z[q]};
    st3(s.ucont, c, v);
    // the wall face m-2 below a right boundary plane (zero for every reader above)
    if (right && wall_patch(p, patch)) {
        if (dir == 0 && j <= g.my - 2 && k <= g.mz - 2) s.ucont.x[c - 1] = 0.0;
        if (dir == 1 && k <= g.mz - 2) s.ucont.y[c - g.mx] = 0.0;
        if (dir == 2) s.ucont.z[c - g.mx * g.my] = 0.0;
    }
    // Ucat: ghosts of periodic directions
    const int ui = wrap1(i, g.mx, g.pi), uj = wrap1(j, g.my, g.pj), uk = wrap1(k, g.mz, g.pk);
    if (ui == i && uj == j && uk == k) return;
    const StageField f{g, t, s, p};
    st3(s.ucat, c, R3<double>{f.u(2, uk, uj, ui), f.u(0, uk, uj, ui), f.u(1, uk, uj, ui)});
}

// ----------------------------------------------------------- face assembly
// k_rhs_faces (ueqn_solvers.c:1008-1035 and the sources of ExplicitRhsU): the
// face value scale * aj_face * central(S . fp) needs one component of fp at
// the two cells of the face, weighted by the inverse distance across it.
// kind as there: 0 R += scale FormU; 1 ExplicitRhsU stored in R; 2 masked at
// the non-resolved faces and applied by the explicit update. from_p: dP is
// formed again from p (the same products; a stage of a step, where dP is that of
// p), one value and its neighbours instead of three: a step of 256 x 256 x 128
// 3.125 -> 3.098 ms, of 192 x 128 x 64 0.825 -> 0.818 ms.
template <int kind, bool from_p>
__global__ void __launch_bounds__(256, 8) k_rhs_tensor(Grid g, Tensor t, State s, V3f<double> fp, V3f<double> R, double scale, Params p, int ab2, RkArgs rk)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1, k = blockIdx.z * blockDim.z + threadIdx.z + 1;
    if (i > g.mx - 2 || j > g.my - 2 || k > g.mz - 2) return;
    const int c = g.lin(k, j, i), pl = g.mx * g.my;
    R3<double> o;
    if (kind == 0) {
        o = ld3(R, c);
    } else {
        const R3<double> dp = from_p ? grad_p_cell(g, t, s.p, k, j, i, c) : ld3(s.dp, c);
        o = R3<double>{0.0 - dp.x, 0.0 - dp.y, 0.0 - dp.z};
        if (p.buoyancy) {
            const R3<double> b = ld3(s.btheta, c);
            if (ab2) { o = o + (3.0 / 2.0) * b; o = o + (-1.0 / 2.0) * ld3(s.btheta_o, c); }
            else o = o + b;
        }
        if (p.farm) o = o + ld3(s.farmcont, c);
    }
    // the neighbour beyond the last interior cell: the opposite first cell
    // (periodic) or a copy of this one (ueqn_solvers.c:949-990)
    const int ie = i < g.mx - 2 ? c + 1 : (g.pi ? g.lin(k, j, 1) : c);
    const int jn = j < g.my - 2 ? c + g.mx : (g.pj ? g.lin(k, 1, i) : c);
    const int kt = k < g.mz - 2 ? c + pl : (g.pk ? g.lin(1, j, i) : c);
    const double h = 0.5 * scale;
    o.x += (h * t.rdyf[i]) * (fp.y[c] + fp.y[ie]);
    o.y += (h * t.rdzf[j]) * (fp.z[c] + fp.z[jn]);
    o.z += (h * t.rdxf[k]) * (fp.x[c] + fp.x[kt]);
    if (kind >= 1 && (p.source || p.mean_grad_p)) {
        const double dx = t.dx[k], dy = t.dy[i], dz = t.dz[j];
        if (p.source) {
            // sourceU (ueqn_solvers.c:1369, ueqn_sources.c:2884-2980)
            const V3f<double> &f = s.source;
            o.x += 0.5 * (f.y[c] + f.y[c + 1]) * (dx * dz);
            o.y += 0.5 * (f.z[c] + f.z[c + g.mx]) * (dx * dy);
            o.z += 0.5 * (f.x[c] + f.x[c + pl]) * (dy * dz);
        }
        if (p.mean_grad_p) {
            o.x += p.mgp[1] * (dx * dz);
            o.y += p.mgp[2] * (dx * dy);
            o.z += p.mgp[0] * (dy * dz);
        }
    }
    if (kind == 2) {
        mask_last_faces(g, s, p, k, j, i, c, o);
        rk_point(s.ucont.x + c, s.utmp.x + c, s.ucont_o.x + c, o.x, rk);
        rk_point(s.ucont.y + c, s.utmp.y + c, s.ucont_o.y + c, o.y, rk);
        rk_point(s.ucont.z + c, s.utmp.z + c, s.ucont_o.z + c, o.z, rk);
        // resetNoPenetrationFluxes, which follows every stage
        if (i == g.mx - 2 && wall_patch(p, TG_IRIGHT)) s.ucont.x[c] = 0.0;
        if (j == g.my - 2 && wall_patch(p, TG_JRIGHT)) s.ucont.y[c] = 0.0;
        if (k == g.mz - 2 && wall_patch(p, TG_KRIGHT)) s.ucont.z[c] = 0.0;
    } else {
        st3(R, c, o);
    }
}

// ------------------------------------ pressure update and ProjectVelocity
// From the compact Poisson solution x in one pass: phi and p with their ghosts
// (phiToPhi, UpdatePressure, UpdatePhiBCs, UpdatePressureBCs; peqn.c:1579-1636,
// 2909-2962, boundary.c:3051-3255), the gauge p -= *ref if ref is given
// (SyncPressureAcrossDomains, overset.c:263-315), and the projection of the faces
// (peqn.c:2495-2905). A cell writes its own value to the ghost points that copy
// it, so no point is read after another thread wrote it. 80 bytes per cell; the
// separate passes (two conversions, six ghost launches, update, projection,
// gauge) took 0.30 ms at 256 x 256 x 128.
__global__ void __launch_bounds__(256) k_pressure_project(Grid g, Tensor t, State s, const double *x, const double *ref, double dt)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1, k = blockIdx.z * blockDim.z + threadIdx.z + 1;
    const int mx = g.mx, my = g.my, mz = g.mz;
    if (i > mx - 2 || j > my - 2 || k > mz - 2) return;
    const int nx = mx - 2, ny = my - 2, nz = mz - 2, pl = mx * my, cpl = nx * ny;
    const int c = g.lin(k, j, i), cc = (k - 1) * cpl + (j - 1) * nx + i - 1;
    const double phi = x[cc], dx = t.dx[k], dy = t.dy[i], dz = t.dz[j];
    double p = s.p[c] + phi;
    if (ref) p -= ref[0];
    const double fi = dx * dz, fj = dx * dy, fk = dy * dz;
    if (i < mx - 2 || g.pi) s.ucont.x[c] -= ((x[i < mx - 2 ? cc + 1 : cc + 1 - nx] - phi) * (fi * t.rdyf[i])) * dt;
    if (j < my - 2 || g.pj) s.ucont.y[c] -= ((x[j < my - 2 ? cc + nx : cc + nx - cpl] - phi) * (fj * t.rdzf[j])) * dt;
    if (k < mz - 2 || g.pk) s.ucont.z[c] -= ((x[k < mz - 2 ? cc + cpl : cc + cpl - cpl * nz] - phi) * (fk * t.rdxf[k])) * dt;
    // face 0 of a periodic direction
    if (i == 1 && g.pi) s.ucont.x[c - 1] -= ((phi - x[cc + nx - 1]) * (fi * t.rdyf[0])) * dt;
    if (j == 1 && g.pj) s.ucont.y[c - mx] -= ((phi - x[cc + cpl - nx]) * (fj * t.rdzf[0])) * dt;
    if (k == 1 && g.pk) s.ucont.z[c - pl] -= ((phi - x[cc + cpl * nz - cpl]) * (fk * t.rdxf[0])) * dt;
    // the indices that copy this cell's: its own, and the ghost next to it or
    // (periodic) opposite
    auto image = [](int l, int m, int per) { return l == 1 ? (per ? m - 1 : 0) : l == m - 2 ? (per ? 0 : m - 1) : l; };
    const int gi_ = image(i, mx, g.pi), gj_ = image(j, my, g.pj), gk_ = image(k, mz, g.pk);
    s.phi[c] = phi;
    s.p[c] = p;
    if (gi_ == i && gj_ == j && gk_ == k) return;
    for (int b = 1; b < 8; b++) {
        if (((b & 1) && gi_ == i) || ((b & 2) && gj_ == j) || ((b & 4) && gk_ == k)) continue;
        const int q = g.lin((b & 4) ? gk_ : k, (b & 2) ? gj_ : j, (b & 1) ? gi_ : i);
        s.phi[q] = phi;
        s.p[q] = p;
    }
}

// contravariantToCartesian of the projected Ucont with the divergence maximum of
// ContinuityErrorsOptimized (peqn.c:4114-4181), block partials: both read the six
// faces of a cell
__global__ void __launch_bounds__(256) k_contra_div_tensor(Grid g, Tensor t, State s, double *part)
{
    const int lane = threadIdx.x & 31, nJ = g.my - 2, nrow = nJ * (g.mz - 2), pl = g.mx * g.my;
    double v[1] = {0.0};
    for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < nrow; row += (gridDim.x * blockDim.x) >> 5) {
        const int j = row % nJ + 1, k = row / nJ + 1;
        const double rx = t.rdx[k], rz = t.rdz[j], rxz = rx * rz;
        for (int i = 1 + lane; i <= g.mx - 2; i += 32) {
            const int c = g.lin(k, j, i);
            const double ry = t.rdy[i];
            const double x1 = s.ucont.x[c], x0 = s.ucont.x[c - 1], y1 = s.ucont.y[c], y0 = s.ucont.y[c - g.mx], z1 = s.ucont.z[c], z0 = s.ucont.z[c - pl];
            s.ucat.x[c] = (0.5 * (z0 + z1)) * (ry * rz);
            s.ucat.y[c] = (0.5 * (x0 + x1)) * rxz;
            s.ucat.z[c] = (0.5 * (y0 + y1)) * (rx * ry);
            v[0] = nanmax(v[0], fabs((x1 - x0 + y1 - y0 + z1 - z0) * (rxz * ry)));
        }
    }
    block_reduce<256>(v, RedNanMax{});
    if (threadIdx.x == 0) part[blockIdx.x] = v[0];
}

inline dim3 gi(const Grid &g) { return grid3(g.mx - 2, g.my - 2, g.mz - 2); }

template <int mode, bool LES, int KZ>
void launch_fp(tg_ctx *C, const Box &b)
{
    constexpr int bytes = PTX * PTY * (KZ + 2) * 8 * (LES && mode != 1 ? 4 : 3);
    static_assert(bytes <= 110 * 1024, "two blocks per SM, as the registers allow");
    const int nbi = (b.i1 - b.i0 + PX) / PX, nbj = (b.j1 - b.j0 + PY) / PY, nbk = (b.k1 - b.k0 + KZ) / KZ, nbnd = boundary_blocks(C->g);
    TG_PROF(C, "formu_cell_fp", (k_fp_tensor<mode, LES, KZ><<<nbnd + nbi * nbj * nbk, dim3(PX, PY), bytes, C->stream>>>(C->g, C->ts, C->s, C->fw.fp, C->prm, b, nbnd, nbi, nbj)));
}

template <int mode>
void form_fp(tg_ctx *C)
{
    const Grid g = C->g;
    const Box b{2, g.pi ? g.mx - 2 : g.mx - 3, 2, g.pj ? g.my - 2 : g.my - 3, 2, g.pk ? g.mz - 2 : g.mz - 3};
    // four cells per thread share most of a tile; two where that would leave
    // SMs without a block
    const int64_t cols = (int64_t)((b.i1 - b.i0 + PX) / PX) * ((b.j1 - b.j0 + PY) / PY);
    const bool deep = cols * ((b.k1 - b.k0 + 4) / 4) >= 148 * 3;
    if (C->prm.les) { if (deep) launch_fp<mode, true, 4>(C, b); else launch_fp<mode, true, 2>(C, b); }
    else { if (deep) launch_fp<mode, false, 4>(C, b); else launch_fp<mode, false, 2>(C, b); }
}

template <bool LES>
void launch_stage_fp(tg_ctx *C)
{
    const Grid g = C->g;
    const int nbi = (g.mx - 2 + PX - 1) / PX, nbj = (g.my - 2 + PY - 1) / PY, nk = g.mz - 2;
    // planes per block: every chunk costs about three planes of start-up, every
    // started wave of two blocks per SM a chunk
    int kc = nk;
    int64_t best = INT64_MAX;
    for (int ch = 1; ch <= std::max(1, nk / 4); ch++) {
        const int c = (nk + ch - 1) / ch;
        const int64_t waves = ((int64_t)nbi * nbj * ((nk + c - 1) / c) + 2 * 148 - 1) / (2 * 148), cost = waves * (c + 3);
        if (cost < best) { best = cost; kc = c; }
    }
    const int nedge = (edge_threads(g) + PX * PY - 1) / (PX * PY), nb = nedge + nbi * nbj * ((nk + kc - 1) / kc);
    TG_PROF(C, "formu_stage_fp", (k_stage_fp<LES><<<nb, dim3(PX, PY), STAGE_SMEM, C->stream>>>(g, C->ts, C->s, C->fw.fp, C->prm, nedge, nbi, nbj, kc)));
}

template <int mode, bool LES, int KZ>
void set_fp_attr()
{
    constexpr int bytes = PTX * PTY * (KZ + 2) * 8 * (LES && mode != 1 ? 4 : 3);
    TG_CUDA(cudaFuncSetAttribute((const void *)k_fp_tensor<mode, LES, KZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}
template <int mode>
void set_fp_attrs()
{
    set_fp_attr<mode, true, 4>(); set_fp_attr<mode, true, 2>(); set_fp_attr<mode, false, 4>(); set_fp_attr<mode, false, 2>();
}

}  // namespace

namespace {
constexpr double EPS = 2.220446049250313e-16;
// coordinates of the planes 0 .. m-2 of direction q (x, y, z) through the first node
std::vector<double> plane_line(const Grid &g, const double *nodes, int q)
{
    const int n = (q == 0 ? g.mz : q == 1 ? g.mx : g.my) - 1;
    const int64_t st = q == 0 ? (int64_t)g.mx * g.my : q == 1 ? 1 : g.mx;
    std::vector<double> X(n);
    for (int l = 0; l < n; l++) X[l] = nodes[3 * st * l + q];
    return X;
}
double largest(const std::vector<double> &X)
{
    double r = 0.0;
    for (double x : X) r = std::max(r, std::fabs(x));
    return r;
}
}  // namespace

// Is the mesh one of planes (x depends on k alone, y on i, z on j)? The question is
// put to the nodes and not to the metrics: those form the same size by sums of
// different nodes and differ from each other by some units of rounding of the
// coordinates over the spacing (2e-13 at 1300 cells of 7.3 m, 1.4e-11 at map
// coordinates of 500 km), which says nothing about the planes. A node may be off
// its plane by four units of rounding of the largest coordinate.
bool planes_of_nodes(const Grid &g, const double *nodes)
{
    const std::vector<double> X = plane_line(g, nodes, 0), Y = plane_line(g, nodes, 1), Z = plane_line(g, nodes, 2);
    const double ox = 4 * EPS * largest(X), oy = 4 * EPS * largest(Y), oz = 4 * EPS * largest(Z);
    for (int k = 0; k < g.mz - 1; k++)
        for (int j = 0; j < g.my - 1; j++) {
            const double *x = nodes + 3 * (int64_t)g.lin(k, j, 0);
            bool on = true;
            for (int i = 0; i < g.mx - 1; i++, x += 3)
                on = on && std::fabs(x[0] - X[k]) <= ox && std::fabs(x[1] - Y[i]) <= oy && std::fabs(x[2] - Z[j]) <= oz;
            if (!on) return false;
        }
    return true;
}

// The spacings of a mesh of planes from its nodes, into C->ts. planes: as
// planes_of_nodes; without it the caller found the cross components of the metrics
// to vanish to 1e-12, and every metric has to be its product to 1e-12. false if
// the metrics are not these products.
bool tensor_setup(tg_ctx *C, const double *nodes, bool planes)
{
    const Grid g = C->g;
    cudaStream_t st = C->stream;
    const int n[3] = {g.mz, g.mx, g.my};                       // x, y, z
    const int per[3] = {g.pk, g.pi, g.pj};
    std::vector<double> X[3];                                  // planes 0 .. n-2
    double round = 0.0;
    for (int q = 0; q < 3; q++) {
        X[q] = plane_line(g, nodes, q);
        double h = HUGE_VAL;
        for (int l = 1; l < n[q] - 1; l++) h = std::min(h, std::fabs(X[q][l] - X[q][l - 1]));
        round += EPS * largest(X[q]) / h;
    }
    if (!std::isfinite(round)) return false;                   // coinciding planes
    constexpr int NA = 7;        // arrays per direction
    if (!C->ts_mem) C->ts_mem = dallocd(C, NA * ((size_t)g.mx + g.my + g.mz));
    double *mem = C->ts_mem;
    Tensor &t = C->ts;
    const double **d[3][NA] = {{&t.dx, &t.rdx, &t.dxf, &t.rdxf, &t.qx, &t.rqx, &t.rqxf},
                               {&t.dy, &t.rdy, &t.dyf, &t.rdyf, &t.qy, &t.rqy, &t.rqyf},
                               {&t.dz, &t.rdz, &t.dzf, &t.rdzf, &t.qz, &t.rqz, &t.rqzf}};
    for (int q = 0; q < 3; q++) {
        // cell sizes with those of the ghosts (mirrored, or the opposite cell's), and the
        // distances across the faces 0 .. m-2 as the face metrics take them
        // (mesh.c:1354-1930): half the distance of the planes on either side, one-sided at
        // an end, averaged over the seam at face m-2 of a periodic direction
        const int m = n[q];
        std::vector<double> h(NA * (size_t)m, 0.0);
        auto size = [&](int l) { return X[q][l] - X[q][l - 1]; };
        for (int l = 0; l < m; l++) {
            const double s = size(l == 0 ? (per[q] ? m - 2 : 1) : l == m - 1 ? (per[q] ? 1 : m - 2) : l);
            const double f = l == 0 ? size(1) : l < m - 2 ? 0.5 * (X[q][l + 1] - X[q][l - 1]) : per[q] ? 0.5 * (size(1) + size(m - 2)) : size(m - 2);
            h[l] = s; h[m + l] = 1.0 / s;
            if (l < m - 1) { h[2 * m + l] = f; h[3 * m + l] = 1.0 / f; }
            auto sq = [](double x) { return std::cbrt(x) * std::cbrt(x); };
            h[4 * m + l] = sq(h[l]);                            // (dx dy dz)^(2/3) by factors
            h[5 * m + l] = sq(h[m + l]);
            if (l < m - 1) h[6 * m + l] = sq(h[3 * m + l]);
        }
        TG_CUDA(cudaMemcpyAsync(mem, h.data(), sizeof(double) * h.size(), cudaMemcpyHostToDevice, st));
        TG_CUDA(cudaStreamSynchronize(st));
        for (int e = 0; e < NA; e++) *d[q][e] = mem + (size_t)e * m;
        mem += h.size();
    }
    // The metrics against their products. On planes this is a guard: a size by a sum of
    // eight nodes is off by up to 3.5 units of rounding over the spacing, by 8 more
    // if the nodes are off their planes by four on either side, and a product has the
    // directions' sum.
    k_tensor_check<<<C->red_blocks, 256, 0, st>>>(g, C->fm64, C->ts, C->d_red);
    std::vector<double> part(C->red_blocks);
    TG_CUDA(cudaMemcpyAsync(part.data(), C->d_red, sizeof(double) * part.size(), cudaMemcpyDeviceToHost, st));
    TG_CUDA(cudaStreamSynchronize(st));
    const double tol = planes ? std::max(1e-12, 12 * round) : 1e-12;
    bool ok = true;
    for (double v : part) ok = ok && v <= tol;
    if (ok) {
        set_fp_attrs<0>(); set_fp_attrs<1>(); set_fp_attrs<2>();
        TG_CUDA(cudaFuncSetAttribute((const void *)k_stage_fp<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, STAGE_SMEM));
        TG_CUDA(cudaFuncSetAttribute((const void *)k_stage_fp<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, STAGE_SMEM));
    }
    return ok;
}

void contra_to_cart_tensor(tg_ctx *C, const char *name)
{
    TG_PROF(C, name, k_contra_tensor<<<gi(C->g), block3(), 0, C->stream>>>(C->g, C->ts, C->s));
}
void smagorinsky_tensor(tg_ctx *C)
{
    TG_PROF(C, "smagorinsky", k_smagorinsky_tensor<<<gi(C->g), block3(), 0, C->stream>>>(C->g, C->ts, C->s, C->prm.cs));
}
void grad_p_tensor(tg_ctx *C)
{
    TG_PROF(C, "grad_p", k_grad_p_tensor<<<gi(C->g), block3(), 0, C->stream>>>(C->g, C->ts, C->s));
}
void form_fp_tensor(tg_ctx *C, int mode)
{
    if (mode == 1) form_fp<1>(C);
    else if (mode == 2) form_fp<2>(C);
    else form_fp<0>(C);
}
void stage_fp_tensor(tg_ctx *C)
{
    if (C->prm.les) launch_stage_fp<true>(C);
    else launch_stage_fp<false>(C);
}
void stage_tail_tensor(tg_ctx *C)
{
    const Grid g = C->g;
    const dim3 gr((std::max(g.mx, g.my) + 31) / 32, (std::max(g.my, g.mz) + 7) / 8, 6);
    TG_PROF(C, "stage_tail", k_stage_tail<<<gr, dim3(32, 8), 0, C->stream>>>(g, C->ts, C->s, C->prm));
}
void rhs_faces_tensor(tg_ctx *C, int kind, V3f<double> rhs, double scale, int ab2, const RkArgs &rk, bool from_p)
{
    const Grid g = C->g;
    const V3f<double> fp = C->fw.fp;
    auto go = [&](auto kernel) {
        TG_PROF(C, "formu_rhs_faces", kernel<<<gi(g), block3(), 0, C->stream>>>(g, C->ts, C->s, fp, rhs, scale, C->prm, ab2, rk));
    };
    if (kind == 0) go(k_rhs_tensor<0, false>);
    else if (kind == 1) go(k_rhs_tensor<1, false>);
    else if (from_p) go(k_rhs_tensor<2, true>);
    else go(k_rhs_tensor<2, false>);
}
void pressure_project_tensor(tg_ctx *C, const double *x, const double *ref)
{
    TG_PROF(C, "pressure_project", k_pressure_project<<<gi(C->g), block3(), 0, C->stream>>>(C->g, C->ts, C->s, x, ref, C->prm.dt));
}
void contra_div_tensor(tg_ctx *C)
{
    TG_PROF(C, "contra_div_final", k_contra_div_tensor<<<C->red_blocks, 256, 0, C->stream>>>(C->g, C->ts, C->s, C->d_red));
}

}  // namespace tg
