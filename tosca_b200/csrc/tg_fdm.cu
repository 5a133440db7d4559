// Direct solve of the 7-point pressure operator on a tensor-product mesh, the
// preconditioner of the CG pressure solve there.
//
// On a mesh of planes (not necessarily equidistant) the face coefficients
// separate,
//     aE = kx_i my_j mz_k,  aN = mx_i ky_j mz_k,  aT = mx_i my_j kz_k,
// so the operator is Kx(My)(Mz) + (Mx)Ky(Mz) + (Mx)(My)Kz with tridiagonal
// (cyclic where periodic) K and diagonal M. With the eigenvectors of the pencils
// (Kx, Mx) and (Kz, Mz) it decouples into one tridiagonal system along j per
// pair of modes (fast diagonalisation: Lynch, Rice and Thomas 1964):
//     z = (Phi_x Phi_z) T^-1 (Phi_x Phi_z)^T r.
// A periodic j is diagonalised as well. CG on the pinned operator with this
// preconditioner stops after one iteration (two at tolerances near rounding),
// against 2 to 5 with a multigrid V-cycle of some 60 launches.
//
// The transforms are dense products with the eigenvector matrix, not FFTs, so
// every size runs the same kernel: FP64 matrix instructions (mma.sync
// m8n8k4), a block per panel of columns held in shared memory and transformed
// in place. Equidistant directions use the trigonometric eigenvectors about
// the half-points i + 1/2, which are even or odd under i -> n-1-i; folding the
// panel halves the products (groups of modes), and a periodic direction with
// n a multiple of 4 folds twice. Work per cell and pass is 2 n / G operations
// for G groups. At 256 x 256 x 128 a pass takes 72 to 99 us against 21 us for its
// bytes and 29 us for its products at the 37 TFLOP/s that register-only
// m8n8k4 reaches (load, product and store phases of a block alternate; two or
// three blocks per SM overlap them in part), the j lines 58 us against 31 us for their bytes:
// 0.39 ms for the solve, against 1.06 ms for one multigrid V-cycle. Operands in
// fragment order (one 512-byte load per step) took a pass from 110 to 77 us.
#include <algorithm>
#include <cmath>
#include <vector>

#include "tg_fdm.cuh"

namespace tg {

// one transformed direction
struct FdmDir {
    int n = 0, G = 1;         // cells, groups of modes (1, 2 or 4)
    bool uni = false, per = false;   // equidistant, periodic
    int gs = 0, gp = 0;       // rows per group, rounded up to 8
    // eigenvectors, mode m of group g at fold row i, in the order of the matrix
    // instruction's fragments (frag_index): W with m as row, Wt with i as row
    double *W = nullptr, *Wt = nullptr;
    double *lam = nullptr;    // eigenvalues in storage order (group by group)
};

struct Fdm {
    int nx, ny, nz, pj;
    int64_t n;
    FdmDir x, y, z;           // y: periodic j only
    FdmOp op;
    double dev;               // largest relative deviation of the coefficients from the factors
    double *minv;             // 1 / pivots of the j-line systems, per mode pair
};

namespace {

// ------------------------------------------------------------- transforms
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d[0]), "+d"(d[1]) : "d"(a), "d"(b));
}

struct XformArgs {
    const double *src;
    double *dst;
    const double *A;          // W (forward) or Wt (inverse)
    int n, gs, gp;
    int64_t se;               // stride of the transformed direction
    int ncol;                 // columns of the grid
    int colw;                 // columns c, c+1 .. are adjacent within runs of colw
    int64_t colrun;           // stride between runs
    int64_t colst;            // stride within a run
    const double *d_sum;      // forward: entry 0 of src reads -d_sum[0]
    const double *lx, *ly, *lz;   // scaling of the j transform of a periodic j: 1 / (lx + ly + lz)
    int sx;                   // its run length (modes along i)
};

constexpr int XT = 256;       // threads per block
constexpr int XW = XT / 32;

// rows of a [column][row] panel, padded to 4 mod 16
__host__ __device__ constexpr int x_stride(int rows) { return ((rows + 15) / 16) * 16 + 4; }

// ROWC: the transformed direction is the contiguous one; the panel is kept
// [column][row], else [row][column]. The padded strides (4 mod 16 doubles) make
// the B fragment reads (4 rows x 8 columns) free of bank conflicts.
template <int G, bool INV, bool ROWC, int NC>
__global__ void __launch_bounds__(XT) k_fdm_xform(XformArgs a)
{
    extern __shared__ double X[];
    const int n = a.n, gs = a.gs, gp = a.gp;
    const int SR = x_stride(G * gp);
    constexpr int SC = NC + 4;
    auto sx = [&](int row, int col) { return ROWC ? col * SR + row : row * SC + col; };
    const int c0 = blockIdx.x * NC;
    auto base = [&](int c) -> int64_t {
        const int q = c / a.colw;
        return (int64_t)q * a.colrun + (int64_t)(c - q * a.colw) * a.colst;
    };
    const int h = n >> 1;
    // ---- load (forward: folded)
    const int rows = INV ? G * gp : gp;
    for (int t = threadIdx.x; t < rows * NC; t += XT) {
        int r, col;
        if (ROWC) { col = t / rows; r = t - col * rows; }
        else { r = t / NC; col = t - r * NC; }
        const int c = c0 + col;
        const bool on = c < a.ncol;
        const int64_t b = on ? base(c) : 0;
        if (INV) {
            const int g = r / gp, m = r - g * gp;
            // the last group of an odd direction has one mode less
            const int cnt = (G == 2 && g == 1) ? n - gs : gs;
            X[sx(r, col)] = (on && m < cnt) ? a.src[b + (int64_t)(g * gs + m) * a.se] : 0.0;
        } else {
            auto ld = [&](int i) {
                const int64_t q = b + (int64_t)i * a.se;
                return (a.d_sum && q == 0) ? -a.d_sum[0] : a.src[q];
            };
            const bool in = on && r < gs;
            if (G == 1) {
                X[sx(r, col)] = in ? ld(r) : 0.0;
            } else if (G == 2) {
                double v0 = 0.0, v1 = 0.0;
                if (in) {
                    const double p = ld(r);
                    if (2 * r + 1 == n) v0 = p;               // middle of an odd direction
                    else { const double q = ld(n - 1 - r); v0 = p + q; v1 = p - q; }
                }
                X[sx(r, col)] = v0;
                X[sx(gp + r, col)] = v1;
            } else {
                double v[4] = {0.0, 0.0, 0.0, 0.0};
                if (in) {
                    const double p = ld(r), q = ld(h - 1 - r), u = ld(n - 1 - r), w = ld(h + r);
                    const double s0 = p + u, s1 = q + w, d0 = p - u, d1 = q - w;
                    v[0] = s0 + s1; v[1] = s0 - s1; v[2] = d0 + d1; v[3] = d0 - d1;
                }
                #pragma unroll
                for (int g = 0; g < 4; g++) X[sx(g * gp + r, col)] = v[g];
            }
        }
    }
    __syncthreads();
    // ---- products. The two operand fragments of mma m8n8k4 have one layout, so
    // the panel is the column operand where rows are contiguous in memory and
    // the row operand where columns are: in both cases eight lanes store eight
    // adjacent doubles.
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, lr = lane >> 2, lc = lane & 3;
    const int nt = gp >> 3;
    auto step = [&](double (&d)[2], double wv, double xv) {
        if (ROWC) mma_f64(d, wv, xv);
        else mma_f64(d, xv, wv);
    };
    // column and row (in its tile of 8) of accumulator element e of column tile q
    auto colof = [&](int q, int e) { return q * 8 + (ROWC ? lc * 2 + e : lr); };
    auto rowof = [&](int e) { return ROWC ? lr : lc * 2 + e; };
    const double2 *A2 = reinterpret_cast<const double2 *>(a.A) + lane;
    const int tstep = (gp >> 3) * 32;                             // double2 per (group, row tile)
    if (!INV) {
        constexpr int CT = NC >= 32 ? 4 : NC / 8, NCH = NC / (8 * CT);   // column tiles per task, tasks per row tile
        for (int task = w; task < G * nt * NCH; task += XW) {
            const int ch = task % NCH, tile = task / NCH, g = tile / nt, m0 = (tile - g * nt) * 8;
            const double2 *A = A2 + (int64_t)tile * tstep;
            double acc[CT][2] = {};
            #pragma unroll 4
            for (int k = 0; k < gp; k += 8) {
                const double2 av = A[(k >> 3) * 32];
                #pragma unroll
                for (int q = 0; q < CT; q++) {
                    step(acc[q], av.x, X[sx(g * gp + k + lc, (ch * CT + q) * 8 + lr)]);
                    step(acc[q], av.y, X[sx(g * gp + k + 4 + lc, (ch * CT + q) * 8 + lr)]);
                }
            }
            const int cnt = (G == 2 && g == 1) ? n - gs : gs;
            #pragma unroll
            for (int q = 0; q < CT; q++)
                #pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int c = c0 + colof(ch * CT + q, e), m = m0 + rowof(e);
                    if (c >= a.ncol || m >= cnt) continue;
                    double v = acc[q][e];
                    if (a.ly) {
                        const double l = a.lx[c % a.sx] + a.ly[g * gs + m] + a.lz[c / a.sx];
                        v = l > 0.0 ? v / l : 0.0;
                    }
                    a.dst[base(c) + (int64_t)(g * gs + m) * a.se] = v;
                }
        }
    } else {
        constexpr int CT = NC >= 16 ? 2 : 1, NCH = NC / (8 * CT);
        for (int task = w; task < nt * NCH; task += XW) {
            const int ch = task % NCH, tile = task / NCH, i0 = tile * 8;
            double acc[G][CT][2] = {};
            #pragma unroll 2
            for (int k = 0; k < gp; k += 8) {
                #pragma unroll
                for (int g = 0; g < G; g++) {
                    const double2 av = A2[(int64_t)(g * nt + tile) * tstep + (k >> 3) * 32];
                    #pragma unroll
                    for (int q = 0; q < CT; q++) {
                        step(acc[g][q], av.x, X[sx(g * gp + k + lc, (ch * CT + q) * 8 + lr)]);
                        step(acc[g][q], av.y, X[sx(g * gp + k + 4 + lc, (ch * CT + q) * 8 + lr)]);
                    }
                }
            }
            #pragma unroll
            for (int q = 0; q < CT; q++)
                #pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int c = c0 + colof(ch * CT + q, e), i = i0 + rowof(e);
                    if (c >= a.ncol || i >= gs) continue;
                    double *d = a.dst + base(c);
                    if (G == 1) {
                        d[(int64_t)i * a.se] = acc[0][q][e];
                    } else if (G == 2) {
                        const double p = acc[0][q][e], u = acc[G > 1 ? 1 : 0][q][e];
                        d[(int64_t)i * a.se] = p + u;
                        if (2 * i + 1 != n) d[(int64_t)(n - 1 - i) * a.se] = p - u;
                    } else {
                        const double v0 = acc[0][q][e], v1 = acc[G > 1 ? 1 : 0][q][e], v2 = acc[G > 2 ? 2 : 0][q][e], v3 = acc[G > 3 ? 3 : 0][q][e];
                        const double sp = v0 + v1, sm = v0 - v1, dp = v2 + v3, dm = v2 - v3;
                        d[(int64_t)i * a.se] = sp + dp;
                        d[(int64_t)(h - 1 - i) * a.se] = sm + dm;
                        d[(int64_t)(n - 1 - i) * a.se] = sp - dp;
                        d[(int64_t)(h + i) * a.se] = sm - dm;
                    }
                }
        }
    }
}

// ---------------------------------------------------------- j-line systems
// T = (lx + lz) My + Ky, factors 1/m_j with m_j = t_jj - ky_{j-1}^2 / m_{j-1};
// the singular pair of constant modes gets ky_0 added to its first pivot, which
// fixes the free constant
__global__ void k_fdm_factors(int nx, int ny, int nz, const double *lx, const double *lz, const double *my, const double *ky,
                              double *minv)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= nx || k >= nz) return;
    const double l = lx[i] + lz[k];
    double kl = 0.0, mi = 0.0;
    for (int j = 0; j < ny; j++) {
        const double kr = j < ny - 1 ? ky[j] : 0.0;
        double m = l * my[j] + kl + kr - kl * kl * mi;
        if (j == 0 && l <= 0.0) m += kr;
        mi = 1.0 / m;
        minv[((int64_t)k * ny + j) * nx + i] = mi;
        kl = kr;
    }
}

// Line solve, in place. A block takes 32 adjacent lines (lanes) and one chunk of
// CJ cells per warp; a thread keeps its chunk of z and of the factors in
// registers, so every array is read or written once. The forward and backward
// recurrences are affine in the value that enters the chunk: a first pass from
// zero gives each chunk's (offset, multiplier), the warps chain those of the
// chunks before theirs, and a second pass from the entering value gives the
// chunk's cells.
template <int CJ, int MAXW>
__global__ void __launch_bounds__(32 * MAXW) k_fdm_lines_chunk(int nx, int ny, int nz, const double *__restrict__ ky,
                                                          const double *__restrict__ minv, double *z)
{
    __shared__ double SO[MAXW][32], SM[MAXW][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int line = blockIdx.x * 32 + lane;
    const bool on = line < nx * nz;
    const int k = on ? line / nx : 0, i = line - k * nx, j0 = w * CJ;
    const int64_t b = ((int64_t)k * ny + j0) * nx + i;
    // r: right-hand side, then d', then x; f: ky_j / m_j
    double r[CJ], f[CJ];
    #pragma unroll
    for (int u = 0; u < CJ; u++) {
        const bool in = on && j0 + u < ny;
        r[u] = in ? z[b + (int64_t)u * nx] : 0.0;
        f[u] = in ? minv[b + (int64_t)u * nx] : 0.0;
    }
    // forward: d_j = (r_j + ky_{j-1} d_{j-1}) / m_j
    double o = 0.0, m = 1.0;
    #pragma unroll
    for (int u = 0; u < CJ; u++) {
        const double kl = (j0 + u > 0 && j0 + u < ny) ? ky[j0 + u - 1] : 0.0;
        o = (r[u] + kl * o) * f[u];
        m *= kl * f[u];
    }
    SO[w][lane] = o;
    SM[w][lane] = m;
    __syncthreads();
    double d = 0.0;
    for (int q = 0; q < w; q++) d = SO[q][lane] + SM[q][lane] * d;
    #pragma unroll
    for (int u = 0; u < CJ; u++) {
        const double kl = (j0 + u > 0 && j0 + u < ny) ? ky[j0 + u - 1] : 0.0;
        d = (r[u] + kl * d) * f[u];
        r[u] = d;
        f[u] *= j0 + u < ny - 1 ? ky[j0 + u] : 0.0;
    }
    // backward: x_j = d_j + (ky_j / m_j) x_{j+1}
    o = 0.0; m = 1.0;
    #pragma unroll
    for (int u = CJ - 1; u >= 0; u--) {
        o = r[u] + f[u] * o;
        m *= f[u];
    }
    __syncthreads();
    SO[w][lane] = o;
    SM[w][lane] = m;
    __syncthreads();
    double x = 0.0;
    for (int q = nw - 1; q > w; q--) x = SO[q][lane] + SM[q][lane] * x;
    #pragma unroll
    for (int u = CJ - 1; u >= 0; u--) {
        x = r[u] + f[u] * x;
        if (on && j0 + u < ny) z[b + (int64_t)u * nx] = x;
    }
}

// lines of more than 256 cells: one thread per line, in place, adjacent threads
// on adjacent lines; the loads of TU steps are issued ahead of the chain
constexpr int TU = 8;
__global__ void __launch_bounds__(64) k_fdm_lines(int nx, int ny, int nz, const double *__restrict__ ky,
                                                  const double *__restrict__ minv, double *z)
{
    const int line = blockIdx.x * blockDim.x + threadIdx.x;
    if (line >= nx * nz) return;
    const int k = line / nx, i = line - k * nx;
    const int64_t b = (int64_t)k * ny * nx + i;
    double d = 0.0, r[TU], m[TU];
    for (int j = 0; j < ny; j += TU) {
        #pragma unroll
        for (int u = 0; u < TU; u++)
            if (j + u < ny) { r[u] = z[b + (int64_t)(j + u) * nx]; m[u] = minv[b + (int64_t)(j + u) * nx]; }
        #pragma unroll
        for (int u = 0; u < TU; u++)
            if (j + u < ny) {
                d = (r[u] + (j + u > 0 ? ky[j + u - 1] : 0.0) * d) * m[u];
                z[b + (int64_t)(j + u) * nx] = d;
            }
    }
    double x = d;
    for (int j = ny - 2; j >= 0; j -= TU) {
        #pragma unroll
        for (int u = 0; u < TU; u++)
            if (j - u >= 0) { r[u] = z[b + (int64_t)(j - u) * nx]; m[u] = minv[b + (int64_t)(j - u) * nx] * ky[j - u]; }
        #pragma unroll
        for (int u = 0; u < TU; u++)
            if (j - u >= 0) {
                x = r[u] + m[u] * x;
                z[b + (int64_t)(j - u) * nx] = x;
            }
    }
}

void launch_lines(const double *ky, const double *minv, double *z, int nx, int ny, int nz, cudaStream_t st)
{
    const int nb = (nx * nz + 31) / 32;
    // 4 to 8 chunks per line, up to 16 of the longest chunk that fits the registers
    if (ny <= 32) k_fdm_lines_chunk<4, 8><<<nb, 32 * ((ny + 3) / 4), 0, st>>>(nx, ny, nz, ky, minv, z);
    else if (ny <= 64) k_fdm_lines_chunk<8, 8><<<nb, 32 * ((ny + 7) / 8), 0, st>>>(nx, ny, nz, ky, minv, z);
    else if (ny <= 256) k_fdm_lines_chunk<16, 16><<<nb, 32 * ((ny + 15) / 16), 0, st>>>(nx, ny, nz, ky, minv, z);
    else k_fdm_lines<<<(nx * nz + 63) / 64, 64, 0, st>>>(nx, ny, nz, ky, minv, z);
}

// largest relative deviation of the coefficients from their factors
__global__ void __launch_bounds__(256) k_fdm_check(int nx, int ny, int nz, int pi, int pj, int pk, const double *aE, const double *aN,
                                                   const double *aT, const double *kx, const double *mx, const double *ky,
                                                   const double *my, const double *kz, const double *mz, double *part)
{
    const int64_t n = (int64_t)nx * ny * nz;
    double mm = 0.0;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(t % nx);
        const int64_t r = t / nx;
        const int j = (int)(r % ny), k = (int)(r / ny);
        if (i < nx - 1 || pi) mm = nanmax(mm, fabs(aE[t] / (kx[i] * my[j] * mz[k]) - 1.0));
        if (j < ny - 1 || pj) mm = nanmax(mm, fabs(aN[t] / (mx[i] * ky[j] * mz[k]) - 1.0));
        if (k < nz - 1 || pk) mm = nanmax(mm, fabs(aT[t] / (mx[i] * my[j] * kz[k]) - 1.0));
    }
    double v[1] = {mm};
    block_reduce<256>(v, RedNanMax{});
    if (threadIdx.x == 0) part[blockIdx.x] = v[0];
}

// ------------------------------------------------------------------ set-up
// Eigenpairs of the symmetric tridiagonal matrix (d, e) by implicitly shifted
// QR steps (Golub and Van Loan, section 8.3): d becomes the eigenvalues, row m
// of V (n x n, identity on entry) the eigenvector of d[m]. false if it does not
// converge.
bool tridiag_eig(std::vector<double> &d, std::vector<double> &e, std::vector<double> &V, int n)
{
    int hi = n - 1, sweeps = 0;
    while (hi > 0) {
        // deflate from the end, then find the unreduced block ending at hi
        if (std::fabs(e[hi - 1]) <= 1e-16 * (std::fabs(d[hi - 1]) + std::fabs(d[hi]))) { e[hi - 1] = 0.0; hi--; sweeps = 0; continue; }
        if (++sweeps > 200) return false;
        int lo = hi - 1;
        while (lo > 0 && std::fabs(e[lo - 1]) > 1e-16 * (std::fabs(d[lo - 1]) + std::fabs(d[lo]))) lo--;
        // Wilkinson shift: the eigenvalue of the trailing 2 x 2 block nearer d[hi]
        const double t = 0.5 * (d[hi - 1] - d[hi]), f = e[hi - 1];
        const double mu = d[hi] - f * f / (t + (t >= 0 ? 1.0 : -1.0) * std::hypot(t, f));
        double x = d[lo] - mu, z = e[lo];
        for (int k = lo; k < hi; k++) {
            const double r = std::hypot(x, z), c = r > 0 ? x / r : 1.0, s = r > 0 ? z / r : 0.0;
            if (k > lo) e[k - 1] = r;
            const double a = d[k], b = d[k + 1], g = e[k];
            d[k] = c * c * a + 2 * c * s * g + s * s * b;
            d[k + 1] = s * s * a - 2 * c * s * g + c * c * b;
            e[k] = c * s * (b - a) + (c * c - s * s) * g;
            if (k < hi - 1) {
                x = e[k];
                z = s * e[k + 1];
                e[k + 1] *= c;
            }
            double *p = &V[(size_t)k * n], *q = &V[(size_t)(k + 1) * n];
            for (int i = 0; i < n; i++) { const double u = p[i], w = q[i]; p[i] = c * u + s * w; q[i] = c * w - s * u; }
        }
    }
    return true;
}

bool is_uniform(const std::vector<double> &v, int cnt)
{
    for (int q = 1; q < cnt; q++)
        if (!(std::fabs(v[q] - v[0]) <= 1e-10 * std::fabs(v[0]))) return false;
    return true;
}

// The rows per group of the two transformed directions together: the transforms'
// work per cell grows with it, that of a multigrid cycle does not. Measured,
// ms per step (mixed) of the direct solve against the multigrid: 1024 x 512 x 32
// (384 rows) 12.2 against 16.4, 75 x 75 x 25 (76) 0.36 against 1.38; 2048 x 32 x 32
// (520) 2.84 against 2.71, 2047 x 32 x 32 open in x (1032) 3.64 against 3.29. A
// periodic j has the bound for itself: its rows are not added to the two, because
// the multigrid is slower there as well (point instead of line sweeps): 1.90 direct
// and 2.42 multigrid at 32 x 32 x 2048 (16 + 512 rows), 5.16 and 8.52 at 64 x 64 x 2048
// (32 + 512), 6.23 and 15.6 at 128 x 128 x 1024 (64 + 256). The bound also keeps the
// panels in shared memory and the set-up of an unfolded direction (n^3) at a tenth
// of a second.
constexpr int FDM_MAX_ROWS = 512;

template <class T>
T *to_device(tg_ctx *C, const std::vector<T> &h)
{
    T *d = (T *)dalloc(C, sizeof(T) * h.size());
    TG_CUDA(cudaMemcpyAsync(d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice, C->stream));
    TG_CUDA(cudaStreamSynchronize(C->stream));
    return d;
}

// place of element (row, col) of group g: tiles of 8 rows, within a tile steps
// of 8 columns, within a step the 32 lanes of a fragment (row % 8, col % 4) with
// their two fragments (col / 4 % 2) adjacent, so that a warp loads 512
// contiguous bytes per step
size_t frag_index(int gp, int g, int row, int col)
{
    const size_t tile = (size_t)g * (gp >> 3) + (row >> 3);
    return ((tile * (gp >> 3) + (col >> 3)) * 32 + (row & 7) * 4 + (col & 3)) * 2 + ((col >> 2) & 1);
}

// The groups and rows of one direction from its coefficients: k[i] that of face
// i+1/2, m the masses. false when the direction is not supported. This decides
// before any eigenproblem (n^3 for an unfolded direction, 0.05 to 0.13 s at
// 500 cells) and any allocation.
bool plan_dir(FdmDir &D, int n, bool periodic, const std::vector<double> &k, const std::vector<double> &m)
{
    D.n = n;
    D.uni = is_uniform(k, periodic ? n : n - 1) && is_uniform(m, n);
    D.per = periodic;
    D.G = !D.uni ? 1 : (periodic && n % 4 == 0) ? 4 : 2;
    D.gs = (n + D.G - 1) / D.G;
    D.gp = (D.gs + 7) / 8 * 8;
    return (D.uni || !periodic) && D.gs <= FDM_MAX_ROWS;
}

// eigenvectors and eigenvalues of (K, M) of a planned direction, on the host
struct FdmVectors { std::vector<double> W, Wt, lam; };
bool solve_dir(const FdmDir &D, const std::vector<double> &k, const std::vector<double> &m, FdmVectors &E)
{
    const int n = D.n, G = D.G, gs = D.gs, gp = D.gp;
    const bool periodic = D.per;
    std::vector<double> &W = E.W, &Wt = E.Wt, &lam = E.lam;
    W.assign((size_t)G * gp * gp, 0.0);
    Wt = W;
    lam.assign(n, 0.0);
    auto put = [&](int g, int q, int i, double v) {
        W[frag_index(gp, g, q, i)] = v;
        Wt[frag_index(gp, g, i, q)] = v;
    };
    if (D.uni) {
        const double rm = 1.0 / std::sqrt(m[0]), ratio = k[0] / m[0];
        // mode of frequency f (angle pi f (i + 1/2) / n): cosine or sine,
        // normalised over the n points; its angle is reduced exactly in units
        // of pi / (2 n)
        auto mode = [&](int g, int q, int f, bool sine) {
            const bool half = sine ? (f == n) : (f == 0);      // norm n instead of n / 2
            const double s = std::sqrt((half ? 1.0 : 2.0) / n) * rm;
            for (int i = 0; i < gs; i++) {
                const int64_t a = (int64_t)f * (2 * i + 1) % (4 * (int64_t)n);
                const double th = M_PI * (double)a / (2.0 * n);
                // an odd direction has no odd part at its middle cell
                if (G == 2 && g == 1 && 2 * i + 1 == n) continue;
                put(g, q, i, s * (sine ? std::sin(th) : std::cos(th)));
            }
            const double sn = std::sin(M_PI * f / (2.0 * n));
            lam[(size_t)g * gs + q] = 4.0 * ratio * sn * sn;
        };
        if (!periodic) {                 // cos(pi f (i+1/2) / n): even f symmetric
            for (int f = 0; f < n; f++) mode(f & 1, f >> 1, f, false);
        } else if (G == 2) {             // frequencies 2 m
            for (int q = 0; 2 * q < n; q++) mode(0, q, 2 * q, false);
            for (int q = 1; 2 * q <= n; q++) mode(1, q - 1, 2 * q, true);
        } else {                         // second fold: parity of m
            const int h = n / 2;
            for (int q = 0; q < h; q++) mode(q & 1, q >> 1, 2 * q, false);
            for (int q = 1; q <= h; q++) mode((q & 1) ? 2 : 3, (q - 1) >> 1, 2 * q, true);
        }
    } else {
        std::vector<double> d(n), e(n, 0.0), V((size_t)n * n, 0.0);
        for (int i = 0; i < n; i++) {
            d[i] = ((i > 0 ? k[i - 1] : 0.0) + (i < n - 1 ? k[i] : 0.0)) / m[i];
            if (i < n - 1) e[i] = -k[i] / std::sqrt(m[i] * m[i + 1]);
            V[(size_t)i * n + i] = 1.0;
        }
        if (!tridiag_eig(d, e, V, n)) return false;
        const int z = (int)(std::min_element(d.begin(), d.end()) - d.begin());
        for (int q = 0; q < n; q++) {
            lam[q] = q == z ? 0.0 : d[q];          // constants are the null space
            for (int i = 0; i < n; i++) put(0, q, i, V[(size_t)q * n + i] / std::sqrt(m[i]));
        }
    }
    return true;
}
void upload_dir(tg_ctx *C, FdmDir &D, const FdmVectors &E)
{
    D.W = to_device(C, E.W);
    D.Wt = to_device(C, E.Wt);
    D.lam = to_device(C, E.lam);
}

// Columns per panel: the widest whose panel of the contiguous direction takes at
// most a third of the shared memory, so that three blocks share an SM there; the
// narrowest in any case. The strided directions take the same width: their panels
// pad each row instead of each column and can be a little larger (82 KB at 288 and
// at 512 rows, two blocks), but narrower ones gain 6 % at 512 and lose 25 % at 288.
// Forward / inverse at 128 x 64 columns, us, width in brackets: 256 cells 26.5 / 29.0 (32), 24.9 / 35.1 (16);
// 288 31.5 / 36.4 (32), 30.0 / 53.6 (16), 36.1 / 45.4 (8); 512 80.4 / 86.4 (16), 72.2 / 84.8 (8).
int panel_cols(const FdmDir &D)
{
    for (int nc : {32, 16}) if ((size_t)nc * x_stride(D.G * D.gp) * 8 <= 75 * 1024) return nc;
    return 8;
}
size_t panel_smem(const FdmDir &D, bool rowc, int nc)
{
    return sizeof(double) * (rowc ? (size_t)nc * x_stride(D.G * D.gp) : (size_t)D.G * D.gp * (nc + 4));
}

template <int G, bool INV, bool ROWC>
void launch_xform_g(const FdmDir &D, const XformArgs &a, cudaStream_t st)
{
    const int nc = panel_cols(D), nb = (a.ncol + nc - 1) / nc;
    const size_t sm = panel_smem(D, ROWC, nc);
    if (nc == 32) k_fdm_xform<G, INV, ROWC, 32><<<nb, XT, sm, st>>>(a);
    else if (nc == 16) k_fdm_xform<G, INV, ROWC, 16><<<nb, XT, sm, st>>>(a);
    else k_fdm_xform<G, INV, ROWC, 8><<<nb, XT, sm, st>>>(a);
}
template <bool INV, bool ROWC>
void launch_xform(const FdmDir &D, XformArgs a, cudaStream_t st)
{
    a.n = D.n; a.gs = D.gs; a.gp = D.gp;
    a.A = INV ? D.Wt : D.W;
    if (D.G == 4) launch_xform_g<4, INV, ROWC>(D, a, st);
    else if (D.G == 2) launch_xform_g<2, INV, ROWC>(D, a, st);
    else launch_xform_g<1, INV, ROWC>(D, a, st);
}

template <int G, bool INV, bool ROWC>
void set_attr_g()
{
    auto set = [](const void *f) { TG_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024)); };
    set((const void *)k_fdm_xform<G, INV, ROWC, 32>);
    set((const void *)k_fdm_xform<G, INV, ROWC, 16>);
    set((const void *)k_fdm_xform<G, INV, ROWC, 8>);
}
void set_attrs()
{
    set_attr_g<1, false, false>(); set_attr_g<1, false, true>(); set_attr_g<1, true, false>(); set_attr_g<1, true, true>();
    set_attr_g<2, false, false>(); set_attr_g<2, false, true>(); set_attr_g<2, true, false>(); set_attr_g<2, true, true>();
    set_attr_g<4, false, false>(); set_attr_g<4, false, true>(); set_attr_g<4, true, false>(); set_attr_g<4, true, true>();
}

}  // namespace

Fdm *fdm_create(tg_ctx *C, const Tensor *t, const double *aE, const double *aN, const double *aT,
                int nx, int ny, int nz, int pi, int pj, int pk)
{
    cudaStream_t st = C->stream;
    const size_t pl = (size_t)nx * ny;
    auto line = [&](const double *a, size_t stride, int n) {
        std::vector<double> h(n);
        TG_CUDA(cudaMemcpy2DAsync(h.data(), sizeof(double), a, stride * sizeof(double), sizeof(double), n, cudaMemcpyDeviceToHost, st));
        TG_CUDA(cudaStreamSynchronize(st));
        return h;
    };
    std::vector<double> kx, mx, ky, my, kz, mz;
    if (t) {
        // cells 1 .. of the DMDA; the masses are the sizes, and a factor has one
        // rounding where one read off the coefficients has three
        kx = line(t->rdyf + 1, 1, nx); mx = line(t->dy + 1, 1, nx);
        ky = line(t->rdzf + 1, 1, ny); my = line(t->dz + 1, 1, ny);
        kz = line(t->rdxf + 1, 1, nz); mz = line(t->dx + 1, 1, nz);
        // two axes may run downwards; the coefficients' sign is checked below
        for (auto *v : {&kx, &mx, &ky, &my, &kz, &mz})
            for (double &q : *v) q = std::fabs(q);
    } else {
        // lines of coefficients through cell (0, 0, 0), normalised to mx_0 = my_0 = mz_0 = 1
        kx = line(aE, 1, nx); mx = line(aN, 1, nx); ky = line(aN, nx, ny); mz = line(aN, pl, nz); my = line(aT, nx, ny); kz = line(aT, pl, nz);
        const double n0 = ky[0], t0 = kz[0];
        for (double &v : mx) v /= n0;
        for (double &v : mz) v /= n0;
        for (double &v : my) v /= t0;
    }
    auto positive = [](const std::vector<double> &v, int cnt) {
        for (int q = 0; q < cnt; q++) if (!(v[q] > 0.0) || !std::isfinite(v[q])) return false;
        return true;
    };
    if (!positive(kx, pi ? nx : nx - 1) || !positive(mx, nx) || !positive(ky, pj ? ny : ny - 1) || !positive(mz, nz) ||
        !positive(my, ny) || !positive(kz, pk ? nz : nz - 1)) return nullptr;
    FdmDir dx, dy, dz;
    if (!plan_dir(dx, nx, pi, kx, mx) || !plan_dir(dz, nz, pk, kz, mz) || (pj && !plan_dir(dy, ny, true, ky, my)) ||
        dx.gs + dz.gs > FDM_MAX_ROWS) return nullptr;
    Fdm *F = new Fdm();
    F->nx = nx; F->ny = ny; F->nz = nz; F->pj = pj;
    F->n = (int64_t)nx * ny * nz;
    F->x = dx; F->y = dy; F->z = dz;
    try {
        double *dv[6];
        const std::vector<double> *hv[6] = {&kx, &mx, &ky, &my, &kz, &mz};
        for (int q = 0; q < 6; q++) dv[q] = to_device(C, *hv[q]);
        k_fdm_check<<<C->red_blocks, 256, 0, st>>>(nx, ny, nz, pi, pj, pk, aE, aN, aT, dv[0], dv[1], dv[2], dv[3], dv[4], dv[5], C->d_red);
        std::vector<double> part(C->red_blocks);
        TG_CUDA(cudaMemcpyAsync(part.data(), C->d_red, sizeof(double) * part.size(), cudaMemcpyDeviceToHost, st));
        TG_CUDA(cudaStreamSynchronize(st));
        bool ok = true;
        // rounding of the metrics leaves about 1e-15; the factors only have to
        // be close, as CG iterates on the exact operator
        F->dev = 0.0;
        for (double v : part) { ok = ok && v <= 1e-10; F->dev = std::max(F->dev, v); }
        FdmVectors ex, ey, ez;
        ok = ok && solve_dir(dx, kx, mx, ex) && solve_dir(dz, kz, mz, ez) && (!pj || solve_dir(dy, ky, my, ey));
        if (!ok) { delete F; return nullptr; }
        upload_dir(C, F->x, ex);
        upload_dir(C, F->z, ez);
        if (pj) upload_dir(C, F->y, ey);
        F->op = FdmOp{dv[0], dv[1], dv[2], dv[3], dv[4], dv[5]};
        if (!pj) {
            F->minv = dallocd(C, (size_t)F->n);
            k_fdm_factors<<<dim3((nx + 31) / 32, (nz + 3) / 4), dim3(32, 4), 0, st>>>(nx, ny, nz, F->x.lam, F->z.lam, F->op.my, F->op.ky, F->minv);
        }
        set_attrs();
        TG_CUDA(cudaGetLastError());
    } catch (...) {
        delete F;
        throw;
    }
    return F;
}

bool fdm_factors(const Fdm *F, FdmOp *op) { *op = F->op; return F->dev <= 1e-13; }

void fdm_destroy(Fdm *F) { delete F; }   // the device buffers go with the solver's

void fdm_apply(tg_ctx *C, Fdm *F, const double *r, const double *d_sum, double *z)
{
    cudaStream_t st = C->stream;
    const int nx = F->nx, ny = F->ny, nz = F->nz, pl = nx * ny;
    XformArgs ax{}, ay{}, az{};
    ax.se = 1; ax.ncol = ny * nz; ax.colw = ny * nz; ax.colst = nx;
    az.se = pl; az.ncol = pl; az.colw = pl; az.colst = 1;
    ay.se = nx; ay.ncol = nx * nz; ay.colw = nx; ay.colst = 1; ay.colrun = pl;
    ax.src = r; ax.dst = z; ax.d_sum = d_sum;
    az.dst = ay.dst = z;
    az.src = ay.src = z;
    TG_PROF(C, "fdm_x_fwd", (launch_xform<false, true>(F->x, ax, st)));
    TG_PROF(C, "fdm_z_fwd", (launch_xform<false, false>(F->z, az, st)));
    if (F->pj) {
        ay.lx = F->x.lam; ay.ly = F->y.lam; ay.lz = F->z.lam; ay.sx = nx;
        TG_PROF(C, "fdm_y_fwd", (launch_xform<false, false>(F->y, ay, st)));
        ay.ly = nullptr;
        TG_PROF(C, "fdm_y_inv", (launch_xform<true, false>(F->y, ay, st)));
    } else {
        TG_PROF(C, "fdm_lines", launch_lines(F->op.ky, F->minv, z, nx, ny, nz, st));
    }
    TG_PROF(C, "fdm_z_inv", (launch_xform<true, false>(F->z, az, st)));
    ax.src = z; ax.d_sum = nullptr;
    TG_PROF(C, "fdm_x_inv", (launch_xform<true, true>(F->x, ax, st)));
}

}  // namespace tg
