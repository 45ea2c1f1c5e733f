// Multigrid passes (mg_fused.h).
//
// Large levels stream: one thread per (x, y) column marching z, four planes of loads in flight, no
// index divided; the two pre-smoothings from zero are one pass.
//
// On coarse levels a launch costs more than its work (3.5 us per pass on grids of 33^3 and below,
// whatever it does), so a level of up to MG_TILE_MAX points is two launches:
//   down  both pre-smoothings, the residual and its restriction, in shared memory on a tile of
//         4 x 2 x 2 coarse points and the fine points it needs (the halo is recomputed);
//   up    interpolation and both post-smoothings on a tile of 8 x 4 x 4 fine points.
// The tiles are small so that a 17^3 level still spreads over 75 blocks (tiles of eight times the points
// took 11 to 13 us each there).  A cluster per field that ran all passes of these levels in one
// launch with a cluster barrier between them took 64 us where these launches take 30: each pass paid an L2
// round trip and the barrier.
//
// The restriction weights and interpolation cells of every level come from a table (mg_tables; one launch per
// Poisson solve, and per cycle of the eigensolver's preconditioner and the mixer): a tile's own divisions took
// longer than its passes.
//
// Every pass keeps the operations and the order of the separate passes it replaces (divisions by the
// diagonal through exact_div.cuh), so the preconditioner's results are the same bits however a level is
// cut.
// Measured: poisson start + cycles + stop at 128^3 8.9 -> 4.2 ms.
#include <algorithm>
#include <cmath>

#include "exact_div.cuh"
#include "mg_fused.h"
#include "neural.h"

namespace dftb {

namespace {

constexpr long long MG_TILE_MAX = 40000;
constexpr int DX = 4, DY = 2, DZ = 2;                 // coarse points of a down tile
// residual points that 4 (2) coarse points at most 2 fine spacings apart draw on: the closed
// interval of 4 + 1 (2 + 1) coarse spacings holds at most 11 (7), ends of no or rounding weight included
constexpr int RX = 11, RY = 7, RZ = 7;
constexpr int VX = RX + 2, VY = RY + 2, VZ = RZ + 2;  // with the neighbours of the residual
constexpr int SX = VX + 2, SY = VY + 2, SZ = VZ + 2;  // with the neighbours of the second smoothing
constexpr int UX = SX + 2, UY = SY + 2, UZ = SZ + 2;  // and those of the first
constexpr int FX = 8, FY = 4, FZ = 4;                 // fine points of an up tile
constexpr int MT = 512;

template <int W, int H>
__device__ __forceinline__ void split(int p, int& x, int& y, int& z) {
    z = p / (W * H);
    const int r = p - z * (W * H);
    y = r / W;
    x = r - y * W;
}

struct Box {  // grid limits: inside the grid, and points that are unknowns
    int nx, ny, nz, lo, hx, hy, hz;
    __device__ __forceinline__ Box(const Grid& g, int open)
        : nx(g.nx), ny(g.ny), nz(g.nz), lo(open ? 0 : 1), hx(g.nx - lo), hy(g.ny - lo), hz(g.nz - lo) {}
    __device__ __forceinline__ bool in(int x, int y, int z) const {
        return (unsigned)x < (unsigned)nx && (unsigned)y < (unsigned)ny && (unsigned)z < (unsigned)nz;
    }
    __device__ __forceinline__ bool unknown(int x, int y, int z) const {
        return x >= lo && x < hx && y >= lo && y < hy && z >= lo && z < hz;
    }
};

// sum of w v over the six neighbours (those outside the grid are zero in a)
__device__ __forceinline__ double weighted(const Grid& g, double xm, double xp, double ym, double yp, double zm,
                                           double zp) {
    return fma(g.iy2, yp, fma(g.iy2, ym, fma(g.ix2, xp, fma(g.ix2, xm, g.iz2 * (zm + zp)))));
}
template <int W, int WH>
__device__ __forceinline__ double neighbours(const Grid& g, const double* a, int i) {
    return weighted(g, a[i - 1], a[i + 1], a[i - W], a[i + W], a[i - WH], a[i + WH]);
}
// one weighted-Jacobi step at a point with value v, neighbour sum nb and right-hand side b (scale s)
__device__ __forceinline__ double smoothed(double v, double nb, double s, double b, const ExactDiv& d) {
    return fma(MG_OMEGA, divide(fma(s, b, nb), d) - v, v);
}
__device__ __forceinline__ double residual(double v, double nb, double s, double b, const ExactDiv& d) {
    return fma(s, b, -fma(d.b, v, -nb));
}

// Restriction weights (transposed trilinear) of coarse index C along an axis: fine points lo .. lo + 4, zero where
// a point is outside the grid or beyond one coarse spacing.  first: the unclipped lo.
__device__ __forceinline__ int hat(int C, double h, double H, int nf, double (&w)[5]) {
    const double X = C * H;
    const int lo = (int)ceil((X - H) / h);
    const int hi = min(nf - 1, (int)floor((X + H) / h));
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int fi = lo + k;
        const double wgt = 1.0 - fabs(fi * h - X) / H;
        w[k] = fi >= 0 && fi <= hi && wgt > 0.0 ? wgt : 0.0;
    }
    return lo;
}

// One cell and weight of the trilinear interpolation along an axis.
__device__ __forceinline__ void cell(int i, int nc, double h, double H, int& I, double& w) {
    const double u = i * h / H;
    I = min(max((int)floor(u), 0), nc - 2);
    w = fmin(fmax(u - I, 0.0), 1.0);
}
// the bilinear value in one coarse plane, e at its lower corner
__device__ __forceinline__ double bilinear(const double* e, int nx, double wx, double wy) {
    const double e00 = __ldg(e), e01 = __ldg(e + 1), e10 = __ldg(e + nx), e11 = __ldg(e + nx + 1);
    return (1.0 - wy) * ((1.0 - wx) * e00 + wx * e01) + wy * ((1.0 - wx) * e10 + wx * e11);
}

// Streaming passes: one thread per (x, y) column and z chunk.  blockIdx.z = field * nzc + chunk.
constexpr int CBX = 32, CBY = 8;

// ZERO: both smoothings from zero in one pass (the first is pointwise); SMOOTH: one smoothing from v;
// RESIDUAL: out = s src - (d v - sum), zero where nothing is unknown
enum { SMOOTH, ZERO_TWICE, RESIDUAL };
template <int MODE>
__global__ void __launch_bounds__(CBX* CBY, 2)
    mg_column_kernel(Grid f, int open, double s, const double* __restrict__ shift, const double* __restrict__ src,
                     const int* __restrict__ map, long long ld, const double* __restrict__ v, double* __restrict__ out,
                     int zc, int nzc, MGHistory* hist) {
    constexpr bool ZERO = MODE == ZERO_TWICE;
    constexpr int U = 4;  // planes whose loads are in flight together
    const int i = blockIdx.x * CBX + threadIdx.x, j = blockIdx.y * CBY + threadIdx.y;
    const int a = blockIdx.z / nzc, kc = blockIdx.z - a * nzc;
    if (hist && i == 0 && j == 0 && blockIdx.z == 0) hist->r[++hist->count & 63] = 0;
    if (i >= f.nx || j >= f.ny) return;
    const ExactDiv d = exact_div(2.0 * (f.ix2 + f.iy2 + f.iz2) + (shift ? shift[a] : 0.0));
    const double k1 = MG_OMEGA * s;
    const double* __restrict__ q = src + (long long)(map ? map[a] : a) * ld;
    const double* __restrict__ u = ZERO ? q : v + (long long)a * ld;  // the field whose neighbours are read
    double* __restrict__ o = out + (long long)a * ld;
    const int lo = open ? 0 : 1, sxy = f.nx * f.ny, col = j * f.nx + i;
    const int kb = kc * zc, ke = min(f.nz, kb + zc);
    // fixed points keep their value (residual: zero)
    const bool edge = i < lo || i >= f.nx - lo || j < lo || j >= f.ny - lo;
    if (edge) {
        for (int k = kb; k < ke; ++k) o[k * sxy + col] = MODE == SMOOTH ? __ldg(u + k * sxy + col) : 0.0;
        return;
    }
    if (lo && kb == 0) o[col] = MODE == SMOOTH ? __ldg(u + col) : 0.0;
    if (lo && ke == f.nz) o[(ke - 1) * sxy + col] = MODE == SMOOTH ? __ldg(u + (ke - 1) * sxy + col) : 0.0;
    const int k0 = max(kb, lo), k1e = min(ke, f.nz - lo);
    if (k0 >= k1e) return;
    // A neighbour outside the grid (from zero: or fixed) counts as zero: its load goes to the point
    // itself and its weight is zero, which leaves the sum as it is.
    const int e0 = ZERO ? lo : 0;
    const bool xl = i > e0, xr = i + 1 < f.nx - e0, yl = j > e0, yr = j + 1 < f.ny - e0;
    const int oxm = xl ? -1 : 0, oxp = xr ? 1 : 0, oym = yl ? -f.nx : 0, oyp = yr ? f.nx : 0;
    const double wxm = xl ? f.ix2 : 0.0, wxp = xr ? f.ix2 : 0.0, wym = yl ? f.iy2 : 0.0, wyp = yr ? f.iy2 : 0.0;
    const int zl = e0, zr = f.nz - e0;
    // the first smoothing's value (ZERO), by the fast quotient or, on a second try, the general one
    auto first = [&](double b, bool slow, bool& bad) {
        if (!ZERO) return b;
        if (slow) return divide(k1 * b, d);
        bool t;
        const double r = divide_fast(k1 * b, d, t);
        bad |= t;
        return r;
    };
    bool none = false;
    double below = k0 - 1 >= zl ? first(__ldg(u + (k0 - 1) * sxy + col), true, none) : 0.0;
    double cur = first(__ldg(u + k0 * sxy + col), true, none);
    for (int k = k0; k < k1e; k += U) {
        double ab[U], xm[U], xp[U], ym[U], yp[U], b[U], r[U];
#pragma unroll
        for (int t = 0; t < U; ++t) {  // past the end: the last plane again, not stored
            const int p = min(k + t, k1e - 1) * sxy + col;
            const double* w = u + p;
            ab[t] = k + t + 1 < zr ? __ldg(w + sxy) : 0.0;
            xm[t] = __ldg(w + oxm);
            xp[t] = __ldg(w + oxp);
            ym[t] = __ldg(w + oym);
            yp[t] = __ldg(w + oyp);
            b[t] = __ldg(q + p);
        }
        double lower, here;
        auto group = [&](bool slow) {
            bool bad = false;
            lower = below, here = cur;
#pragma unroll
            for (int t = 0; t < U; ++t) {
                const double above = first(ab[t], slow, bad);
                double nb = f.iz2 * (lower + above);
                nb = fma(wxm, first(xm[t], slow, bad), nb);
                nb = fma(wxp, first(xp[t], slow, bad), nb);
                nb = fma(wym, first(ym[t], slow, bad), nb);
                nb = fma(wyp, first(yp[t], slow, bad), nb);
                if (MODE == RESIDUAL) {
                    r[t] = residual(here, nb, s, b[t], d);
                } else {
                    const double num = fma(s, b[t], nb);
                    double vj;
                    if (slow) {
                        vj = divide(num, d);
                    } else {
                        bool out_of_range;
                        vj = divide_fast(num, d, out_of_range);
                        bad |= out_of_range;
                    }
                    r[t] = fma(MG_OMEGA, vj - here, here);
                }
                lower = here;
                here = above;
            }
            return bad;
        };
        if (group(false) || (MODE != RESIDUAL && d.general)) group(true);
        below = lower, cur = here;
#pragma unroll
        for (int t = 0; t < U; ++t)
            if (k + t < k1e) o[(k + t) * sxy + col] = r[t];
    }
}

// csrc = R(r), one axis after the other, each rounded to its own values: a block restricts along x all rows
// that its 16 x 4 x 4 coarse points draw on (at most 11 x 11: coarse points are at most 2 fine spacings apart),
// then along y and z in shared memory.  Restricting point by point read every row 2.25 times,
// one dependent row after the other: 28 us at 128^3, 17 us here.
constexpr int CX = 16, CY = 4, CZ = 4, CR = 11;
__global__ void __launch_bounds__(256)
    mg_restrict_kernel(Grid f, Grid c, MGTable T, const double* __restrict__ r, long long f_ld, double* __restrict__ csrc,
                       long long c_ld, int nz_blocks) {
    __shared__ double w[CX + CY + CZ][5];
    __shared__ int lo[CX + CY + CZ];
    __shared__ double A[CR * CR * CX], B[CR * CY * CX];
    const int a = blockIdx.z / nz_blocks, bz = blockIdx.z - a * nz_blocks;
    const int I0 = blockIdx.x * CX, J0 = blockIdx.y * CY, K0 = bz * CZ, tid = threadIdx.x;
    if (tid < 5 * (CX + CY + CZ)) {
        const int e = tid / 5, k = tid - 5 * e;
        const int C = e < CX ? I0 + e : e < CX + CY ? J0 + e - CX : K0 + e - CX - CY;
        const int m = e < CX ? c.nx : e < CX + CY ? c.ny : c.nz;
        const int at = (e < CX ? 0 : e < CX + CY ? c.nx : c.nx + c.ny) + min(C, m - 1);
        w[e][k] = C < m ? T.w[5 * at + k] : 0.0;
        if (k == 0) lo[e] = T.lo[at];
    }
    __syncthreads();
    const int y0 = lo[CX], z0 = lo[CX + CY], x = tid & (CX - 1);
    const double sx = f.dx / c.dx, sy = f.dy / c.dy, sz = f.dz / c.dz;
    const int sxy = f.nx * f.ny;
    double wx[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) wx[i] = w[x][i];
    const double* q = r + (long long)a * f_ld + lo[x];
#pragma unroll 4
    for (int row = tid / CX; row < CR * CR; row += 256 / CX) {
        const int z = row / CR, gy = y0 + row - z * CR, gz = z0 + z;
        const bool in = gy >= 0 && gy < f.ny && gz >= 0 && gz < f.nz;
        double v[5];
#pragma unroll
        for (int i = 0; i < 5; ++i) v[i] = in && wx[i] > 0.0 ? __ldg(q + gz * sxy + gy * f.nx + i) : 0.0;
        double t = 0.0;
#pragma unroll
        for (int i = 0; i < 5; ++i) t = fma(wx[i], v[i], t);
        A[row * CX + x] = t * sx;
    }
    __syncthreads();
    auto taps = [](const double* from, int stride, const double* wt) {
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < 5; ++k)
            if (wt[k] > 0.0) t = fma(wt[k], from[k * stride], t);
        return t;
    };
    for (int p = tid; p < CR * CY * CX; p += 256) {
        const int y = p / CX % CY, z = p / (CX * CY);
        B[p] = taps(A + (z * CR + lo[CX + y] - y0) * CX + x, CX, w[CX + y]) * sy;
    }
    __syncthreads();
    const int y = tid / CX % CY, z = tid / (CX * CY), I = I0 + x, J = J0 + y, K = K0 + z;
    if (I < c.nx && J < c.ny && K < c.nz)
        csrc[(long long)a * c_ld + ((long long)K * c.ny + J) * c.nx + I] =
            taps(B + (lo[CX + CY + z] - z0) * CY * CX + y * CX + x, CY * CX, w[CX + CY + z]) * sz;
}

// v += P e where v is unknown; the bilinear values of a coarse plane serve the fine planes around it
__global__ void __launch_bounds__(CBX* CBY)
    mg_correct_kernel(Grid f, Grid c, MGTable T, int open, long long f_ld, const double* __restrict__ e, long long c_ld,
                      double* __restrict__ v, int zc, int nzc) {
    const int i = blockIdx.x * CBX + threadIdx.x, j = blockIdx.y * CBY + threadIdx.y;
    const int a = blockIdx.z / nzc, kc = blockIdx.z - a * nzc;
    const int lo = open ? 0 : 1;
    if (i < lo || i >= f.nx - lo || j < lo || j >= f.ny - lo) return;
    const int I = T.ic[i], J = T.ic[f.nx + j];
    const double wx = T.iw[i], wy = T.iw[f.nx + j];
    const int cxy = c.nx * c.ny, fxy = f.nx * f.ny;
    const int* ic = T.ic + f.nx + f.ny;
    const double* iw = T.iw + f.nx + f.ny;
    const double* q = e + (long long)a * c_ld + J * c.nx + I;
    double* o = v + (long long)a * f_ld + (long long)j * f.nx + i;
    auto plane = [&](int K) { return bilinear(q + (long long)K * cxy, c.nx, wx, wy); };
    int at = -2;
    double p0 = 0.0, p1 = 0.0;
    const int k1 = min(f.nz - lo, (kc + 1) * zc);
    for (int k = max(lo, kc * zc); k < k1; k += 4) {
        double x[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) x[t] = k + t < k1 ? o[(long long)(k + t) * fxy] : 0.0;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            if (k + t >= k1) break;
            const int K = __ldg(ic + k + t);
            const double wz = __ldg(iw + k + t);
            if (K != at) {
                p0 = K == at + 1 ? p1 : plane(K);
                p1 = plane(K + 1);
                at = K;
            }
            o[(long long)(k + t) * fxy] = x[t] + ((1.0 - wz) * p0 + wz * p1);
        }
    }
}

// max |s src - (d v - sum)| over the interior
__global__ void __launch_bounds__(CBX* CBY)
    mg_residual_max_kernel(Grid f, double s, const double* __restrict__ src, const double* __restrict__ v,
                           MGHistory* hist, int zc) {
    __shared__ double sh[CBX * CBY / 32];
    const int i = blockIdx.x * CBX + threadIdx.x, j = blockIdx.y * CBY + threadIdx.y;
    const double d = 2.0 * (f.ix2 + f.iy2 + f.iz2);
    const int sxy = f.nx * f.ny;
    double m = 0.0;
    if (i >= 1 && i + 1 < f.nx && j >= 1 && j + 1 < f.ny) {
        const int kb = max(1, (int)blockIdx.z * zc), ke = min(f.nz - 1, (int)(blockIdx.z + 1) * zc);
        long long p = (long long)kb * sxy + (long long)j * f.nx + i;
        double below = kb < ke ? __ldg(v + p - sxy) : 0.0, cur = kb < ke ? __ldg(v + p) : 0.0;
#pragma unroll 2
        for (int k = kb; k < ke; ++k, p += sxy) {
            const double above = __ldg(v + p + sxy);
            const double nb = fma(f.iz2, below + above, fma(f.iy2, __ldg(v + p - f.nx) + __ldg(v + p + f.nx),
                                                            f.ix2 * (__ldg(v + p - 1) + __ldg(v + p + 1))));
            m = fmax(m, fabs(fma(s, __ldg(src + p), nb - d * cur)));
            below = cur;
            cur = above;
        }
    }
    m = warp_max(m);
    const int t = threadIdx.y * CBX + threadIdx.x;
    if ((t & 31) == 0) sh[t >> 5] = m;
    __syncthreads();
    if (t == 0) {
        for (int w = 1; w < CBX * CBY / 32; ++w) m = fmax(m, sh[w]);
        atomicMax(&hist->r[hist->count & 63], (unsigned long long)__double_as_longlong(m));
    }
}

__global__ void mg_start_cycle_kernel(MGHistory* hist) { hist->r[++hist->count & 63] = 0; }

// out = trilinear interpolation of e on the interior of f, 0 on its faces
__global__ void __launch_bounds__(CBX* CBY) mg_interpolate_kernel(Grid f, Grid c, const double* __restrict__ e,
                                                                 double* __restrict__ out, int zc) {
    const int i = blockIdx.x * CBX + threadIdx.x, j = blockIdx.y * CBY + threadIdx.y;
    if (i >= f.nx || j >= f.ny) return;
    const bool edge = i == 0 || i + 1 == f.nx || j == 0 || j + 1 == f.ny;
    int I, J;
    double wx, wy;
    cell(i, c.nx, f.dx, c.dx, I, wx);
    cell(j, c.ny, f.dy, c.dy, J, wy);
    const long long cxy = (long long)c.nx * c.ny, fxy = (long long)f.nx * f.ny;
    const int kb = blockIdx.z * zc, ke = min(f.nz, kb + zc);
    for (int k = kb; k < ke; ++k) {
        double r = 0.0;
        if (!edge && k > 0 && k + 1 < f.nz) {
            int K;
            double wz;
            cell(k, c.nz, f.dz, c.dz, K, wz);
            const double* e0 = e + K * cxy + (long long)J * c.nx + I;
            const double p0 = bilinear(e0, c.nx, wx, wy), p1 = bilinear(e0 + cxy, c.nx, wx, wy);
            r = (1.0 - wz) * p0 + wz * p1;
        }
        out[k * fxy + (long long)j * f.nx + i] = r;
    }
}

// Coarsest level, fixed faces: `sweeps` red-black SOR sweeps (relaxation omega) from zero in one block's shared
// memory.  A thread keeps its K points per colour and their sources in registers: a half
// sweep is six reads, a handful of FP64 operations and a barrier (it was integer divisions, an FP64
// division and a global read per point: 32 us for 9^3, 7 here).
template <int K>
__device__ void sor_block(const Grid& g, const double* src, double s, double* e, int sweeps, double omega, double* x) {
    const int n = (int)g.N, nt = blockDim.x, sxy = g.nx * g.ny;
    for (int p = threadIdx.x; p < n; p += nt) x[p] = 0.0;
    const double den = 2.0 * (g.ix2 + g.iy2 + g.iz2), inv = 1.0 / den;
    const int half = (g.nx - 1) / 2, cols = half * (g.ny - 2), total = cols * (g.nz - 2);
    int at[2][K];
    double b[2][K];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int q = 0; q < K; ++q) {
            const int t = threadIdx.x + q * nt;
            at[c][q] = -1;
            b[c][q] = 0.0;
            if (t >= total) continue;
            const int k = 1 + t / cols, r = t % cols, j = 1 + r / half;
            const int i = 1 + 2 * (r % half) + ((1 + j + k + c) & 1);
            if (i > g.nx - 2) continue;
            at[c][q] = (k * g.ny + j) * g.nx + i;
            b[c][q] = s * __ldcg(src + at[c][q]);
        }
    __syncthreads();
    for (int it = 0; it < sweeps; ++it)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
            for (int q = 0; q < K; ++q) {
                const int p = at[c][q];
                if (p < 0) continue;
                const double nb = fma(g.iz2, x[p - sxy] + x[p + sxy],
                                      fma(g.iy2, x[p - g.nx] + x[p + g.nx], g.ix2 * (x[p - 1] + x[p + 1])));
                const double old = x[p];
                x[p] = fma(omega, fma(nb + b[c][q], inv, -old), old);
            }
            __syncthreads();
        }
    for (int p = threadIdx.x; p < n; p += nt) e[p] = x[p];
}

template <int K>
__global__ void __launch_bounds__(1024) mg_coarsest_sor_kernel(Grid g, const double* __restrict__ src, double s,
                                                               double* __restrict__ e, int sweeps, double omega) {
    extern __shared__ double sm[];
    sor_block<K>(g, src, s, e, sweeps, omega, sm);
}

// Doubles of shared memory that jacobi_block uses: two iterates with a border of zeros.
__host__ __device__ inline int jacobi_block_doubles(const Grid& g) { return 2 * (g.nx + 2) * (g.ny + 2) * (g.nz + 2); }

// Coarsest level by Jacobi sweeps from zero in one block; fixed faces (open 0) or none.  A thread
// keeps its K points' sources in registers; the border of zeros stands for the outside.  With a shift
// the sweeps converge well before their number is up: from the first one that changes nothing
// all further ones would repeat it, and the block stops.
template <int K>
__device__ void jacobi_block(const Grid& g, int open, const double* src, double s, const ExactDiv& d, double* e, int sweeps,
                             double* sm) {
    const int n = (int)g.N, nt = blockDim.x, sxy = g.nx * g.ny;
    const int wx = g.nx + 2, wxy = wx * (g.ny + 2), half = wxy * (g.nz + 2);
    for (int p = threadIdx.x; p < 2 * half; p += nt) sm[p] = 0.0;
    double b[K];
    int at[K];
    bool live[K];
#pragma unroll
    for (int q = 0; q < K; ++q) {
        const int p = threadIdx.x + q * nt;
        const int k = p / sxy, r = p - k * sxy, j = r / g.nx, i = r - j * g.nx;
        const bool face = i == 0 || i == g.nx - 1 || j == 0 || j == g.ny - 1 || k == 0 || k == g.nz - 1;
        live[q] = p < n && (open || !face);
        at[q] = p < n ? (k + 1) * wxy + (j + 1) * wx + i + 1 : wxy + wx + 1;
        b[q] = p < n ? __ldcg(src + p) : 0.0;
    }
    __syncthreads();
    int it = 0;
    for (bool moved = true; it < sweeps && moved; ++it) {
        const double* u = sm + (it & 1 ? half : 0);
        double* o = sm + (it & 1 ? 0 : half);
        bool change = false, bad = d.general;
        double num[K], r[K];
#pragma unroll
        for (int q = 0; q < K; ++q) {
            const double* c = u + at[q];
            double nb = g.ix2 * c[-1];
            nb = fma(g.ix2, c[1], nb);
            nb = fma(g.iy2, c[-wx], nb);
            nb = fma(g.iy2, c[wx], nb);
            nb = fma(g.iz2, c[-wxy], nb);
            nb = fma(g.iz2, c[wxy], nb);
            num[q] = fma(s, b[q], nb);
            bool t;
            r[q] = divide_fast(num[q], d, t);
            bad |= t && live[q];
        }
        if (bad)
#pragma unroll
            for (int q = 0; q < K; ++q) r[q] = divide(num[q], d);
#pragma unroll
        for (int q = 0; q < K; ++q)
            if (live[q]) {
                change |= r[q] != u[at[q]];
                o[at[q]] = r[q];
            }
        moved = __syncthreads_or(change);
    }
    const double* u = sm + (it & 1 ? half : 0);
#pragma unroll
    for (int q = 0; q < K; ++q)
        if (threadIdx.x + q * nt < n) e[threadIdx.x + q * nt] = u[at[q]];
}

template <int K>
__global__ void __launch_bounds__(1024) mg_coarsest_jacobi_kernel(Grid g, int open, long long ld,
                                                                  const double* __restrict__ src,
                                                                  const int* __restrict__ map, double s,
                                                                  const double* __restrict__ shift,
                                                                  double* __restrict__ e, int sweeps) {
    extern __shared__ double sm[];
    const int a = blockIdx.x;
    const ExactDiv d = exact_div(2.0 * (g.ix2 + g.iy2 + g.iz2) + (shift ? shift[a] : 0.0));
    jacobi_block<K>(g, open, src + (long long)(map ? map[a] : a) * ld, s, d, e + (long long)a * ld, sweeps, sm);
}

// The same for coarsest levels of too many points for that: iterates without a border, neighbours masked.
__global__ void __launch_bounds__(1024) mg_coarsest_wide_kernel(Grid g, int open, long long ld,
                                                                const double* __restrict__ src,
                                                                const int* __restrict__ map, double s,
                                                                const double* __restrict__ shift,
                                                                double* __restrict__ e, int sweeps) {
    extern __shared__ double sm[];
    const int a = blockIdx.x, n = (int)g.N, nt = blockDim.x, sxy = g.nx * g.ny;
    src += (long long)(map ? map[a] : a) * ld;
    e += (long long)a * ld;
    double *x = sm, *y = sm + n;
    const ExactDiv d = exact_div(2.0 * (g.ix2 + g.iy2 + g.iz2) + (shift ? shift[a] : 0.0));
    for (int p = threadIdx.x; p < n; p += nt) x[p] = y[p] = 0.0;
    __syncthreads();
    int it = 0;
    for (bool moved = true; it < sweeps && moved; ++it) {
        const double* u = (it & 1) ? y : x;
        double* o = (it & 1) ? x : y;
        bool change = false;
        for (int p = threadIdx.x; p < n; p += nt) {
            const int k = p / sxy, r = p - k * sxy, j = r / g.nx, i = r - j * g.nx;
            if (!open && (i == 0 || i == g.nx - 1 || j == 0 || j == g.ny - 1 || k == 0 || k == g.nz - 1)) continue;
            double nb = 0.0;
            if (i > 0) nb = fma(g.ix2, u[p - 1], nb);
            if (i + 1 < g.nx) nb = fma(g.ix2, u[p + 1], nb);
            if (j > 0) nb = fma(g.iy2, u[p - g.nx], nb);
            if (j + 1 < g.ny) nb = fma(g.iy2, u[p + g.nx], nb);
            if (k > 0) nb = fma(g.iz2, u[p - sxy], nb);
            if (k + 1 < g.nz) nb = fma(g.iz2, u[p + sxy], nb);
            const double v = divide(fma(s, src[p], nb), d);
            change |= v != u[p];
            o[p] = v;
        }
        moved = __syncthreads_or(change);
    }
    const double* u = (it & 1) ? y : x;
    for (int p = threadIdx.x; p < n; p += nt) e[p] = u[p];
}

// ---------------------------------------------------------------- tables ------------------
struct TableJob {
    Grid f[10], c[10];
    double* w[10];
    int* lo[10];
    double* iw[10];
    int* ic[10];
};
__global__ void __launch_bounds__(256) mg_tables_kernel(const __grid_constant__ TableJob J) {
    const int q = blockIdx.x;
    const Grid &f = J.f[q], &c = J.c[q];
    const int nc = c.nx + c.ny + c.nz, nf = f.nx + f.ny + f.nz;
    for (int p = threadIdx.x; p < nc; p += 256) {
        const int ax = p < c.nx ? 0 : p < c.nx + c.ny ? 1 : 2;
        const int C = p - (ax == 0 ? 0 : ax == 1 ? c.nx : c.nx + c.ny);
        double t[5];
        J.lo[q][p] = hat(C, ax == 0 ? f.dx : ax == 1 ? f.dy : f.dz, ax == 0 ? c.dx : ax == 1 ? c.dy : c.dz,
                         ax == 0 ? f.nx : ax == 1 ? f.ny : f.nz, t);
#pragma unroll
        for (int k = 0; k < 5; ++k) J.w[q][5 * p + k] = t[k];
    }
    for (int p = threadIdx.x; p < nf; p += 256) {
        const int ax = p < f.nx ? 0 : p < f.nx + f.ny ? 1 : 2;
        const int C = p - (ax == 0 ? 0 : ax == 1 ? f.nx : f.nx + f.ny);
        cell(C, ax == 0 ? c.nx : ax == 1 ? c.ny : c.nz, ax == 0 ? f.dx : ax == 1 ? f.dy : f.dz,
             ax == 0 ? c.dx : ax == 1 ? c.dy : c.dz, J.ic[q][p], J.iw[q][p]);
    }
}

// ---------------------------------------------------------------- tile passes --------------
// ZERO: the pre-smoothings start from zero (the first is pointwise), else from v.  The iterate after
// them goes to vout.
template <bool ZERO>
__global__ void __launch_bounds__(MT)
    mg_down_kernel(Grid f, Grid c, MGTable T, int open, double s, const double* __restrict__ shift,
                   const double* __restrict__ src, const int* __restrict__ map, long long f_ld,
                   const double* __restrict__ v, double* __restrict__ vout, double* __restrict__ csrc, long long c_ld,
                   MGHistory* hist) {
    __shared__ double tw[DX + DY + DZ][5];
    __shared__ int tl[DX + DY + DZ];
    __shared__ double S[SX * SY * SZ];                        // the first smoothing
    __shared__ double V[VX * VY * VZ];                        // the second smoothing
    __shared__ double R[ZERO ? RX * RY * RZ : UX * UY * UZ];  // the residual (before: v)
    double* A = S;                 // DX x RY x RZ, over S once S is done with
    double* B = A + DX * RY * RZ;  // DX x DY x RZ
    const int tid = threadIdx.x, a = blockIdx.y;
    const int ntx = (c.nx + DX - 1) / DX, nty = (c.ny + DY - 1) / DY;
    const int I0 = (blockIdx.x % ntx) * DX, J0 = (blockIdx.x / ntx % nty) * DY, K0 = (blockIdx.x / (ntx * nty)) * DZ;
    if (hist && blockIdx.x == 0 && a == 0 && tid == 0) hist->r[++hist->count & 63] = 0;
    const int cy = c.nx, cz = c.nx + c.ny;  // the axes' places in the tables
    // first residual point; this tile's own fine points: from its first coarse point to the next tile's
    const int rx = T.lo[I0], ry = T.lo[cy + J0], rz = T.lo[cz + K0];
    // (the point after the first with weight on one side only: half way through the five)
    const int x0 = I0 == 0 ? 0 : rx + 1, y0 = J0 == 0 ? 0 : ry + 1, z0 = K0 == 0 ? 0 : rz + 1;
    const int x1 = I0 + DX < c.nx ? T.lo[I0 + DX] + 1 : f.nx;
    const int y1 = J0 + DY < c.ny ? T.lo[cy + J0 + DY] + 1 : f.ny;
    const int z1 = K0 + DZ < c.nz ? T.lo[cz + K0 + DZ] + 1 : f.nz;
    const Box box(f, open);
    const int sxy = f.nx * f.ny;
    const ExactDiv d = exact_div(2.0 * (f.ix2 + f.iy2 + f.iz2) + (shift ? shift[a] : 0.0));
    const double k1 = MG_OMEGA * s;
    const double* q = src + (long long)(map ? map[a] : a) * f_ld;
    if (tid < 5 * (DX + DY + DZ)) {
        const int e = tid / 5, k = tid - 5 * e;
        const int C = e < DX ? I0 + e : e < DX + DY ? J0 + e - DX : K0 + e - DX - DY;
        const int n = e < DX ? c.nx : e < DX + DY ? c.ny : c.nz;
        const int at = (e < DX ? 0 : e < DX + DY ? cy : cz) + min(C, n - 1);
        tw[e][k] = C < n ? T.w[5 * at + k] : 0.0;
        if (k == 0) tl[e] = T.lo[at] - (e < DX ? rx : e < DX + DY ? ry : rz);
    }
    if (ZERO) {
#pragma unroll
        for (int p = tid; p < SX * SY * SZ; p += MT) {
            int x, y, z;
            split<SX, SY>(p, x, y, z);
            x += rx - 2, y += ry - 2, z += rz - 2;
            S[p] = box.unknown(x, y, z) ? divide(k1 * __ldg(q + z * sxy + y * f.nx + x), d) : 0.0;
        }
    } else {
        const double* vi = v + (long long)a * f_ld;
#pragma unroll
        for (int p = tid; p < UX * UY * UZ; p += MT) {
            int x, y, z;
            split<UX, UY>(p, x, y, z);
            x += rx - 3, y += ry - 3, z += rz - 3;
            R[p] = box.in(x, y, z) ? __ldg(vi + z * sxy + y * f.nx + x) : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int p = tid; p < SX * SY * SZ; p += MT) {
            int x, y, z;
            split<SX, SY>(p, x, y, z);
            const int ui = ((z + 1) * UY + y + 1) * UX + x + 1;
            x += rx - 2, y += ry - 2, z += rz - 2;
            double r = R[ui];
            if (box.unknown(x, y, z))
                r = smoothed(r, neighbours<UX, UX * UY>(f, R, ui), s, __ldg(q + z * sxy + y * f.nx + x), d);
            S[p] = r;
        }
    }
    __syncthreads();
    double* o = vout + (long long)a * f_ld;
#pragma unroll
    for (int p = tid; p < VX * VY * VZ; p += MT) {
        int x, y, z;
        split<VX, VY>(p, x, y, z);
        const int si = ((z + 1) * SY + y + 1) * SX + x + 1;
        x += rx - 1, y += ry - 1, z += rz - 1;
        double r = S[si];
        if (box.unknown(x, y, z))
            r = smoothed(r, neighbours<SX, SX * SY>(f, S, si), s, __ldg(q + z * sxy + y * f.nx + x), d);
        V[p] = r;
        if (x >= x0 && x < x1 && y >= y0 && y < y1 && z >= z0 && z < z1) o[z * sxy + y * f.nx + x] = r;
    }
    __syncthreads();
#pragma unroll
    for (int p = tid; p < RX * RY * RZ; p += MT) {
        int x, y, z;
        split<RX, RY>(p, x, y, z);
        const int vi = ((z + 1) * VY + y + 1) * VX + x + 1;
        x += rx, y += ry, z += rz;
        double r = 0.0;
        if (box.unknown(x, y, z))
            r = residual(V[vi], neighbours<VX, VX * VY>(f, V, vi), s, __ldg(q + z * sxy + y * f.nx + x), d);
        R[p] = r;
    }
    __syncthreads();
    // one axis after the other, each rounded to its own values
    auto taps = [](const double* from, int stride, const double* w) {
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < 5; ++k)
            if (w[k] > 0.0) t = fma(w[k], from[k * stride], t);
        return t;
    };
    for (int p = tid; p < DX * RY * RZ; p += MT) {
        const int x = p & (DX - 1), row = p / DX;
        A[p] = taps(R + row * RX + tl[x], 1, tw[x]) * (f.dx / c.dx);
    }
    __syncthreads();
    for (int p = tid; p < DX * DY * RZ; p += MT) {
        const int x = p & (DX - 1), y = p / DX % DY, z = p / (DX * DY);
        B[p] = taps(A + (z * RY + tl[DX + y]) * DX + x, DX, tw[DX + y]) * (f.dy / c.dy);
    }
    __syncthreads();
    if (tid < DX * DY * DZ) {
        const int x = tid & (DX - 1), y = tid / DX % DY, z = tid / (DX * DY);
        const int I = I0 + x, J = J0 + y, K = K0 + z;
        if (I < c.nx && J < c.ny && K < c.nz)
            csrc[(long long)a * c_ld + ((long long)K * c.ny + J) * c.nx + I] =
                taps(B + (tl[DX + DY + z] * DY + y) * DX + x, DX * DY, tw[DX + DY + z]) * (f.dz / c.dz);
    }
}

// out = v + P e, smoothed twice, on a tile of FX x FY x FZ points
__global__ void __launch_bounds__(MT)
    mg_up_kernel(Grid f, Grid c, MGTable T, int open, double s, const double* __restrict__ shift,
                 const double* __restrict__ src, const int* __restrict__ map, long long f_ld,
                 const double* __restrict__ v, const double* __restrict__ e, long long c_ld, double* __restrict__ out) {
    constexpr int PX = FX + 4, PY = FY + 4, PZ = FZ + 4;  // interpolated points
    constexpr int QX = FX + 2, QY = FY + 2, QZ = FZ + 2;  // first smoothing
    __shared__ double P[PX * PY * PZ];
    __shared__ double Q[QX * QY * QZ];
    const int tid = threadIdx.x, a = blockIdx.y;
    const int ntx = (f.nx + FX - 1) / FX, nty = (f.ny + FY - 1) / FY;
    const int x0 = (blockIdx.x % ntx) * FX, y0 = (blockIdx.x / ntx % nty) * FY, z0 = (blockIdx.x / (ntx * nty)) * FZ;
    const Box box(f, open);
    const int sxy = f.nx * f.ny, cxy = c.nx * c.ny;
    const ExactDiv d = exact_div(2.0 * (f.ix2 + f.iy2 + f.iz2) + (shift ? shift[a] : 0.0));
    const double* q = src + (long long)(map ? map[a] : a) * f_ld;
    const double* vi = v + (long long)a * f_ld;
    const double* ei = e + (long long)a * c_ld;
    double* o = out + (long long)a * f_ld;
#pragma unroll
    for (int p = tid; p < PX * PY * PZ; p += MT) {
        int x, y, z;
        split<PX, PY>(p, x, y, z);
        x += x0 - 2, y += y0 - 2, z += z0 - 2;
        double r = 0.0;
        if (box.in(x, y, z)) {
            r = __ldg(vi + z * sxy + y * f.nx + x);
            if (box.unknown(x, y, z)) {
                const int fy = f.nx + y, fz = f.nx + f.ny + z;
                const double* e0 = ei + (__ldg(T.ic + fz) * c.ny + __ldg(T.ic + fy)) * c.nx + __ldg(T.ic + x);
                const double wx = __ldg(T.iw + x), wy = __ldg(T.iw + fy), wz = __ldg(T.iw + fz);
                const double p0 = bilinear(e0, c.nx, wx, wy), p1 = bilinear(e0 + cxy, c.nx, wx, wy);
                r += (1.0 - wz) * p0 + wz * p1;
            }
        }
        P[p] = r;
    }
    __syncthreads();
    if (tid < QX * QY * QZ) {
        int x, y, z;
        split<QX, QY>(tid, x, y, z);
        const int pi = ((z + 1) * PY + y + 1) * PX + x + 1;
        x += x0 - 1, y += y0 - 1, z += z0 - 1;
        double r = P[pi];
        if (box.unknown(x, y, z))
            r = smoothed(r, neighbours<PX, PX * PY>(f, P, pi), s, __ldg(q + z * sxy + y * f.nx + x), d);
        Q[tid] = r;
    }
    __syncthreads();
    if (tid < FX * FY * FZ) {
        int x, y, z;
        split<FX, FY>(tid, x, y, z);
        const int qi = ((z + 1) * QY + y + 1) * QX + x + 1;
        x += x0, y += y0, z += z0;
        if (box.in(x, y, z)) {
            const int gi = z * sxy + y * f.nx + x;
            double r = Q[qi];
            if (box.unknown(x, y, z)) r = smoothed(r, neighbours<QX, QX * QY>(f, Q, qi), s, __ldg(q + gi), d);
            o[gi] = r;
        }
    }
}
static_assert((FX + 2) * (FY + 2) * (FZ + 2) <= MT, "one point per thread");

Grid half_grid(const Grid& g) {
    dft_grid d{coarse_points(g.nx), coarse_points(g.ny), coarse_points(g.nz), g.xmin, g.xmax, g.ymin,
               g.ymax,          g.zmin,          g.zmax};
    return make_grid(&d);
}

// blocks of a column pass over nb fields, and its z chunk
struct Columns {
    dim3 grid, block;
    int zc, nzc;
};
Columns columns(dft_context* ctx, const Grid& g, int nb) {
    const int bx = (g.nx + CBX - 1) / CBX, by = (g.ny + CBY - 1) / CBY;
    int zc = 32;  // at least the planes that a thread keeps in flight
    while (zc > 4 && (long long)bx * by * nb * ((g.nz + zc - 1) / zc) < 4LL * ctx->num_sms) zc >>= 1;
    while ((long long)nb * ((g.nz + zc - 1) / zc) > 65535) zc *= 2;
    const int nzc = (g.nz + zc - 1) / zc;
    return {dim3(bx, by, nb * nzc), dim3(CBX, CBY), zc, nzc};
}

template <int MODE>
void column(dft_context* ctx, const MGLevel& f, const double* src, const int* map, const double* v, double* out,
            int open, double s, const double* shift, int nb, MGHistory* hist = nullptr) {
    const Columns c = columns(ctx, f.g, nb);
    mg_column_kernel<MODE><<<c.grid, c.block, 0, ctx->stream>>>(f.g, open, s, shift, src, map, f.ld, v, out, c.zc, c.nzc,
                                                                hist);
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
}

void restrict_fields(dft_context* ctx, const MGLevel& l, const Grid& c, long long c_ld, const double* r, double* csrc,
                     int nb) {
    const Grid& f = l.g;
    const long long f_ld = l.ld;
    const int nzb = (c.nz + CZ - 1) / CZ, fields = std::max(1, 65535 / nzb);
    for (int a0 = 0; a0 < nb; a0 += fields) {
        const dim3 grid((c.nx + CX - 1) / CX, (c.ny + CY - 1) / CY, nzb * std::min(fields, nb - a0));
        mg_restrict_kernel<<<grid, 256, 0, ctx->stream>>>(f, c, l.table, r + (long long)a0 * f_ld, f_ld,
                                                          csrc + (long long)a0 * c_ld, c_ld, nzb);
        DFT_LAUNCH_CHECK();
        count_launch(ctx);
    }
}

// Optimal SOR relaxation for the 7-point operator on grid g (from the Jacobi spectral radius
// of the Dirichlet problem) and the sweeps that cut the error by 1e-4.
void sor_parameters(const Grid& g, double* omega, int* sweeps) {
    const double pi = 3.14159265358979323846;
    const double rj = (g.ix2 * std::cos(pi / (g.nx - 1)) + g.iy2 * std::cos(pi / (g.ny - 1)) +
                       g.iz2 * std::cos(pi / (g.nz - 1))) /
                      (g.ix2 + g.iy2 + g.iz2);
    *omega = 2.0 / (1.0 + std::sqrt(std::max(0.0, 1.0 - rj * rj)));
    const double rate = std::max(*omega - 1.0, 1e-3);
    const int need = (int)std::ceil(std::log(1e-4) / std::log(rate));
    *sweeps = std::min(8 * std::max({g.nx, g.ny, g.nz}), std::max(4, need));
}

template <int K>
void coarsest_sor_launch(dft_context* ctx, const MGLevel& l, const double* src, double s, int sweeps, double omega,
                         int threads) {
    const size_t smem = sizeof(double) * (size_t)l.g.N;
    DFT_CUDA(cudaFuncSetAttribute(mg_coarsest_sor_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(sizeof(double) * MG_COARSEST_MAX)));
    mg_coarsest_sor_kernel<K><<<1, threads, smem, ctx->stream>>>(l.g, src, s, l.v, sweeps, omega);
}

// l.v = the coarsest level's solution for s src
void coarsest(dft_context* ctx, const MGLevel& l, const double* src, const int* map, int open, double s,
              const double* shift, int nb, bool sor) {
    const Grid& g = l.g;
    if (sor) {
        double omega;
        int sweeps;
        sor_parameters(g, &omega, &sweeps);
        const int total = (g.nx - 1) / 2 * (g.ny - 2) * (g.nz - 2);
        const int threads = std::max(32, std::min(1024, (total + 31) / 32 * 32));
        const int k = (total + threads - 1) / threads;
        if (k <= 1) coarsest_sor_launch<1>(ctx, l, src, s, sweeps, omega, threads);
        else if (k <= 2) coarsest_sor_launch<2>(ctx, l, src, s, sweeps, omega, threads);
        else coarsest_sor_launch<6>(ctx, l, src, s, sweeps, omega, threads);
    } else {
        const int sweeps = 8 * std::max({g.nx, g.ny, g.nz});
        // three points a thread: independent chains, and a barrier of few warps (9^3: 8)
        const int threads = (int)std::min<long long>(1024, (g.N + 95) / 96 * 32);
        if (g.N <= 3LL * threads) {
            const size_t smem = sizeof(double) * jacobi_block_doubles(g);  // 197 KB for 2 x 2 x 768 points
            DFT_CUDA(cudaFuncSetAttribute(mg_coarsest_jacobi_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          200 * 1024));
            mg_coarsest_jacobi_kernel<3><<<nb, threads, smem, ctx->stream>>>(g, open, l.ld, src, map, s, shift, l.v,
                                                                             sweeps);
        } else {
            DFT_CUDA(cudaFuncSetAttribute(mg_coarsest_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)(sizeof(double) * 2 * MG_COARSEST_MAX)));
            mg_coarsest_wide_kernel<<<nb, 1024, sizeof(double) * 2 * (size_t)g.N, ctx->stream>>>(
                g, open, l.ld, src, map, s, shift, l.v, sweeps);
        }
    }
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
}

inline unsigned down_tiles(const Grid& c) {
    return (unsigned)(((c.nx + DX - 1) / DX) * ((c.ny + DY - 1) / DY) * ((c.nz + DZ - 1) / DZ));
}
inline unsigned up_tiles(const Grid& f) {
    return (unsigned)(((f.nx + FX - 1) / FX) * ((f.ny + FY - 1) / FY) * ((f.nz + FZ - 1) / FZ));
}

// v == nullptr: pre-smoothings from zero
void down(dft_context* ctx, const MGLevel& f, const MGLevel& c, const double* src, const int* map, const double* v,
          double* vout, int open, double s, const double* shift, int nb, MGHistory* hist) {
    for (int a0 = 0; a0 < nb; a0 += 65535) {
        const dim3 grid(down_tiles(c.g), std::min(nb - a0, 65535));
        const long long off = (long long)a0 * f.ld;
        const double *q = map ? src : src + off, *h = shift ? shift + a0 : nullptr;
        const int* m = map ? map + a0 : nullptr;
        double* e = c.src + (long long)a0 * c.ld;
        if (v)
            mg_down_kernel<false><<<grid, MT, 0, ctx->stream>>>(f.g, c.g, f.table, open, s, h, q, m, f.ld, v + off,
                                                                vout + off, e, c.ld, hist);
        else
            mg_down_kernel<true><<<grid, MT, 0, ctx->stream>>>(f.g, c.g, f.table, open, s, h, q, m, f.ld, nullptr,
                                                               vout + off, e, c.ld, hist);
        DFT_LAUNCH_CHECK();
        count_launch(ctx);
    }
}

void up(dft_context* ctx, const MGLevel& f, const MGLevel& c, const double* src, const int* map, const double* v,
        double* out, int open, double s, const double* shift, int nb) {
    for (int a0 = 0; a0 < nb; a0 += 65535) {
        const int n = std::min(nb - a0, 65535);
        const long long off = (long long)a0 * f.ld;
        mg_up_kernel<<<dim3(up_tiles(f.g), n), MT, 0, ctx->stream>>>(
            f.g, c.g, f.table, open, s, shift ? shift + a0 : nullptr, map ? src : src + off, map ? map + a0 : nullptr,
            f.ld, v + off, c.v + (long long)a0 * c.ld, c.ld, out + off);
        DFT_LAUNCH_CHECK();
        count_launch(ctx);
    }
}

}  // namespace

void mg_coarsest_solve(dft_context* ctx, const MGLevel& l, const double* src, bool sor) {
    coarsest(ctx, l, src, nullptr, 0, 1.0, nullptr, 1, sor);
}

std::vector<MGLevel> mg_levels(const Grid& fine) {
    std::vector<MGLevel> L;
    MGLevel f{};
    f.g = fine;
    f.ld = fine.N;
    L.push_back(f);
    Grid cur = fine;
    while (cur.N > MG_COARSEST_MAX || std::min({cur.nx, cur.ny, cur.nz}) > 9) {
        const Grid c = half_grid(cur);
        if (c.nx == cur.nx && c.ny == cur.ny && c.nz == cur.nz) break;
        MGLevel l{};
        l.g = c;
        l.ld = c.N;
        L.push_back(l);
        cur = c;
        if (L.size() >= 10) break;
    }
    return L;
}

void mg_restrict(dft_context* ctx, const MGLevel& f, const Grid& c, const double* in, double* out) {
    restrict_fields(ctx, f, c, c.N, in, out, 1);
}

size_t mg_table_doubles(const std::vector<MGLevel>& L) {
    size_t n = 0;
    for (size_t i = 0; i + 1 < L.size(); ++i) {
        const Grid &f = L[i].g, &c = L[i + 1].g;
        n += 6 * (size_t)(c.nx + c.ny + c.nz) + 2 * (size_t)(f.nx + f.ny + f.nz) + 4;
    }
    return n;
}

void mg_tables(dft_context* ctx, std::vector<MGLevel>& L, double* slab) {
    TableJob J{};
    int jobs = 0;
    for (size_t i = 0; i + 1 < L.size(); ++i) {
        const Grid &f = L[i].g, &c = L[i + 1].g;
        const int nc = c.nx + c.ny + c.nz, nf = f.nx + f.ny + f.nz;
        J.f[jobs] = f;
        J.c[jobs] = c;
        J.w[jobs] = slab;
        J.lo[jobs] = (int*)(slab + 5 * nc);
        J.iw[jobs] = slab + 6 * nc;
        J.ic[jobs] = (int*)(slab + 6 * nc + nf);
        L[i].table = {J.w[jobs], J.lo[jobs], J.iw[jobs], J.ic[jobs]};
        slab += 6 * nc + 2 * nf + 4;
        if (++jobs < 10 && i + 2 < L.size()) continue;
        mg_tables_kernel<<<jobs, 256, 0, ctx->stream>>>(J);
        DFT_LAUNCH_CHECK();
        count_launch(ctx);
        jobs = 0;
    }
}

void mg_cycle(dft_context* ctx, std::vector<MGLevel>& L, size_t i, const double* src, const int* map, const double* from,
              int open, double s, const double* shift, int nb, bool sor, MGHistory* hist) {
    MGLevel& l = L[i];
    if (i + 1 == L.size()) {
        if (hist) mg_start_cycle(ctx, hist);
        coarsest(ctx, l, src, map, open, s, shift, nb, sor);
        if (hist) mg_residual_max(ctx, l.g, src, s, l.v, hist);
        return;
    }
    MGLevel& c = L[i + 1];
    // flat grids, whose coarse spacing may be the finer one along an axis, stream: the tiles count on
    // coarse points being 1 to 2 fine spacings apart
    const bool tiles = l.g.N * nb <= MG_TILE_MAX && c.g.dx >= l.g.dx && c.g.dy >= l.g.dy && c.g.dz >= l.g.dz;
    if (tiles) {
        down(ctx, l, c, src, map, from, l.tmp, open, s, shift, nb, hist);
        mg_cycle(ctx, L, i + 1, c.src, nullptr, nullptr, open, 1.0, shift, nb, sor, nullptr);
        up(ctx, l, c, src, map, l.tmp, l.v, open, s, shift, nb);
        if (hist) mg_residual_max(ctx, l.g, src, s, l.v, hist);
        return;
    }
    if (from) {
        column<SMOOTH>(ctx, l, src, map, from, l.tmp, open, s, shift, nb);
        column<SMOOTH>(ctx, l, src, map, l.tmp, l.v, open, s, shift, nb);
    } else {
        column<ZERO_TWICE>(ctx, l, src, map, nullptr, l.v, open, s, shift, nb);
    }
    column<RESIDUAL>(ctx, l, src, map, l.v, l.tmp, open, s, shift, nb, hist);
    restrict_fields(ctx, l, c.g, c.ld, l.tmp, c.src, nb);
    mg_cycle(ctx, L, i + 1, c.src, nullptr, nullptr, open, 1.0, shift, nb, sor, nullptr);
    const Columns q = columns(ctx, l.g, nb);
    mg_correct_kernel<<<q.grid, q.block, 0, ctx->stream>>>(l.g, c.g, l.table, open, l.ld, c.v, c.ld, l.v, q.zc, q.nzc);
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
    column<SMOOTH>(ctx, l, src, map, l.v, l.tmp, open, s, shift, nb);
    column<SMOOTH>(ctx, l, src, map, l.tmp, l.v, open, s, shift, nb);
    if (hist) mg_residual_max(ctx, l.g, src, s, l.v, hist);
}

void mg_start_cycle(dft_context* ctx, MGHistory* hist) {
    mg_start_cycle_kernel<<<1, 1, 0, ctx->stream>>>(hist);
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
}

void mg_interpolate(dft_context* ctx, const Grid& f, const Grid& c, const double* e, double* out) {
    const Columns q = columns(ctx, f, 1);
    mg_interpolate_kernel<<<q.grid, q.block, 0, ctx->stream>>>(f, c, e, out, q.zc);
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
}

void mg_residual_max(dft_context* ctx, const Grid& g, const double* src, double s, const double* v, MGHistory* hist) {
    const Columns q = columns(ctx, g, 1);
    mg_residual_max_kernel<<<q.grid, q.block, 0, ctx->stream>>>(g, s, src, v, hist, q.zc);
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
}

}  // namespace dftb
