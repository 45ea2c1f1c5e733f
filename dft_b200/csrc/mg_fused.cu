// Fused multigrid passes (mg_fused.h).
//
// The separate passes of a cycle (two smoothings, residual, three restriction passes, interpolation, two
// smoothings) are bound by launches on the coarse levels (3.5 us each on grids of 33^3 and below) and by index
// arithmetic and L2 traffic on the fine ones.  Here a level costs two launches:
//   down  both pre-smoothings from zero, the residual and its restriction, in shared memory on a tile
//         of 8 x 4 x 4 coarse points and the fine points it needs (the halo is recomputed);
//   up    interpolation and both post-smoothings on a tile of 16 x 8 x 8 fine points.
// Recomputing costs about 2.8 times the smoothing work, so levels above MG_FUSED_MAX points take the
// smoothings one by one (a z march that streams) and fuse residual with restriction and interpolation
// with the first post-smoothing only.  Break-even on B200 (modelled from 1,060 cycles per 1,024 points for the
// short tile passes, 5,700 for the long ones and 2.5 us per launch) is near 600,000 points.
// Measured, poisson start + cycles + stop at 128^3: MGF_BEFORE -> MGF_AFTER ms.
//
// Divisions by the diagonal are multiplications by its reciprocal: a smoother's rounding does not
// move the fixed point.
#include <algorithm>
#include <cmath>

#include "mg_fused.h"
#include "neural.h"

namespace dftb {

namespace {

constexpr long long MG_FUSED_MAX = 600000;
constexpr int CX = 8, CY = 4, CZ = 4;                 // coarse points of a down tile
// residual points that 8 (4) coarse points at most 2 fine spacings apart draw on: the open
// interval of (8 + 1) (4 + 1) coarse spacings holds at most 18 (10)
constexpr int RX = 18, RY = 10, RZ = 10;
constexpr int VX = RX + 2, VY = RY + 2, VZ = RZ + 2;  // with the neighbours of the residual
constexpr int SX = VX + 2, SY = VY + 2, SZ = VZ + 2;  // with the neighbours of the second smoothing
constexpr int FX = 16, FY = 8, FZ = 8;                // fine points of an up tile
constexpr int MT = 256;

// p < n of a box of W x H columns: its coordinates
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

template <int W, int WH>
__device__ __forceinline__ double neighbours(const Grid& g, const double* a, int i) {
    return fma(g.iz2, a[i - WH] + a[i + WH], fma(g.iy2, a[i - W] + a[i + W], g.ix2 * (a[i - 1] + a[i + 1])));
}

// coarse point index -> first fine point that a tile starting there owns
__device__ __forceinline__ int first_fine(int I, int nc, int nf, double h, double H) {
    return I >= nc ? nf : min(nf, (int)ceil(I * H / h));
}

// FROM 0: the iterate v is given; 1: it is the second smoothing from zero, also written to vout;
// 2: src is the residual itself.
template <int FROM>
__global__ void __launch_bounds__(MT, FROM == 1 ? 3 : 4)
    mg_down_kernel(Grid f, Grid c, int open, double s, const double* __restrict__ shift,
                   const double* __restrict__ src, const int* __restrict__ map, long long f_ld,
                   const double* __restrict__ v, double* __restrict__ vout, double* __restrict__ csrc, long long c_ld,
                   MGHistory* hist) {
    extern __shared__ double sm[];
    __shared__ double tw[3][CX][4];  // restriction weights of each coarse point per axis
    __shared__ int ts[3][CX];        // and the first residual point they apply to
    double* V = sm;                                  // VX x VY x VZ (not FROM 2)
    double* R = FROM == 2 ? sm : V + VX * VY * VZ;   // RX x RY x RZ
    double* S = R + RX * RY * RZ;                    // SX x SY x SZ (FROM 1)
    double* A = S;                                   // CX x RY x RZ, over S once S is done with
    double* B = A + CX * RY * RZ;                    // CX x CY x RZ
    const int tid = threadIdx.x, a = blockIdx.y;
    const int ntx = (c.nx + CX - 1) / CX, nty = (c.ny + CY - 1) / CY;
    const int I0 = (blockIdx.x % ntx) * CX, J0 = (blockIdx.x / ntx % nty) * CY, K0 = (blockIdx.x / (ntx * nty)) * CZ;
    if (hist && blockIdx.x == 0 && a == 0 && tid == 0) hist->r[++hist->count & 63] = 0;
    // first residual point: strictly above (I0 - 1) H
    const int rx = (int)floor((I0 - 1) * c.dx / f.dx) + 1, ry = (int)floor((J0 - 1) * c.dy / f.dy) + 1,
              rz = (int)floor((K0 - 1) * c.dz / f.dz) + 1;
    const Box box(f, open);
    const int sxy = f.nx * f.ny;
    const double d = 2.0 * (f.ix2 + f.iy2 + f.iz2) + (shift ? shift[a] : 0.0);
    const double* q = src + (long long)(map ? map[a] : a) * f_ld;
    if (tid < CX + CY + CZ) {
        const int ax = tid < CX ? 0 : tid < CX + CY ? 1 : 2, t = tid - (ax == 0 ? 0 : ax == 1 ? CX : CX + CY);
        const int I = (ax == 0 ? I0 : ax == 1 ? J0 : K0) + t, r0 = ax == 0 ? rx : ax == 1 ? ry : rz;
        const double h = ax == 0 ? f.dx : ax == 1 ? f.dy : f.dz, H = ax == 0 ? c.dx : ax == 1 ? c.dy : c.dz;
        const int nf = ax == 0 ? f.nx : ax == 1 ? f.ny : f.nz, len = ax == 0 ? RX : ax == 1 ? RY : RZ;
        const double X = I * H;
        const int st = max(0, min(len - 4, (int)floor((X - H) / h) + 1 - r0));
        ts[ax][t] = st;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = r0 + st + k;
            const double w = 1.0 - fabs(i * h - X) / H;
            tw[ax][t][k] = i >= 0 && i < nf && w > 0.0 ? w : 0.0;
        }
    }
    if (FROM == 1) {
#pragma unroll 4
        for (int p = tid; p < SX * SY * SZ; p += MT) {
            int x, y, z;
            split<SX, SY>(p, x, y, z);
            x += rx - 2, y += ry - 2, z += rz - 2;
            S[p] = box.unknown(x, y, z) ? __ldg(q + (long long)z * sxy + y * f.nx + x) : 0.0;
        }
        __syncthreads();
        // this tile's own fine points
        const int x0 = first_fine(I0, c.nx, f.nx, f.dx, c.dx), x1 = first_fine(I0 + CX, c.nx, f.nx, f.dx, c.dx);
        const int y0 = first_fine(J0, c.ny, f.ny, f.dy, c.dy), y1 = first_fine(J0 + CY, c.ny, f.ny, f.dy, c.dy);
        const int z0 = first_fine(K0, c.nz, f.nz, f.dz, c.dz), z1 = first_fine(K0 + CZ, c.nz, f.nz, f.dz, c.dz);
        const double wd = MG_OMEGA / d, k1 = wd * s;
        double* o = vout + (long long)a * f_ld;
        for (int p = tid; p < VX * VY * VZ; p += MT) {
            int x, y, z;
            split<VX, VY>(p, x, y, z);
            const int si = ((z + 1) * SY + y + 1) * SX + x + 1;
            x += rx - 1, y += ry - 1, z += rz - 1;
            double r = 0.0;
            if (box.unknown(x, y, z)) {
                const double v1 = k1 * S[si];
                r = fma(wd, fma(k1, neighbours<SX, SX * SY>(f, S, si), fma(s, S[si], -d * v1)), v1);
            }
            V[p] = r;
            if (x >= x0 && x < x1 && y >= y0 && y < y1 && z >= z0 && z < z1) o[(long long)z * sxy + y * f.nx + x] = r;
        }
        __syncthreads();
    } else if (FROM == 0) {
        const double* vi = v + (long long)a * f_ld;
#pragma unroll 4
        for (int p = tid; p < VX * VY * VZ; p += MT) {
            int x, y, z;
            split<VX, VY>(p, x, y, z);
            x += rx - 1, y += ry - 1, z += rz - 1;
            V[p] = box.in(x, y, z) ? __ldg(vi + (long long)z * sxy + y * f.nx + x) : 0.0;
        }
        __syncthreads();
    }
#pragma unroll 2
    for (int p = tid; p < RX * RY * RZ; p += MT) {
        int x, y, z;
        split<RX, RY>(p, x, y, z);
        const int vi = ((z + 1) * VY + y + 1) * VX + x + 1, si = ((z + 2) * SY + y + 2) * SX + x + 2;
        x += rx, y += ry, z += rz;
        double r = 0.0;
        if (FROM == 2) {
            if (box.in(x, y, z)) r = __ldg(q + (long long)z * sxy + y * f.nx + x);
        } else if (box.unknown(x, y, z)) {
            const double b = FROM == 1 ? S[si] : __ldg(q + (long long)z * sxy + y * f.nx + x);
            r = fma(s, b, neighbours<VX, VX * VY>(f, V, vi) - d * V[vi]);
        }
        R[p] = r;
    }
    __syncthreads();
    for (int p = tid; p < CX * RY * RZ; p += MT) {
        const int x = p & (CX - 1), row = p / CX;
        const double* r = R + row * RX + ts[0][x];
        A[p] = tw[0][x][0] * r[0] + tw[0][x][1] * r[1] + tw[0][x][2] * r[2] + tw[0][x][3] * r[3];
    }
    __syncthreads();
    for (int p = tid; p < CX * CY * RZ; p += MT) {
        const int x = p & (CX - 1), y = p / CX % CY, z = p / (CX * CY);
        const double* r = A + (z * RY + ts[1][y]) * CX + x;
        B[p] = tw[1][y][0] * r[0] + tw[1][y][1] * r[CX] + tw[1][y][2] * r[2 * CX] + tw[1][y][3] * r[3 * CX];
    }
    __syncthreads();
    if (tid < CX * CY * CZ) {
        const int x = tid & (CX - 1), y = tid / CX % CY, z = tid / (CX * CY);
        const int I = I0 + x, J = J0 + y, K = K0 + z;
        if (I < c.nx && J < c.ny && K < c.nz) {
            const double* r = B + (ts[2][z] * CY + y) * CX + x;
            const double t = tw[2][z][0] * r[0] + tw[2][z][1] * r[CX * CY] + tw[2][z][2] * r[2 * CX * CY] +
                             tw[2][z][3] * r[3 * CX * CY];
            csrc[(long long)a * c_ld + ((long long)K * c.ny + J) * c.nx + I] =
                t * ((f.dx / c.dx) * (f.dy / c.dy) * (f.dz / c.dz));
        }
    }
}

// One cell and weight of the trilinear interpolation along an axis.
__device__ __forceinline__ void cell(int i, int nc, double h, double H, int& I, double& w) {
    const double u = i * h / H;
    I = min(max((int)floor(u), 0), nc - 2);
    w = fmin(fmax(u - I, 0.0), 1.0);
}

// out = v + P e, smoothed NS times (1 or 2), on a tile of FX x FY x FZ points
template <int NS>
__global__ void __launch_bounds__(MT, 4)
    mg_up_kernel(Grid f, Grid c, int open, double s, const double* __restrict__ shift, const double* __restrict__ src,
                 const int* __restrict__ map, long long f_ld, const double* __restrict__ v,
                 const double* __restrict__ e, long long c_ld, double* __restrict__ out) {
    constexpr int PX = FX + 2 * NS, PY = FY + 2 * NS, PZ = FZ + 2 * NS;  // interpolated points
    constexpr int QX = FX + 2, QY = FY + 2, QZ = FZ + 2;                 // first smoothing (NS 2)
    __shared__ double P[PX * PY * PZ];
    __shared__ double Q[NS == 2 ? QX * QY * QZ : 1];
    __shared__ double wt[3][PX];
    __shared__ int ci[3][PX];
    const int tid = threadIdx.x, a = blockIdx.y;
    const int ntx = (f.nx + FX - 1) / FX, nty = (f.ny + FY - 1) / FY;
    const int x0 = (blockIdx.x % ntx) * FX, y0 = (blockIdx.x / ntx % nty) * FY, z0 = (blockIdx.x / (ntx * nty)) * FZ;
    const Box box(f, open);
    const int sxy = f.nx * f.ny, cxy = c.nx * c.ny;
    const double d = 2.0 * (f.ix2 + f.iy2 + f.iz2) + (shift ? shift[a] : 0.0), wd = MG_OMEGA / d;
    const double* q = src + (long long)(map ? map[a] : a) * f_ld;
    const double* vi = v + (long long)a * f_ld;
    const double* ei = e + (long long)a * c_ld;
    double* o = out + (long long)a * f_ld;
    if (tid < PX + PY + PZ) {
        const int ax = tid < PX ? 0 : tid < PX + PY ? 1 : 2, t = tid - (ax == 0 ? 0 : ax == 1 ? PX : PX + PY);
        const int i = (ax == 0 ? x0 : ax == 1 ? y0 : z0) + t - NS;
        cell(i, ax == 0 ? c.nx : ax == 1 ? c.ny : c.nz, ax == 0 ? f.dx : ax == 1 ? f.dy : f.dz,
             ax == 0 ? c.dx : ax == 1 ? c.dy : c.dz, ci[ax][t], wt[ax][t]);
    }
    __syncthreads();
#pragma unroll 2
    for (int p = tid; p < PX * PY * PZ; p += MT) {
        int x, y, z;
        split<PX, PY>(p, x, y, z);
        const int gx = x0 + x - NS, gy = y0 + y - NS, gz = z0 + z - NS;
        double r = 0.0;
        if (box.in(gx, gy, gz)) {
            r = __ldg(vi + (long long)gz * sxy + gy * f.nx + gx);
            if (box.unknown(gx, gy, gz)) {
                const double* e0 = ei + (long long)ci[2][z] * cxy + ci[1][y] * c.nx + ci[0][x];
                const double* e1 = e0 + cxy;
                const double wx = wt[0][x], wy = wt[1][y], wz = wt[2][z];
                const double a0 = fma(wx, __ldg(e0 + 1) - __ldg(e0), __ldg(e0));
                const double a1 = fma(wx, __ldg(e0 + c.nx + 1) - __ldg(e0 + c.nx), __ldg(e0 + c.nx));
                const double b0 = fma(wx, __ldg(e1 + 1) - __ldg(e1), __ldg(e1));
                const double b1 = fma(wx, __ldg(e1 + c.nx + 1) - __ldg(e1 + c.nx), __ldg(e1 + c.nx));
                const double p0 = fma(wy, a1 - a0, a0), p1 = fma(wy, b1 - b0, b0);
                r += fma(wz, p1 - p0, p0);
            }
        }
        P[p] = r;
    }
    __syncthreads();
    if (NS == 2) {
#pragma unroll 2
        for (int p = tid; p < QX * QY * QZ; p += MT) {
            int x, y, z;
            split<QX, QY>(p, x, y, z);
            const int pi = ((z + 1) * PY + y + 1) * PX + x + 1;
            x += x0 - 1, y += y0 - 1, z += z0 - 1;
            double r = P[pi];
            if (box.unknown(x, y, z))
                r = fma(wd, fma(s, __ldg(q + (long long)z * sxy + y * f.nx + x),
                                neighbours<PX, PX * PY>(f, P, pi) - d * r), r);
            Q[p] = r;
        }
        __syncthreads();
    }
#pragma unroll 2
    for (int p = tid; p < FX * FY * FZ; p += MT) {
        int x, y, z;
        split<FX, FY>(p, x, y, z);
        const int pi = ((z + 1) * (NS == 2 ? QY : PY) + y + 1) * (NS == 2 ? QX : PX) + x + 1;
        x += x0, y += y0, z += z0;
        if (!box.in(x, y, z)) continue;
        const long long gi = (long long)z * sxy + y * f.nx + x;
        double r = NS == 2 ? Q[pi] : P[pi];
        if (box.unknown(x, y, z)) {
            const double nb = NS == 2 ? neighbours<QX, QX * QY>(f, Q, pi) : neighbours<PX, PX * PY>(f, P, pi);
            r = fma(wd, fma(s, __ldg(q + gi), nb - d * r), r);
        }
        o[gi] = r;
    }
}

// Streaming passes: one thread per (x, y) column and z chunk.  blockIdx.z = field * nzc + chunk.
constexpr int CBX = 32, CBY = 8;

// ZERO: both smoothings from zero in one pass (the first is pointwise); else one smoothing from v
template <bool ZERO>
__global__ void __launch_bounds__(CBX* CBY)
    mg_column_kernel(Grid f, int open, double s, const double* __restrict__ shift, const double* __restrict__ src,
                     const int* __restrict__ map, long long ld, const double* __restrict__ v, double* __restrict__ out,
                     int zc, int nzc) {
    const int i = blockIdx.x * CBX + threadIdx.x, j = blockIdx.y * CBY + threadIdx.y;
    const int a = blockIdx.z / nzc, kc = blockIdx.z - a * nzc;
    if (i >= f.nx || j >= f.ny) return;
    const double d = 2.0 * (f.ix2 + f.iy2 + f.iz2) + (shift ? shift[a] : 0.0), wd = MG_OMEGA / d, k1 = wd * s;
    const double* __restrict__ q = src + (long long)(map ? map[a] : a) * ld;
    const double* __restrict__ u = ZERO ? q : v + (long long)a * ld;  // the field whose neighbours are read
    double* __restrict__ o = out + (long long)a * ld;
    const int lo = open ? 0 : 1, sxy = f.nx * f.ny;
    const bool col = i >= lo && i < f.nx - lo && j >= lo && j < f.ny - lo;
    // ZERO: values of fixed points count as zero, whatever src holds there
    const int z0 = ZERO ? lo : 0, z1 = ZERO ? f.nz - lo : f.nz, e0 = ZERO ? lo : 0;
    const bool xl = i > e0, xr = i + 1 < f.nx - e0, yl = j > e0, yr = j + 1 < f.ny - e0;
    const int kb = kc * zc, ke = min(f.nz, kb + zc);
    long long p = (long long)kb * sxy + (long long)j * f.nx + i;
    const bool live = !ZERO || col;
    auto at = [&](int k, long long pp) { return live && k >= z0 && k < z1 ? __ldg(u + pp) : 0.0; };
    double below = at(kb - 1, p - sxy), cur = at(kb, p);
    for (int k = kb; k < ke; ++k, p += sxy) {
        const double above = at(k + 1, p + sxy);
        double r = ZERO ? 0.0 : cur;
        if (col && k >= lo && k < f.nz - lo) {
            const double x = (xl ? __ldg(u + p - 1) : 0.0) + (xr ? __ldg(u + p + 1) : 0.0);
            const double y = (yl ? __ldg(u + p - f.nx) : 0.0) + (yr ? __ldg(u + p + f.nx) : 0.0);
            const double nb = fma(f.iz2, below + above, fma(f.iy2, y, f.ix2 * x));
            if (ZERO) {
                const double v1 = k1 * cur;
                r = fma(wd, fma(k1, nb, fma(s, cur, -d * v1)), v1);
            } else {
                r = fma(wd, fma(s, __ldg(q + p), nb - d * cur), cur);
            }
        }
        o[p] = r;
        below = cur;
        cur = above;
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
            const double* e1 = e0 + cxy;
            const double p0 = (1.0 - wy) * ((1.0 - wx) * __ldg(e0) + wx * __ldg(e0 + 1)) +
                              wy * ((1.0 - wx) * __ldg(e0 + c.nx) + wx * __ldg(e0 + c.nx + 1));
            const double p1 = (1.0 - wy) * ((1.0 - wx) * __ldg(e1) + wx * __ldg(e1 + 1)) +
                              wy * ((1.0 - wx) * __ldg(e1 + c.nx) + wx * __ldg(e1 + c.nx + 1));
            r = (1.0 - wz) * p0 + wz * p1;
        }
        out[k * fxy + (long long)j * f.nx + i] = r;
    }
}

// Coarsest level, fixed faces: `sweeps` red-black SOR sweeps (relaxation omega) from zero in one block's shared
// memory.  A thread keeps its K points per colour and their sources in registers: a half
// sweep is six reads, a handful of FP64 operations and a barrier (it was integer divisions, an FP64
// division and a global read per point: 32 us for 9^3, MGC_US here).
template <int K>
__global__ void __launch_bounds__(1024) mg_coarsest_sor_kernel(Grid g, const double* __restrict__ src,
                                                               double* __restrict__ e, int sweeps, double omega) {
    extern __shared__ double x[];
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
            b[c][q] = src[at[c][q]];
        }
    __syncthreads();
    for (int s = 0; s < sweeps; ++s)
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

// Coarsest level by Jacobi sweeps from zero, one block per field; fixed faces (open 0) or none.
// A thread keeps its K points' sources and neighbour masks in registers.  A sweep shrinks the error
// by at least rho = (d - shift) / d: sweeps past rho^k < 1e-18 change nothing and are not run.
template <int K>
__global__ void __launch_bounds__(1024) mg_coarsest_jacobi_kernel(Grid g, int open, long long ld,
                                                                  const double* __restrict__ src,
                                                                  const int* __restrict__ map, double s,
                                                                  const double* __restrict__ shift,
                                                                  double* __restrict__ e, int sweeps) {
    extern __shared__ double sm[];
    const int a = blockIdx.x, n = (int)g.N, nt = blockDim.x, sxy = g.nx * g.ny;
    src += (long long)(map ? map[a] : a) * ld;
    e += (long long)a * ld;
    double *x = sm, *y = sm + n;
    const double off = 2.0 * (g.ix2 + g.iy2 + g.iz2), d = off + (shift ? shift[a] : 0.0), inv = 1.0 / d;
    if (d > off) sweeps = min(sweeps, 1 + (int)ceil(-41.5 / log(off / d)));
    double b[K];
    unsigned mask[K];  // neighbours x-, x+, y-, y+, z-, z+ inside the box; bit 6: an unknown
#pragma unroll
    for (int q = 0; q < K; ++q) {
        const int p = threadIdx.x + q * nt;
        mask[q] = 0;
        b[q] = 0.0;
        if (p >= n) continue;
        const int k = p / sxy, r = p - k * sxy, j = r / g.nx, i = r - j * g.nx;
        const bool face = i == 0 || i == g.nx - 1 || j == 0 || j == g.ny - 1 || k == 0 || k == g.nz - 1;
        mask[q] = (i > 0) | (i + 1 < g.nx) << 1 | (j > 0) << 2 | (j + 1 < g.ny) << 3 | (k > 0) << 4 |
                  (k + 1 < g.nz) << 5 | (open || !face) << 6;
        b[q] = s * src[p];
        x[p] = y[p] = 0.0;
    }
    __syncthreads();
    for (int it = 0; it < sweeps; ++it) {
        const double* u = (it & 1) ? y : x;
        double* o = (it & 1) ? x : y;
#pragma unroll
        for (int q = 0; q < K; ++q) {
            const int p = threadIdx.x + q * nt;
            const unsigned m = mask[q];
            if (!(m & 64)) continue;
            const double vx = (m & 1 ? u[p - 1] : 0.0) + (m & 2 ? u[p + 1] : 0.0);
            const double vy = (m & 4 ? u[p - g.nx] : 0.0) + (m & 8 ? u[p + g.nx] : 0.0);
            const double vz = (m & 16 ? u[p - sxy] : 0.0) + (m & 32 ? u[p + sxy] : 0.0);
            o[p] = (fma(g.iz2, vz, fma(g.iy2, vy, g.ix2 * vx)) + b[q]) * inv;
        }
        __syncthreads();
    }
    const double* u = (sweeps & 1) ? y : x;
    for (int p = threadIdx.x; p < n; p += nt) e[p] = u[p];
}

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
    int zc = 32;
    while (zc > 4 && (long long)bx * by * nb * ((g.nz + zc - 1) / zc) < 8LL * ctx->num_sms) zc >>= 1;
    while ((long long)nb * ((g.nz + zc - 1) / zc) > 65535) zc *= 2;
    const int nzc = (g.nz + zc - 1) / zc;
    return {dim3(bx, by, nb * nzc), dim3(CBX, CBY), zc, nzc};
}

inline unsigned down_tiles(const Grid& c) {
    return (unsigned)(((c.nx + CX - 1) / CX) * ((c.ny + CY - 1) / CY) * ((c.nz + CZ - 1) / CZ));
}
inline unsigned up_tiles(const Grid& f) {
    return (unsigned)(((f.nx + FX - 1) / FX) * ((f.ny + FY - 1) / FY) * ((f.nz + FZ - 1) / FZ));
}

template <int FROM>
void down(dft_context* ctx, const Grid& f, long long f_ld, const Grid& c, long long c_ld, const double* src,
          const int* map, const double* v, double* vout, double* csrc, int open, double s, const double* shift, int nb,
          MGHistory* hist) {
    constexpr int V = FROM == 2 ? 0 : VX * VY * VZ, R = RX * RY * RZ;
    constexpr int S = FROM == 1 ? SX * SY * SZ : CX * RY * RZ + CX * CY * RZ;
    constexpr size_t smem = sizeof(double) * (V + R + S);
    if (smem > 40 * 1024)
        DFT_CUDA(cudaFuncSetAttribute(mg_down_kernel<FROM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    for (int a0 = 0; a0 < nb; a0 += 65535) {
        const int n = std::min(nb - a0, 65535);
        const long long off = (long long)a0 * f_ld;
        mg_down_kernel<FROM><<<dim3(down_tiles(c), n), MT, smem, ctx->stream>>>(
            f, c, open, s, shift ? shift + a0 : nullptr, map ? src : src + off, map ? map + a0 : nullptr, f_ld,
            v ? v + off : nullptr, vout ? vout + off : nullptr, csrc + (long long)a0 * c_ld, c_ld, hist);
        DFT_LAUNCH_CHECK();
        count_launch(ctx);
    }
}

template <int NS>
void up(dft_context* ctx, const MGLevel& f, const MGLevel& c, const double* src, const int* map, const double* v,
        double* out, int open, double s, const double* shift, int nb) {
    for (int a0 = 0; a0 < nb; a0 += 65535) {
        const int n = std::min(nb - a0, 65535);
        const long long off = (long long)a0 * f.ld;
        mg_up_kernel<NS><<<dim3(up_tiles(f.g), n), MT, 0, ctx->stream>>>(
            f.g, c.g, open, s, shift ? shift + a0 : nullptr, map ? src : src + off, map ? map + a0 : nullptr, f.ld,
            v + off, c.v + (long long)a0 * c.ld, c.ld, out + off);
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
void coarsest_jacobi_launch(dft_context* ctx, const MGLevel& l, const double* src, const int* map, int open, double s,
                            const double* shift, int nb, int sweeps, int threads) {
    const size_t smem = sizeof(double) * 2 * (size_t)l.g.N;
    DFT_CUDA(cudaFuncSetAttribute(mg_coarsest_jacobi_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(sizeof(double) * 2 * MG_COARSEST_MAX)));
    mg_coarsest_jacobi_kernel<K><<<nb, threads, smem, ctx->stream>>>(l.g, open, l.ld, src, map, s, shift, l.v, sweeps);
}

template <int K>
void coarsest_sor_launch(dft_context* ctx, const MGLevel& l, const double* src, int sweeps, double omega, int threads) {
    const size_t smem = sizeof(double) * (size_t)l.g.N;
    DFT_CUDA(cudaFuncSetAttribute(mg_coarsest_sor_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(sizeof(double) * MG_COARSEST_MAX)));
    mg_coarsest_sor_kernel<K><<<1, threads, smem, ctx->stream>>>(l.g, src, l.v, sweeps, omega);
}

// l.v = the coarsest level's solution for src (scale 1)
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
        if (k <= 1) coarsest_sor_launch<1>(ctx, l, src, sweeps, omega, threads);
        else if (k <= 2) coarsest_sor_launch<2>(ctx, l, src, sweeps, omega, threads);
        else coarsest_sor_launch<6>(ctx, l, src, sweeps, omega, threads);
    } else {
        const int sweeps = 8 * std::max({g.nx, g.ny, g.nz});
        const int threads = (int)std::min<long long>(1024, (g.N + 31) / 32 * 32);
        const int k = (int)((g.N + threads - 1) / threads);
        if (k <= 1) coarsest_jacobi_launch<1>(ctx, l, src, map, open, s, shift, nb, sweeps, threads);
        else if (k <= 2) coarsest_jacobi_launch<2>(ctx, l, src, map, open, s, shift, nb, sweeps, threads);
        else if (k <= 4) coarsest_jacobi_launch<4>(ctx, l, src, map, open, s, shift, nb, sweeps, threads);
        else coarsest_jacobi_launch<12>(ctx, l, src, map, open, s, shift, nb, sweeps, threads);
    }
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
}

}  // namespace

void mg_coarsest_solve(dft_context* ctx, const MGLevel& l, const double* src, bool sor) {
    coarsest(ctx, l, src, nullptr, 0, 1.0, nullptr, 1, sor);
}

void mg_coarsest_fields(dft_context* ctx, const MGLevel& l, const double* src, const int* map, double s,
                        const double* shift, int nb) {
    coarsest(ctx, l, src, map, 1, s, shift, nb, false);
}

bool mg_fused_level(long long n) { return n <= MG_FUSED_MAX; }

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

void mg_residual_restrict(dft_context* ctx, const MGLevel& f, const MGLevel& c, const double* src, const int* map,
                          const double* v, int open, double s, const double* shift, int nb,
                          MGHistory* hist) {
    down<0>(ctx, f.g, f.ld, c.g, c.ld, src, map, v, nullptr, c.src, open, s, shift, nb, hist);
}

void mg_restrict(dft_context* ctx, const Grid& f, const Grid& c, const double* in, double* out) {
    down<2>(ctx, f, f.N, c, c.N, in, nullptr, nullptr, nullptr, out, 0, 1.0, nullptr, 1, nullptr);
}

void mg_smooth_step(dft_context* ctx, const MGLevel& f, const double* src, const int* map, const double* v, double* out,
                    int open, double s, const double* shift, int nb) {
    const Columns c = columns(ctx, f.g, nb);
    mg_column_kernel<false><<<c.grid, c.block, 0, ctx->stream>>>(f.g, open, s, shift, src, map, f.ld, v, out, c.zc, c.nzc);
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
}

void mg_correct_smooth(dft_context* ctx, const MGLevel& f, const MGLevel& c, const double* src, const int* map,
                       const double* v, double* tmp, double* out, int open, double s, const double* shift, int nb) {
    if (mg_fused_level(f.g.N * nb)) {
        up<2>(ctx, f, c, src, map, v, out, open, s, shift, nb);
        return;
    }
    up<1>(ctx, f, c, src, map, v, tmp, open, s, shift, nb);
    mg_smooth_step(ctx, f, src, map, tmp, out, open, s, shift, nb);
}

void mg_cycle_from_zero(dft_context* ctx, std::vector<MGLevel>& L, size_t i, const double* src, const int* map, int open,
                        double s, const double* shift, int nb, bool sor) {
    MGLevel& l = L[i];
    if (i + 1 == L.size()) {
        coarsest(ctx, l, src, map, open, s, shift, nb, sor);
        return;
    }
    MGLevel& c = L[i + 1];
    const bool fused = mg_fused_level(l.g.N * nb);
    if (fused) {
        // v and tmp change roles, so that the cycle ends in v
        down<1>(ctx, l.g, l.ld, c.g, c.ld, src, map, nullptr, l.tmp, c.src, open, s, shift, nb, nullptr);
    } else {
        const Columns q = columns(ctx, l.g, nb);
        mg_column_kernel<true><<<q.grid, q.block, 0, ctx->stream>>>(l.g, open, s, shift, src, map, l.ld, nullptr, l.v,
                                                                    q.zc, q.nzc);
        DFT_LAUNCH_CHECK();
        count_launch(ctx);
        mg_residual_restrict(ctx, l, c, src, map, l.v, open, s, shift, nb, nullptr);
    }
    mg_cycle_from_zero(ctx, L, i + 1, c.src, nullptr, open, 1.0, shift, nb, sor);
    if (fused) mg_correct_smooth(ctx, l, c, src, map, l.tmp, nullptr, l.v, open, s, shift, nb);
    else mg_correct_smooth(ctx, l, c, src, map, l.v, l.tmp, l.v, open, s, shift, nb);
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
