// Multigrid preconditioner for the block eigensolver: one V(2,2) cycle from zero for
// (T + sigma_a) t_a = r_a per correction band, T = -1/2 lap_h with psi = 0 outside the box
// (the kinetic operator of applyMolecularKohnShamHamiltonian, KohnShamHamiltonianMolecule.cpp:90-166),
// sigma_a = max(-theta_a, 1 Ha).  All bands advance together: every kernel takes the band
// index from blockIdx.y.  The reference preconditions with the diagonal of H - theta
// (EigenvalueSolverMolecule.cpp:521-555); this is an option of the block solver, not the
// reference's behaviour.
//
// Per level the equation is (den + c_a) t_p - sum_nb w_d t_nb = s * src_p over every grid point
// (neighbours outside the box are zero), with den = 2 (ix2 + iy2 + iz2), w_d = 1/h_d^2,
// c_a = 2 sigma_a and s = 2 on the finest level (the residual r), 1 on coarse levels.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "mg_fused.h"
#include "neural.h"
#include "ops.h"

namespace dftb {
namespace {

// Column kernels march z over a column (i, j) per thread, like the H psi kernel: the z
// neighbours come from registers and no point index is divided.  blockIdx.z = band * nzc + chunk.
constexpr int PX = 32, PY = 8;

// r = s src - ((den + c) v - sum)
__global__ void __launch_bounds__(PX* PY) pc_residual_kernel(Grid g, long long ld, const double* __restrict__ src,
                                                            double s, const double* __restrict__ shift,
                                                            const double* __restrict__ v, double* __restrict__ r,
                                                            int zc, int nzc) {
    const int i = blockIdx.x * PX + threadIdx.x, j = blockIdx.y * PY + threadIdx.y;
    const int a = blockIdx.z / nzc, kc = blockIdx.z - a * nzc;
    if (i >= g.nx || j >= g.ny) return;
    const double d = 2.0 * (g.ix2 + g.iy2 + g.iz2) + shift[a];
    const double* sa = src + (long long)a * ld;
    const double* va = v + (long long)a * ld;
    double* ra = r + (long long)a * ld;
    const long long sxy = (long long)g.nx * g.ny;
    const int kb = kc * zc, ke = min(g.nz, kb + zc);
    long long p = (long long)kb * sxy + (long long)j * g.nx + i;
    const bool xl = i > 0, xr = i + 1 < g.nx, yl = j > 0, yr = j + 1 < g.ny;
    double below = kb > 0 ? va[p - sxy] : 0.0, cur = va[p];
    for (int k = kb; k < ke; ++k, p += sxy) {
        const double above = k + 1 < g.nz ? va[p + sxy] : 0.0;
        double sum = g.iz2 * (below + above);
        if (xl) sum += g.ix2 * va[p - 1];
        if (xr) sum += g.ix2 * va[p + 1];
        if (yl) sum += g.iy2 * va[p - g.nx];
        if (yr) sum += g.iy2 * va[p + g.nx];
        ra[p] = s * sa[p] - (d * cur - sum);
        below = cur;
        cur = above;
    }
}

// launch shape of the column kernels for nb fields: z chunks long enough to amortise the march,
// enough blocks to fill the machine; gridDim.z = nb * nzc must stay below 65536
struct ColShape {
    dim3 grid, block;
    int zc, nzc;
};
ColShape col_shape(dft_context* ctx, const Grid& g, int nb) {
    const int bx = (g.nx + PX - 1) / PX, by = (g.ny + PY - 1) / PY;
    int zc = 32;
    while (zc > 4 && (long long)bx * by * nb * ((g.nz + zc - 1) / zc) < 4LL * ctx->num_sms) zc >>= 1;
    int nzc = (g.nz + zc - 1) / zc;
    while ((long long)nb * nzc > 65535) {
        zc *= 2;
        nzc = (g.nz + zc - 1) / zc;
    }
    return {dim3(bx, by, nb * nzc), dim3(PX, PY), zc, nzc};
}

// shift[a] = c for every field (the screened Poisson equation of the Kerker mixer)
__global__ void pc_fill_kernel(int nb, double c, double* __restrict__ shift) {
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nb; a += gridDim.x * blockDim.x) shift[a] = c;
}

// c_a = 2 max(-theta[src[a]], 1 Ha): the shift of each correction band, from the Ritz values
__global__ void pc_shift_kernel(int nb, const double* __restrict__ theta, const int* __restrict__ src,
                                double* __restrict__ shift) {
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nb; a += gridDim.x * blockDim.x)
        shift[a] = 2.0 * fmax(-theta[src[a]], 1.0);
}

inline dim3 pc_grid(dft_context* ctx, long long n, int nb) {
    long long bx = (n + 255) / 256;
    const long long cap = std::max<long long>(1, (long long)ctx->num_sms * 8 / std::max(nb, 1));
    bx = std::max<long long>(1, std::min(bx, std::max<long long>(cap, 4)));
    return dim3((unsigned)bx, (unsigned)nb);
}

// One V(2,2) cycle from zero, all nb fields together, for (den + shift_a) t - sum_nb w t_nb =
// s * R_{src[a]} on g (src_dev == nullptr: field a itself), into T.  shift_dev must not live in
// the WS_PG2 workspace.
void vcycle_batch(dft_context* ctx, const Grid& g, const double* R, const int* src_dev, int nb, const double* shift,
                  double s, double* T, long long ld) {
    std::vector<MGLevel> L = mg_levels(g);
    if (L.back().g.N > MG_COARSEST_MAX) fail(DFT_INVALID_ARGUMENT, "grid too small or anisotropic for multigrid");
    L[0].ld = ld;
    // slab: per band one fine scratch field, and right-hand side, iterate and scratch per coarse level
    size_t per_band = (size_t)ld + 2;
    for (size_t i = 1; i < L.size(); ++i) per_band += 3 * (size_t)L[i].g.N + 6;
    double* p = (double*)ws_get(ctx, WS_PG2, sizeof(double) * (per_band * nb + 64 + mg_table_doubles(L)));
    mg_tables(ctx, L, p);
    p += (mg_table_doubles(L) + 1) / 2 * 2;
    auto take = [&](size_t n) {
        double* q = p;
        p += (n * nb + 1) / 2 * 2;
        return q;
    };
    L[0].v = T;
    L[0].tmp = take((size_t)ld);
    for (size_t i = 1; i < L.size(); ++i) {
        L[i].src = take((size_t)L[i].g.N);
        L[i].v = take((size_t)L[i].g.N);
        L[i].tmp = take((size_t)L[i].g.N);
    }
    mg_cycle(ctx, L, 0, R, src_dev, nullptr, 1, s, shift, nb, false, nullptr);
}

}  // namespace

void precondition_multigrid(dft_context* ctx, const Grid& g, const double* R, const int* src_dev, int nb,
                            const double* theta_dev, double* T, long long ld) {
    if (nb <= 0) return;
    // shifts c_a = 2 sigma_a, computed on the device (no host round trip)
    double* shift = (double*)ws_get(ctx, WS_PG3, sizeof(double) * (size_t)nb + 64);
    pc_shift_kernel<<<(nb + 127) / 128, 128, 0, ctx->stream>>>(nb, theta_dev, src_dev, shift);
    count_launch(ctx);
    vcycle_batch(ctx, g, R, src_dev, nb, shift, 2.0, T, ld);
}

namespace {
__global__ void pc_sigma_shift_kernel(int nb, const double* __restrict__ sigma, double* __restrict__ shift) {
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nb; a += gridDim.x * blockDim.x) shift[a] = 2.0 * sigma[a];
}
__global__ void pc_add_kernel(long long n, long long ld, const double* __restrict__ e, double* __restrict__ x) {
    const int a = blockIdx.y;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x)
        x[(long long)a * ld + p] += e[(long long)a * ld + p];
}
}  // namespace

void helmholtz_refine(dft_context* ctx, const Grid& g, const double* R, int nb, const double* sigma_dev, double* X,
                      long long ld, int cycles, double* res, double* e) {
    if (nb <= 0) return;
    double* shift = (double*)ws_get(ctx, WS_PG3, sizeof(double) * (size_t)nb + 64);
    pc_sigma_shift_kernel<<<(nb + 127) / 128, 128, 0, ctx->stream>>>(nb, sigma_dev, shift);
    count_launch(ctx);
    vcycle_batch(ctx, g, R, nullptr, nb, shift, 2.0, X, ld);
    for (int c = 1; c < cycles; ++c) {
        // res = 2 R - ((den + 2 sigma) X - sum), the equation's residual in the cycle's scaling
        const ColShape cs = col_shape(ctx, g, nb);
        pc_residual_kernel<<<cs.grid, cs.block, 0, ctx->stream>>>(g, ld, R, 2.0, shift, X, res, cs.zc, cs.nzc);
        count_launch(ctx);
        vcycle_batch(ctx, g, res, nullptr, nb, shift, 1.0, e, ld);
        pc_add_kernel<<<pc_grid(ctx, g.N, nb), 256, 0, ctx->stream>>>(g.N, ld, e, X);
        count_launch(ctx);
        DFT_LAUNCH_CHECK();
    }
}

void screened_poisson_vcycle(dft_context* ctx, const Grid& g, const double* src, int nb, double q2, double* x,
                             long long ld, int cycles) {
    if (nb <= 0) return;
    if (!(q2 > 0.0) || !std::isfinite(q2)) fail(DFT_INVALID_ARGUMENT, "screening q^2 must be > 0");
    if (cycles < 1) fail(DFT_INVALID_ARGUMENT, "cycles must be >= 1");
    double* shift = (double*)ws_get(ctx, WS_PG3, sizeof(double) * (size_t)nb + 64);
    pc_fill_kernel<<<(nb + 127) / 128, 128, 0, ctx->stream>>>(nb, q2, shift);
    count_launch(ctx);
    // a cycle reads its right-hand side while it writes x, and the refinement reads it again: a caller's
    // source that x overlaps is copied first
    const size_t block = (size_t)nb * ld;
    const bool overlap = src < x + block && x < src + block;
    const size_t fields = (cycles > 1 ? 2 : 0) + (overlap ? 1 : 0);
    double* scratch = fields ? (double*)ws_get(ctx, WS_PG4, sizeof(double) * fields * block) : nullptr;
    if (overlap) {
        double* copy = scratch + (fields - 1) * block;
        DFT_CUDA(cudaMemcpyAsync(copy, src, sizeof(double) * (block - ld + g.N), cudaMemcpyDeviceToDevice, ctx->stream));
        src = copy;
    }
    vcycle_batch(ctx, g, src, nullptr, nb, shift, 1.0, x, ld);
    if (cycles == 1) return;
    // iterative refinement: res = src - (-lap + q2) x, e = V-cycle(res), x += e
    double *res = scratch, *e = scratch + block;
    for (int c = 1; c < cycles; ++c) {
        const ColShape cs = col_shape(ctx, g, nb);
        pc_residual_kernel<<<cs.grid, cs.block, 0, ctx->stream>>>(g, ld, src, 1.0, shift, x, res, cs.zc, cs.nzc);
        count_launch(ctx);
        vcycle_batch(ctx, g, res, nullptr, nb, shift, 1.0, e, ld);
        pc_add_kernel<<<pc_grid(ctx, g.N, nb), 256, 0, ctx->stream>>>(g.N, ld, e, x);
        count_launch(ctx);
        DFT_LAUNCH_CHECK();
    }
}

}  // namespace dftb
