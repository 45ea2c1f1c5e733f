// Finite-difference gradients of the XC path (device, inline): shared by the whole-grid XC
// kernels (grid_ops.cu) and the z-slab XC energy (zslab.cu), so both compute the same values.
#pragma once

#include "common.cuh"

namespace dftb {

// Reciprocal spacings of the one-sided and the central differences.
struct XCScale {
    double x1, y1, z1, x2, y2, z2;
};
inline XCScale xc_scale(const Grid& g) {
    return {1.0 / g.dx, 1.0 / g.dy, 1.0 / g.dz, 0.5 / g.dx, 0.5 / g.dy, 0.5 / g.dz};
}

// |grad f|, central differences, one-sided on the faces (calculateCartesianDerivative, reference
// ExchangeCorrelationMolecule.cpp:11-170)
__device__ __forceinline__ double grad_of(const Grid& g, const XCScale& h, const double* __restrict__ f, long long p,
                                          int i, int j, int k) {
    const int s1 = g.nx;
    const long long s2 = (long long)g.nx * g.ny;
    const bool xl = i > 0, xr = i + 1 < g.nx, yl = j > 0, yr = j + 1 < g.ny, zl = k > 0, zr = k + 1 < g.nz;
    const double gx = (f[xr ? p + 1 : p] - f[xl ? p - 1 : p]) * (xl && xr ? h.x2 : h.x1);
    const double gy = (f[yr ? p + s1 : p] - f[yl ? p - s1 : p]) * (yl && yr ? h.y2 : h.y1);
    const double gz = (f[zr ? p + s2 : p] - f[zl ? p - s2 : p]) * (zl && zr ? h.z2 : h.z1);
    return sqrt(gx * gx + gy * gy + gz * gz);
}

}  // namespace dftb
