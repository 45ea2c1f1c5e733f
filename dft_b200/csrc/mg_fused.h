// Multigrid passes shared by the Poisson cycles (poisson_start.cu) and the eigensolver's
// preconditioner (precond_mg.cu): weighted-Jacobi V(2,2) on nested grids with the same bounds.
//
// Per level the equation is d v_p - sum_nb w v_nb = s src_p with d = 2 (ix2 + iy2 + iz2) + shift_a and
// w = 1/h^2, for nb fields a at once.  open = 0: the faces are fixed (their residual is zero).
// open = 1: every point is an unknown, neighbours outside the box are zero.
#pragma once

#include <vector>

#include "ops.h"

namespace dftb {

constexpr double MG_OMEGA = 0.8;
constexpr int MG_COARSEST_MAX = 12288;  // most points of the coarsest level

// Per axis point of the next coarser level, x then y then z: five restriction weights from fine point
// lo on; per axis point of this level: interpolation weight and cell.
struct MGTable {
    const double* w;
    const int* lo;
    const double* iw;
    const int* ic;
};

struct MGLevel {
    Grid g;
    long long ld;           // field stride of this level's arrays
    double *src, *v, *tmp;  // coarse levels: right-hand side, iterate, scratch
    MGTable table;          // towards the next coarser level
};

// The nested grids from g down to the coarsest (array pointers unset, ld = N).
std::vector<MGLevel> mg_levels(const Grid& g);

// Residual maxima of a solve's cycles: cycle c (from 1) puts its own into r[c % 64], as the bits of a
// non-negative double.
struct MGHistory {
    unsigned long long r[64];
    unsigned long long count;
};

// One V(2,2) cycle at level i: L[i].v = cycle(from) for the right-hand side s src, from zero when
// from == nullptr (from is kept; it must not be L[i].v or L[i].tmp).  map: field a reads row map[a]
// of src.  sor: the coarsest level (fixed faces, one field) by red-black SOR instead of Jacobi sweeps.
// hist: when given, its next cycle's word is the maximum over the unknowns of |s src - (d v - sum w v)|
// after the cycle (one field).
void mg_cycle(dft_context* ctx, std::vector<MGLevel>& L, size_t i, const double* src, const int* map, const double* from,
              int open, double s, const double* shift, int nb, bool sor, MGHistory* hist);
// out = R(in): the restriction alone (transposed trilinear weights; needs f.table)
void mg_restrict(dft_context* ctx, const MGLevel& f, const Grid& c, const double* in, double* out);
// The levels' transfer tables into slab (mg_table_doubles), one launch.
size_t mg_table_doubles(const std::vector<MGLevel>& L);
void mg_tables(dft_context* ctx, std::vector<MGLevel>& L, double* slab);
// out = P e on the interior, 0 on the faces
void mg_interpolate(dft_context* ctx, const Grid& f, const Grid& c, const double* e, double* out);
// starts the next cycle's word of hist by itself
void mg_start_cycle(dft_context* ctx, MGHistory* hist);
// the current word of hist = max |s src - (d v - sum w v)| over the interior
void mg_residual_max(dft_context* ctx, const Grid& g, const double* src, double s, const double* v, MGHistory* hist);
// l.v = the coarsest level's solution for src by red-black SOR, or by Jacobi sweeps
void mg_coarsest_solve(dft_context* ctx, const MGLevel& l, const double* src, bool sor);

}  // namespace dftb
