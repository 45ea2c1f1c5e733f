// Fused multigrid passes shared by the Poisson cycles (poisson_start.cu) and the eigensolver's
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

struct MGLevel {
    Grid g;
    long long ld;                      // field stride of this level's arrays
    double *src, *v, *tmp;             // coarse levels: right-hand side, iterate, scratch
};

// The nested grids from g down to the coarsest (array pointers unset, ld = N).
std::vector<MGLevel> mg_levels(const Grid& g);

// Residual maxima of a solve's cycles: cycle c (from 1) puts its own into r[c % 64], as the bits of a
// non-negative double.
struct MGHistory {
    unsigned long long r[64];
    unsigned long long count;
};

// c.src = R(s src - (d v - sum w v)): residual and restriction (transposed trilinear weights) in one pass.
// hist: when given, starts the next cycle's word there.
void mg_residual_restrict(dft_context* ctx, const MGLevel& f, const MGLevel& c, const double* src, const int* map,
                          const double* v, int open, double s, const double* shift, int nb,
                          MGHistory* hist);
// out = R(in): the restriction alone
void mg_restrict(dft_context* ctx, const Grid& f, const Grid& c, const double* in, double* out);
// out = one weighted-Jacobi step from v
void mg_smooth_step(dft_context* ctx, const MGLevel& f, const double* src, const int* map, const double* v, double* out,
                    int open, double s, const double* shift, int nb);
// One V(2,2) cycle below and at level i from a zero start on every level: L[i].src -> L[i].v (map: field
// a of level i reads row map[a] of src).  Level i's v and tmp may be swapped; the result is in v.
void mg_cycle_from_zero(dft_context* ctx, std::vector<MGLevel>& L, size_t i, const double* src, const int* map, int open,
                        double s, const double* shift, int nb, bool sor);
// v = (v2 + P e) smoothed twice: out, by way of tmp where the level is large (returns with the result
// in out)
void mg_correct_smooth(dft_context* ctx, const MGLevel& f, const MGLevel& c, const double* src, const int* map,
                       const double* v, double* tmp, double* out, int open, double s, const double* shift, int nb);
// out = P e on the interior, 0 on the faces
void mg_interpolate(dft_context* ctx, const Grid& f, const Grid& c, const double* e, double* out);
// starts the next cycle's word of hist by itself
void mg_start_cycle(dft_context* ctx, MGHistory* hist);
// the current word of hist = max |s src - (d v - sum w v)| over the interior
void mg_residual_max(dft_context* ctx, const Grid& g, const double* src, double s, const double* v, MGHistory* hist);
// L.back().v = the coarsest level's solution for its src by red-black SOR, or by Jacobi sweeps
void mg_coarsest_solve(dft_context* ctx, const MGLevel& l, const double* src, bool sor);
// the same by Jacobi sweeps for nb open fields (map, s, shift as above)
void mg_coarsest_fields(dft_context* ctx, const MGLevel& l, const double* src, const int* map, double s,
                        const double* shift, int nb);
// whether a level of n points in all its fields takes the long tile passes
bool mg_fused_level(long long n);

}  // namespace dftb
