// Batched radial-atom SCF: every run (atom x functional) is one cluster of a single launch, iterating its
// own SCF loop to convergence (reference solveSelfConsistentField, SelfConsistentField.cpp:539-786)
// while the other runs proceed independently on other SMs.  Per-run arrays (2000 points each)
// stay in L2.
//
// A run has four blocks, two or one, as many as the SMs allow: its orbitals are dealt to them (14 warps
// of FP64 chains on one SM wait for each other's issue slots: a Sturm count 218000 cycles, 145000 with
// one orbital).  Everything else each block does for itself on its own copy, so the blocks meet
// only before and after the orbitals.
//
// Inside a block the work that the reference does point by point runs across threads, and
// each (n,l,spin) orbital is owned by one warp:
//  * eigenvalue: the reference's Sturm bisection (EigenvalueSolver.cpp:94-221) with its
//    midpoints and final interval (find_eigenvalue).
//  * eigenvector: inverse iteration with the shifted Thomas factorisation computed once
//    per orbital (identical to refactoring every solve, NumericalMethods.cpp:85-139).
//  * every sum the reference takes sequentially (norms, dots, trapezoid prefix sums,
//    energies) is taken sequentially by one lane, so rounding follows the reference.
// The file is compiled without FMA contraction.  Remaining differences from the reference
// come from the device's transcendental functions (a few ulp) in XC and the start vectors.
//
// Bound by the latency of the serial chains.  60 atoms, 2000 points: 412 -> 59 ms, with the bits that general
// divisions gave (the chains' own quotients differ from those only next to the middle of two numbers; steps
// from global memory 300 cycles -> shared 73 or less; 13 to 19 rounds of counts -> 3; clusters).
#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <vector>

#include <cooperative_groups.h>

#include "exact_div.cuh"
#include "ops.h"
#include "xc_device.cuh"

namespace dftb {

namespace {

constexpr int RT = 512;        // threads per run
constexpr int RW = RT / 32;    // warps per run
constexpr int MAXORB = 16;     // occupied (n,l,spin) orbitals per run
constexpr double EPS = 1.0e-14;

struct RunSpec {
    int Z, kind, norb;
    double pivot_eps;  // |pivot| below this is singular (EPS unless tuned)
    int n[MAXORB], l[MAXORB], spin[MAXORB], el[MAXORB], idx[MAXORB];
};

// per-run global arrays, each n doubles
enum {
    A_DA = 0, A_DB, A_VA, A_VB, A_VH, A_OA, A_OB, A_RD, A_OD, A_T1, A_T2, A_T3, A_T4, A_ENC, A_SIN,
    A_COUNT
};
// per-orbital arrays
enum { O_U = 0, O_DIAG, O_DW, O_F, O_NX, O_ZH, O_COUNT };

__device__ __forceinline__ double eps_guard(double v) { return fabs(v) < EPS ? copysign(EPS, v == 0.0 ? 1.0 : v) : v; }

// ---------------------------------------------------------------- serial chains -------------
// The reference takes its recurrences and sums point by point, and the SCF stops on differences of a few
// last bits, so the order of every chain stays.  A chain costs the latency of its dependent FP64
// operations (8.5 cycles each): arrays come CH points at a time through the warp's shared memory (read
// straight from global memory a step waited 300 cycles for the L2), the next points' loads are in
// flight meanwhile, and whatever does not depend on the chain (products, divisions by known values)
// is done by all lanes.
constexpr int CH = 128;      // points per stage
constexpr int PL = CH / 32;  // of them per lane
constexpr int SB = CH + 2;   // pitch of a stage's arrays
constexpr int WARP_STAGE = 5 * SB;
constexpr int BT = 16;  // points a chain takes into registers together

__device__ __forceinline__ void take(double (&v)[BT], const double* s) {
#pragma unroll
    for (int j = 0; j < BT; j += 2) {
        const double2 t = *(const double2*)(s + j);
        v[j] = t.x;
        v[j + 1] = t.y;
    }
}
__device__ __forceinline__ void give(double* s, const double (&v)[BT]) {
#pragma unroll
    for (int j = 0; j < BT; j += 2) *(double2*)(s + j) = make_double2(v[j], v[j + 1]);
}

__device__ __forceinline__ double shfl_d(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }

// sum_i term(load(i)) in order; every lane gets it
template <class Load, class Term>
__device__ double seq_sum(int n, double* st, Load load, Term term) {
    const int lane = threadIdx.x & 31;
    decltype(load(0)) v[PL];
#pragma unroll
    for (int j = 0; j < PL; ++j) v[j] = load(min(lane + 32 * j, n - 1));
    double s = 0.0;
    for (int i0 = 0; i0 < n; i0 += CH) {
#pragma unroll
        for (int j = 0; j < PL; ++j) {
            const int i = i0 + lane + 32 * j;
            st[lane + 32 * j] = i < n ? term(i, v[j]) : 0.0;
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < PL; ++j) v[j] = load(min(i0 + CH + lane + 32 * j, n - 1));
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < CH; k += BT) {
                double t[BT];
                take(t, st + k);
#pragma unroll
                for (int j = 0; j < BT; ++j) s += t[j];
            }
        }
        __syncwarp();
    }
    return shfl_d(s, 0);
}
__device__ double seq_dot(int n, double* st, const double* a, const double* b) {
    return seq_sum(
        n, st, [&](int i) { return make_double2(a[i], b[i]); }, [](int, double2 v) { return v.x * v.y; });
}

// out[i] = out[i - 1] + term(i), in order (down: out[i] = out[i + 1] + term(i)); the first term is 0
template <bool DOWN, class Load, class Term>
__device__ void seq_prefix(int n, double* st, double* out, Load load, Term term) {
    const int lane = threadIdx.x & 31;
    const auto place = [&](int i) { return DOWN ? n - 1 - i : i; };
    double s = 0.0;
    decltype(load(0)) v[PL];
#pragma unroll
    for (int j = 0; j < PL; ++j) v[j] = load(place(min(lane + 32 * j, n - 1)));
    for (int i0 = 0; i0 < n; i0 += CH) {
#pragma unroll
        for (int j = 0; j < PL; ++j) {
            const int i = i0 + lane + 32 * j;
            st[lane + 32 * j] = i < n ? term(place(i), v[j]) : 0.0;
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < PL; ++j) v[j] = load(place(min(i0 + CH + lane + 32 * j, n - 1)));
        if (lane == 0) {
#pragma unroll 2
            for (int k = 0; k < CH; k += BT) {
                double t[BT];
                take(t, st + k);
#pragma unroll
                for (int j = 0; j < BT; ++j) t[j] = s = s + t[j];
                give(st + k, t);
            }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < PL; ++j) {
            const int i = i0 + lane + 32 * j;
            if (i < n) out[place(i)] = st[lane + 32 * j];
        }
        __syncwarp();
    }
}

// a / g in seven dependent operations (a general division: 126 cycles, here 65).  One step y0 (1 + e + e^2),
// e = 1 - g y0, of Chebyshev's third-order iteration for 1 / g (Traub, Iterative Methods for the Solution of
// Equations, 1964) on the approximate reciprocal y0 (error below 2^-18) gives y1, and a quotient q1 within two
// units in the last place; the remainder's correction is Markstein's (exact_div.cuh).  y1 is not the
// correctly rounded reciprocal, so neither is every quotient: it is wherever a / g is 2^-50 units or more from the
// middle of two neighbouring numbers, and else one of the two (of 12000 operands made to lie closest, all
// were right).  a and g in [2^-100, 2^100].
__device__ __forceinline__ double quotient(double a, double g) {
    double y0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(g));
    const double e = __fma_rn(-g, y0, 1.0), q0 = __dmul_rn(a, y0);
    const double t = __fma_rn(e, e, e);
    const double y1 = __fma_rn(y0, t, y0), q1 = __fma_rn(q0, t, q0);
    return __fma_rn(__fma_rn(-g, q1, a), y1, q1);
}
constexpr int HI_EPS = 0x3D06849B;                  // high word of EPS = 1e-14
constexpr int HI_TOP = (1023 + 100) << 20;          // of 2^100
__device__ __forceinline__ bool plain_divisor(double g) {  // above EPS and below 2^100: no guard, no special case
    return (unsigned)((__double2hiint(g) & 0x7fffffff) - HI_EPS - 1) < (unsigned)(HI_TOP - HI_EPS - 1);
}

// countEigenvaluesBelow (EigenvalueSolver.cpp:13-92) at one E per lane; off-diagonals all equal.  The
// chain runs on divisions without special cases; a stage in which some pivot needs its guard is
// taken again with it.
// top: a bound of |diag|.
__device__ int sturm_count(int n, const double* __restrict__ diag, double oo, double top, double E, double* st) {
    const int lane = threadIdx.x & 31;
    // no pivot beyond 2^100, as oo / EPS, diag and E are below 2^98
    const bool plain = oo >= 0x1p-100 && oo <= 0x1p50 && top <= 0x1p90 && fabs(E) <= 0x1p90;
    double v[PL];
#pragma unroll
    for (int j = 0; j < PL; ++j) v[j] = diag[min(lane + 32 * j, n - 1)];
    int c = 0;
    double prev = 0.0;
    for (int i0 = 0; i0 < n; i0 += CH) {
        const int m = min(CH, n - i0);
#pragma unroll
        for (int j = 0; j < PL; ++j) st[lane + 32 * j] = v[j];
        __syncwarp();
#pragma unroll
        for (int j = 0; j < PL; ++j) v[j] = diag[min(i0 + CH + lane + 32 * j, n - 1)];
        int k0 = 0;
        if (i0 == 0) {
            prev = st[0] - E;
            if (prev < 0.0) ++c;
            prev = eps_guard(prev);
            k0 = 1;
        }
        bool ok = plain;
        double p = prev;
        int cc = 0;
        if (m == CH && k0 == 0 && plain) {
            unsigned low = 2u * (unsigned)__double2hiint(p);  // the smallest |pivot|, high word
#pragma unroll 1
            for (int k = 0; k < CH; k += BT) {
                double t[BT];
                take(t, st + k);
#pragma unroll
                for (int j = 0; j < BT; ++j) {
                    p = (t[j] - E) - quotient(oo, p);
                    cc += (unsigned)__double2hiint(p) >> 31;
                    low = min(low, 2u * (unsigned)__double2hiint(p));
                }
            }
            ok = low > 2u * HI_EPS;
        } else if (plain) {
            ok = plain_divisor(p);
            for (int k = k0; k < m; ++k) {
                p = (st[k] - E) - quotient(oo, p);
                if (p < 0.0) ++cc;
                ok &= plain_divisor(p);
            }
        }
        if (!ok) {
            p = prev;
            cc = 0;
            for (int k = k0; k < m; ++k) {
                const double piv = (st[k] - E) - oo / p;
                if (piv < 0.0) ++cc;
                p = eps_guard(piv);
            }
        }
        prev = p;
        c += cc;
        __syncwarp();
    }
    return c;
}

__device__ __forceinline__ double interval_tol(double lo, double hi) { return 1.0e-13 * fmax(1.0, fmax(fabs(lo), fabs(hi))); }

// warp-wide: the k-th eigenvalue of the radial Hamiltonian in [lo, hi] (findEigenvalue): the reference's
// bisection with its midpoints and final interval.
//
// The count is monotone in E in IEEE arithmetic, guard included (Demmel, Dhillon and Ren, "On the
// correctness of some bisection-like parallel eigenvalue algorithms in floating point arithmetic",
// Electron. Trans. Numer. Anal. 3, 1995).  So two counts, at a with at most `index` eigenvalues below
// and at b with more, decide every midpoint outside (a, b).  The first round counts at 16 distances on
// each side of a guess (1e-13 times powers of 8, relative); only midpoints inside the bracket found are
// counted, five levels at a time: 31 lanes take those of every possible path, then the warp walks down the
// real one.  From the Rayleigh quotient of the last orbital that is 2 to 6 rounds; counting every level
// took 13.
__device__ bool find_eigenvalue(int n, const double* __restrict__ diag, double oo, double top, int index, double lo,
                                double hi, double guess, double* st, double& out) {
    const int lane = threadIdx.x & 31;
    double below = -INFINITY, above = INFINITY;  // at most index eigenvalues below; more
    {
        const double step = ldexp(1.0e-13 * fmax(1.0, fabs(guess)), 3 * (lane >> 1));
        const double p = lane & 1 ? guess + step : guess - step;
        const int c = sturm_count(n, diag, oo, top, p, st);
        if (c <= index) below = p;
        else above = p;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            below = fmax(below, __shfl_xor_sync(0xffffffffu, below, o));
            above = fmin(above, __shfl_xor_sync(0xffffffffu, above, o));
        }
    }
    if (!(below < above)) below = -INFINITY, above = INFINITY;
    // whether more than index eigenvalues lie below x
    const auto more = [&](double x) { return x > below && (x >= above || sturm_count(n, diag, oo, top, x, st) > index); };
    bool mlo = more(lo), mhi = !more(hi);
    double w = hi - lo;
    for (int e = 0; e < 100 && (mlo || mhi); ++e) {
        w *= 2.0;
        if (mlo) lo -= w;
        if (mhi) hi += w;
        if (mlo) mlo = more(lo);
        if (mhi) mhi = !more(hi);
    }
    if (mlo || mhi) return false;
    int iter = 0;
    bool done = false;
    while (!done && iter < 300) {
        // levels that the bracket decides
        bool open = false;
        while (!done && iter < 300 && !open) {
            const double mid = 0.5 * (lo + hi);
            if (mid <= below) lo = mid;
            else if (mid >= above) hi = mid;
            else open = true;
            if (!open) {
                ++iter;
                if (hi - lo <= interval_tol(lo, hi)) done = true;
            }
        }
        if (done || iter >= 300) break;
        // node t of the speculation tree: replay its path from (lo, hi)
        int path[5], depth = 0;
        for (int t = lane < 31 ? lane : 0; t > 0; t = (t - 1) >> 1) path[depth++] = (t & 1);  // 1 = left child (count <= index)
        double a = lo, b = hi;
        for (int s = depth - 1; s >= 0; --s) {
            const double m = 0.5 * (a + b);
            if (path[s]) a = m;
            else b = m;
        }
        const double nmid = 0.5 * (a + b);
        const int ncount = sturm_count(n, diag, oo, top, nmid, st);
        int t = 0;
        for (int level = 0; level < 5 && !done && iter < 300; ++level) {
            const double mid = shfl_d(nmid, t);
            const int c = __shfl_sync(0xffffffffu, ncount, t);
            if (c <= index) {
                lo = mid;
                t = 2 * t + 1;
            } else {
                hi = mid;
                t = 2 * t + 2;
            }
            ++iter;
            if (hi - lo <= interval_tol(lo, hi)) done = true;
        }
    }
    out = 0.5 * (lo + hi);
    return true;
}

// The shifted Thomas factors (NumericalMethods.cpp:85-139): f_i = off / w_{i-1}, w_i = diag_i - shift - f_i off.
// False when a pivot is below pivot_eps.  zh = 1 / w for the solves.
__device__ bool factor(int n, const double* __restrict__ diag, double off, double top, double shift, double pivot_eps,
                       double* f, double* dw, double* zh, double* st) {
    const int lane = threadIdx.x & 31;
    const bool plain = fabs(off) >= 0x1p-50 && fabs(off) <= 0x1p25 && top <= 0x1p90 && fabs(shift) <= 0x1p90 &&
                       pivot_eps <= EPS;  // as in sturm_count
    double v[PL];
#pragma unroll
    for (int j = 0; j < PL; ++j) v[j] = diag[min(lane + 32 * j, n - 1)];
    double w = 0.0;
    bool bad = false;
    for (int i0 = 0; i0 < n && !bad; i0 += CH) {
        const int m = min(CH, n - i0);
#pragma unroll
        for (int j = 0; j < PL; ++j) st[lane + 32 * j] = v[j] - shift;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < PL; ++j) v[j] = diag[min(i0 + CH + lane + 32 * j, n - 1)];
        if (lane == 0) {
            int k = 0;
            if (i0 == 0) {
                w = st[0];
                st[SB] = 0.0;
                k = 1;
            }
            while (k < m && !bad) {
                if (plain && m - k >= BT && (k & 1) == 0) {
                    // BT steps without special cases; taken one by one below if some pivot is small
                    double t[BT], g[BT], x = w;
                    unsigned low = 0xffffffffu;  // the smallest |pivot|, high word
                    take(t, st + k);
#pragma unroll
                    for (int j = 0; j < BT; ++j) {
                        low = min(low, 2u * (unsigned)__double2hiint(x));
                        g[j] = quotient(off, x);
                        t[j] = x = t[j] - g[j] * off;
                    }
                    if (low > 2u * HI_EPS) {
                        give(st + k, t);
                        give(st + SB + k, g);
                        w = x;
                        k += BT;
                        continue;
                    }
                }
                if (fabs(w) < pivot_eps) {
                    bad = true;
                    break;
                }
                const double g = off / w;
                st[SB + k] = g;
                st[k] = w = st[k] - g * off;
                ++k;
            }
        }
        bad = __shfl_sync(0xffffffffu, (int)bad, 0);
        __syncwarp();
#pragma unroll
        for (int j = 0; j < PL; ++j) {
            const int i = i0 + lane + 32 * j;
            if (i >= n || bad) continue;
            const double d = st[lane + 32 * j];
            f[i] = st[SB + lane + 32 * j];
            dw[i] = d;
            zh[i] = 1.0 / d;
        }
        __syncwarp();
    }
    w = shfl_d(w, 0);
    return !bad && !(fabs(w) < pivot_eps);
}

// x = the solution of the factored system for u: forwards y_i = u_i - f_i y_{i-1}, backwards
// x_i = (y_i - off x_{i+1}) / w_i.  The backward chain is four operations: q0 = y_i/w_i - (off/w_i) x_{i+1} from
// products taken before, the numerator, its remainder and the correction q0 + r / w_i.  q0 is off by
// 2^k units when the difference loses k bits; the result is then the correctly rounded quotient
// wherever that is 2^(k-51) units or more from the middle of two neighbouring numbers, and else one of the two.
// k is at most 24 (more are lost at one point in 2^24): a stage where more are lost, or where something
// leaves the range of the theorem, is divided point by point.
__device__ void solve(int n, const double* u, const double* f, const double* dw, const double* zh, double off, double* x,
                      double* st) {
    const int lane = threadIdx.x & 31;
    double *s0 = st, *s1 = st + SB, *s2 = st + 2 * SB, *s3 = st + 3 * SB, *s4 = st + 4 * SB;
    {
        double a[PL], b[PL];
        auto fetch = [&](int i0) {
#pragma unroll
            for (int j = 0; j < PL; ++j) {
                const int i = min(i0 + lane + 32 * j, n - 1);
                a[j] = u[i];
                b[j] = f[i];
            }
        };
        fetch(0);
        double y = 0.0;
        for (int i0 = 0; i0 < n; i0 += CH) {
#pragma unroll
            for (int j = 0; j < PL; ++j) {
                s0[lane + 32 * j] = a[j];
                s1[lane + 32 * j] = b[j];
            }
            __syncwarp();
            fetch(i0 + CH);
            if (lane == 0) {
                for (int k = 0; k < CH; k += BT) {
                    double p[BT], q[BT];
                    take(p, s0 + k);
                    take(q, s1 + k);
#pragma unroll
                    for (int j = 0; j < BT; ++j) p[j] = y = p[j] - q[j] * y;  // f_0 = 0
                    give(s0 + k, p);
                }
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < PL; ++j)
                if (i0 + lane + 32 * j < n) x[i0 + lane + 32 * j] = s0[lane + 32 * j];
            __syncwarp();
        }
    }
    double a[PL], b[PL], c[PL];
    auto fetch = [&](int i0) {
#pragma unroll
        for (int j = 0; j < PL; ++j) {
            const int i = n - 1 - (i0 + lane + 32 * j);  // the chain runs down
            a[j] = i >= 0 ? x[i] : 0.0;
            b[j] = i >= 0 ? dw[i] : 1.0;
            c[j] = i >= 0 ? zh[i] : 1.0;
        }
    };
    fetch(0);
    double y = -0.0;  // off y = +0, which leaves y_{n-1} as it is
    for (int i0 = 0; i0 < n; i0 += CH) {
        bool ok = true;
        double q[PL];
#pragma unroll
        for (int j = 0; j < PL; ++j) {
            s0[lane + 32 * j] = a[j];
            s1[lane + 32 * j] = b[j];
            s2[lane + 32 * j] = c[j];
            s3[lane + 32 * j] = off * c[j];
            s4[lane + 32 * j] = q[j] = a[j] * c[j];
            ok &= fabs(b[j]) >= 0x1p-100 && fabs(b[j]) <= 0x1p100;
        }
        __syncwarp();
        fetch(i0 + CH);
        if (lane == 0) {
            double t = y;
#pragma unroll 2
            for (int k = 0; k < CH; k += 8) {
                double p[8], w[8], z[8], oz[8], pz[8];
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    const double2 v0 = *(const double2*)(s0 + k + j), v1 = *(const double2*)(s1 + k + j);
                    const double2 v2 = *(const double2*)(s2 + k + j), v3 = *(const double2*)(s3 + k + j);
                    const double2 v4 = *(const double2*)(s4 + k + j);
                    p[j] = v0.x, p[j + 1] = v0.y, w[j] = v1.x, w[j + 1] = v1.y, z[j] = v2.x, z[j + 1] = v2.y;
                    oz[j] = v3.x, oz[j + 1] = v3.y, pz[j] = v4.x, pz[j + 1] = v4.y;
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const double q0 = __fma_rn(-oz[j], t, pz[j]);
                    const double num = p[j] - off * t;
                    t = __fma_rn(__fma_rn(-w[j], q0, num), z[j], q0);
                    oz[j] = t;
                }
#pragma unroll
                for (int j = 0; j < 8; j += 2) *(double2*)(s3 + k + j) = make_double2(oz[j], oz[j + 1]);
            }
            y = t;
        }
        __syncwarp();
        // every quotient between 2^-850 and 2^850 and no less than 2^-24 of the first product
#pragma unroll
        for (int j = 0; j < PL; ++j) {
            const double v = fabs(s3[lane + 32 * j]);
            ok &= i0 + lane + 32 * j >= n || (v >= 0x1p-850 && v <= 0x1p850 && v >= 0x1p-24 * fabs(q[j]));
        }
        if (!__all_sync(0xffffffffu, ok)) {
            if (lane == 0) {
                const int m = min(CH, n - i0);
                double t = i0 == 0 ? -0.0 : s0[CH];
                for (int k = 0; k < m; ++k) {
                    t = (s0[k] - off * t) / s1[k];
                    s3[k] = t;
                }
                y = t;
            }
            __syncwarp();
        }
        if (lane == 0) s0[CH] = y;  // the next stage's start
#pragma unroll
        for (int j = 0; j < PL; ++j) {
            const int i = n - 1 - (i0 + lane + 32 * j);
            if (i >= 0) x[i] = s3[lane + 32 * j];
        }
        __syncwarp();
    }
}

// a / r^2; a general division of zero takes its slow path
__device__ __forceinline__ double over_r2(double a, double r) { return a == 0.0 ? a : a / (r * r); }

struct Scal {
    double mixing, prevE, prevD, E[5], effd, resid;
    double dsum[3], dnorm[3];
    double Tpart[MAXORB];
    double respart[MAXORB];
    double ee, eh, exc;
    int conv, status, iter, err_orb;
};

__global__ void __launch_bounds__(RT, 1)
    radial_scf_kernel(const RunSpec* __restrict__ specs, int npts, double rmax, double* __restrict__ ws,
                      long long per_run, dft_atom_result* __restrict__ out) {
    extern __shared__ __align__(16) double r[];
    __shared__ Scal S;
    __shared__ RunSpec sp;
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int cl = cluster.num_blocks(), rank = cluster.block_rank(), run = blockIdx.x / cl;
    if (threadIdx.x == 0) sp = specs[run];
    const int n = npts;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double* st = r + (n + 1) / 2 * 2 + warp * WARP_STAGE;  // this warp's stage
    double* base = ws + (long long)run * per_run;
    auto arr = [&](int a) { return base + (long long)(rank * A_COUNT + a) * n; };
    auto orb = [&](int q, int a) { return base + (long long)(cl * A_COUNT + q * O_COUNT + a) * n; };
    const int q0 = warp * cl + rank, qs = RW * cl;  // this warp's orbitals: q0, q0 + qs, ...
    // after each phase that writes orbitals: they and any failure are known to the whole cluster
    auto join = [&]() {
        cluster.sync();
        int st_ = 0;
        for (int b = 0; b < cl; ++b) st_ = max(st_, *cluster.map_shared_rank(&S.status, b));
        cluster.sync();
        if (tid == 0) S.status = st_;
        __syncthreads();
    };
    const double h = rmax / (double)(n + 1);
    for (int i = tid; i < n; i += RT) r[i] = (double)(i + 1) * h;  // RadialGrid.cpp:16-20
    __syncthreads();
    const double dr = r[1] - r[0];
    const double idr2 = 1.0 / (dr * dr);
    const double off = -0.5 * idr2;
    const double oo = off * off;
    const double fourpi = 4.0 * xcf::PI;
    const int Z = sp.Z, kind = sp.kind, norb = sp.norb;  // after the barrier above
    double *da = arr(A_DA), *db = arr(A_DB), *va = arr(A_VA), *vb = arr(A_VB), *vh = arr(A_VH);
    double *oa = arr(A_OA), *ob = arr(A_OB), *rd = arr(A_RD), *od = arr(A_OD);
    double *t1 = arr(A_T1), *t2 = arr(A_T2), *t3 = arr(A_T3), *t4 = arr(A_T4), *enc = arr(A_ENC);
    double* sine = arr(A_SIN);
    if (tid == 0) {
        S.mixing = 0.25;
        S.prevE = INFINITY;
        S.prevD = INFINITY;
        S.conv = 0;
        S.status = 0;
        S.iter = 0;
        S.err_orb = -1;
        for (int q = 0; q < 5; ++q) S.E[q] = 0.0;
        S.effd = 0.0;
        S.resid = 0.0;
    }
    __syncthreads();

    // ---- hydrogenic start orbitals and densities (SelfConsistentField.cpp:207-339) ------------
    for (int q = q0; q < norb; q += qs) {
        double* u = orb(q, O_U);
        const double ex = fmax(0.15, (double)Z / ((double)sp.n[q] * (double)sp.n[q]));
        for (int i = lane; i < n; i += 32) u[i] = pow(r[i], (double)(sp.l[q] + 1)) * exp(-ex * r[i]);
        __syncwarp();
        const double nn = sqrt(dr * seq_dot(n, st, u, u));
        if (nn < EPS) {
            if (lane == 0) { S.status = DFT_NOT_CONVERGED; S.err_orb = q; }
        } else {
            for (int i = lane; i < n; i += 32) u[i] /= nn;
        }
        __syncwarp();
    }
    // the start vector of every inverse iteration (solveEigenvector): sin(1), sin(2), ... normalised
    if (warp == RW - 1) {
        for (int i = lane; i < n; i += 32) sine[i] = sin((double)(i + 1));
        __syncwarp();
        const double nn = sqrt(seq_dot(n, st, sine, sine));
        for (int i = lane; i < n; i += 32) sine[i] /= nn;
    }
    join();
    // calculateSpinDensity (ElectronDensity.cpp:8-56): orbital order, electrons*u*u/(4 pi r r)
    auto spin_densities = [&](double* a, double* b) {
        for (int i = tid; i < n; i += RT) {
            double sa = 0.0, sb = 0.0;
            // Quotients by the exact reciprocal; the squares of a tail, down to the smallest numbers, scaled
            // by 2^200.  A point with one that fits neither is taken again by general divisions.
            const ExactDiv w = exact_div(fourpi * r[i] * r[i]);
            bool general = w.general;
            for (int q0 = 0; q0 < norb; q0 += 4) {
                double u[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) u[q] = q0 + q < norb ? orb(q0 + q, O_U)[i] : 0.0;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (q0 + q >= norb) break;
                    const double num = (double)sp.el[q0 + q] * u[q] * u[q];
                    const bool tiny = num < 0x1p-800;
                    bool bad;
                    double v = divide_fast(tiny ? num * 0x1p200 : num, w, bad);
                    general |= bad | (tiny & (v != 0.0) & !(v >= 0x1p-800));
                    v = tiny ? v * 0x1p-200 : v;
                    if (sp.spin[q0 + q] == 0) sa += v;
                    else sb += v;
                }
            }
            if (general) {
                sa = sb = 0.0;
#pragma unroll 1
                for (int q = 0; q < norb; ++q) {
                    const double u = orb(q, O_U)[i];
                    const double v = (double)sp.el[q] * u * u / w.b;
                    if (sp.spin[q] == 0) sa += v;
                    else sb += v;
                }
            }
            a[i] = sa;
            b[i] = sb;
        }
    };
    spin_densities(da, db);
    __syncthreads();

    // radial Hartree (HartreePotential.cpp:8-86): trapezoid terms by all lanes, prefix sums in order
    auto hartree = [&](const double* rho, double* v) {
        if (warp == 0)
            seq_prefix<false>(
                n, st, enc, [&](int i) { return make_double2(rho[max(i - 1, 0)], rho[i]); },
                [&](int i, double2 v) {
                    return i == 0 ? 0.0 : 0.5 * (fourpi * r[i - 1] * r[i - 1] * v.x + fourpi * r[i] * r[i] * v.y) * dr;
                });
        else if (warp == 1)
            seq_prefix<true>(
                n, st, t3, [&](int i) { return make_double2(rho[i], rho[min(i + 1, n - 1)]); },
                [&](int i, double2 v) {
                    return i == n - 1 ? 0.0 : 0.5 * (fourpi * r[i] * v.x + fourpi * r[i + 1] * v.y) * dr;
                });
        __syncthreads();
        for (int i = tid; i < n; i += RT) v[i] = enc[i] / r[i] + t3[i];
        __syncthreads();
    };
    // calculateRadialGradient (ExchangeCorrelation.cpp:10-51)
    auto rgrad = [&](const double* f, int i) -> double {
        if (i == 0) return (f[1] - f[0]) / (r[1] - r[0]);
        if (i == n - 1) return (f[n - 1] - f[n - 2]) / (r[n - 1] - r[n - 2]);
        return (f[i + 1] - f[i - 1]) / (r[i + 1] - r[i - 1]);
    };
    // calculateRadialDivergence (:53-150)
    auto rdiv = [&](const double* c, int i) -> double {
        if (r[i] == 0.0) return 0.0;
        if (i == 0) return ((r[1] * r[1] * c[1] - r[0] * r[0] * c[0]) / (r[1] - r[0])) / (r[0] * r[0]);
        if (i == n - 1)
            return ((r[n - 1] * r[n - 1] * c[n - 1] - r[n - 2] * r[n - 2] * c[n - 2]) / (r[n - 1] - r[n - 2])) /
                   (r[n - 1] * r[n - 1]);
        return ((r[i + 1] * r[i + 1] * c[i + 1] - r[i - 1] * r[i - 1] * c[i - 1]) / (r[i + 1] - r[i - 1])) / (r[i] * r[i]);
    };
    auto evaluate = [&](int i, const double* a, const double* b) {
        return kind == 1 ? xcf::pbe96(a[i], b[i], rgrad(a, i), rgrad(b, i)) : xcf::pz81(a[i], b[i]);
    };

    for (int it = 1; it <= 250; ++it) {
        if (S.status) break;
        // ---- buildEffectivePotentials (:341-412) ------------------------------------------
        for (int i = tid; i < n; i += RT) rd[i] = da[i] + db[i];
        __syncthreads();
        hartree(rd, vh);
        for (int i = tid; i < n; i += RT) {
            const xcf::Result x = evaluate(i, da, db);
            t1[i] = x.va;  // d f / d n_alpha
            t2[i] = x.ca;
            t3[i] = x.vb;
            t4[i] = x.cb;
        }
        __syncthreads();
        for (int i = tid; i < n; i += RT) {
            const bool floor = da[i] + db[i] <= xcf::RHO_FLOOR;
            const double xa = floor ? 0.0 : (r[i] == 0.0 ? t1[i] : t1[i] - rdiv(t2, i));
            const double xb = floor ? 0.0 : (r[i] == 0.0 ? t3[i] : t3[i] - rdiv(t4, i));
            const double nuc = -(double)Z / r[i];
            va[i] = xa + (nuc + vh[i]);
            vb[i] = xb + (nuc + vh[i]);
        }
        __syncthreads();
        // ---- orbitals: one warp per (n,l,spin), index counts same-spin states per l (:28-77) --
        cluster.sync();  // the other blocks have read the last orbitals
        for (int q = q0; q < norb; q += qs) {
            const double* V = sp.spin[q] == 0 ? va : vb;
            double* diag = orb(q, O_DIAG);
            const double cc = 0.5 * (double)(sp.l[q] * (sp.l[q] + 1));
            double mn = INFINITY, mx = -INFINITY;
            for (int i = lane; i < n; i += 32) {
                const double d = idr2 + over_r2(cc, r[i]) + V[i];  // KohnShamHamiltonian.cpp:78-86
                diag[i] = d;
                mn = fmin(mn, d);
                mx = fmax(mx, d);
            }
            for (int o = 16; o > 0; o >>= 1) {
                mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            }
            __syncwarp();
            double *u = orb(q, O_U), *dw = orb(q, O_DW), *f = orb(q, O_F), *nx = orb(q, O_NX);
            double* zh = orb(q, O_ZH);
            // Rayleigh quotient of the last orbital, a guess only
            double ra = 0.0, rb = 0.0;
            for (int i = lane; i < n; i += 32) {
                const double ui = u[i], uj = i + 1 < n ? u[i + 1] : 0.0;
                ra += ui * (diag[i] * ui + 2.0 * off * uj);
                rb += ui * ui;
            }
            for (int o = 16; o > 0; o >>= 1) {
                ra += __shfl_xor_sync(0xffffffffu, ra, o);
                rb += __shfl_xor_sync(0xffffffffu, rb, o);
            }
            double E = 0.0;
            const double top = fmax(fabs(mn), fabs(mx));
            if (!find_eigenvalue(n, diag, oo, top, sp.idx[q], mn - 10.0, mx + 10.0, ra / rb, st, E)) {
                if (lane == 0) { S.status = DFT_NOT_CONVERGED; S.err_orb = q; }
                continue;
            }
            // ---- solveEigenvector (:223-321) --------------------------------------------
            for (int i = lane; i < n; i += 32) u[i] = sine[i];
            const double shift = E + 1.0e-10 * fmax(1.0, fabs(E));
            if (!factor(n, diag, off, top, shift, sp.pivot_eps, f, dw, zh, st)) {
                if (lane == 0) { S.status = DFT_SINGULAR; S.err_orb = q; }
                continue;
            }
            __syncwarp();
            for (int ii = 0; ii < 1000; ++ii) {
                solve(n, u, f, dw, zh, off, nx, st);
                const double m = sqrt(seq_dot(n, st, nx, nx));
                if (m < EPS) {
                    if (lane == 0) { S.status = DFT_NOT_CONVERGED; S.err_orb = q; }
                    break;
                }
                const ExactDiv dm = exact_div(m);
                const double sd = seq_sum(
                    n, st, [&](int i) { return make_double2(u[i], nx[i]); },
                    [&](int i, double2 v) { return v.x * (nx[i] = divide(v.y, dm)); });
                double md = 0.0;
#pragma unroll 4
                for (int i = lane; i < n; i += 32) {
                    const double v = sd < 0.0 ? -nx[i] : nx[i];
                    md = fmax(md, fabs(u[i] - v));
                    u[i] = v;
                }
                for (int o = 16; o > 0; o >>= 1) md = fmax(md, __shfl_xor_sync(0xffffffffu, md, o));
                __syncwarp();
                if (md < 1.0e-12) break;
            }
            // normalizeVector(u, r[1]-r[0]) (NumericalMethods.cpp:34-61)
            const double un = sqrt(dr * seq_dot(n, st, u, u));
            const ExactDiv dn = exact_div(un);
#pragma unroll 4
            for (int i = lane; i < n; i += 32) u[i] = divide(u[i], dn);
            if (lane == 0) out[run].eigenvalues[q] = E;
            __syncwarp();
        }
        join();
        if (S.status) break;
        // ---- output densities, V_H(out), energies (:620-680, TotalEnergy.cpp) ------------
        spin_densities(oa, ob);
        __syncthreads();
        for (int i = tid; i < n; i += RT) od[i] = oa[i] + ob[i];
        __syncthreads();
        hartree(od, vh);
        // XC energy integrand (ExchangeCorrelation.cpp:276-371)
        for (int i = tid; i < n; i += RT) {
            const double dn = oa[i] + ob[i];
            double e = 0.0;
            if (dn > xcf::RHO_FLOOR) e = evaluate(i, oa, ob).eps;
            t4[i] = fourpi * r[i] * r[i] * dn * e;
        }
        __syncthreads();
        // sums, one warp each: per orbital kinetic energy and KS residual (TotalEnergy.cpp:10-101,
        // SelfConsistentField.cpp:110-205), three energies, three density differences
        const double none = 0.0;
        for (int q = warp; q < 2 * norb + 9; q += RW) {
            const auto halved = [&](int i, double in) { return i == 0 || i == n - 1 ? 0.5 * in : in; };
            if (q < 2 * norb) {
                const int o = q >> 1;
                const double* u = orb(o, O_U);
                const double* V = sp.spin[o] == 0 ? va : vb;
                const double cc = 0.5 * (double)(sp.l[o] * (sp.l[o] + 1));
                const auto load = [&](int i) {
                    return double4{u[i], i > 0 ? u[i - 1] : none, i + 1 < n ? u[i + 1] : none, V[i]};
                };
                if ((q & 1) == 0) {
                    const double oe = seq_sum(n, st, load, [&](int i, const double4& v) {
                        double ap = (idr2 + over_r2(cc, r[i])) * v.x;
                        if (i > 0) ap += off * v.y;
                        if (i + 1 < n) ap += off * v.z;
                        return v.x * ap;
                    });
                    if (lane == 0) S.Tpart[o] = (double)sp.el[o] * oe * dr;
                } else {
                    const double E = out[run].eigenvalues[o];
                    const double s2 = seq_sum(n, st, load, [&](int i, const double4& v) {
                        double hv = (idr2 + over_r2(cc, r[i]) + v.w) * v.x;
                        if (i > 0) hv += off * v.y;
                        if (i + 1 < n) hv += off * v.z;
                        const double rr = hv - E * v.x;
                        return rr * rr;
                    });
                    if (lane == 0) S.respart[o] = sqrt(s2 * dr);
                }
            } else if (q == 2 * norb) {  // external energy (TotalEnergy.cpp:103-168)
                const double e = seq_sum(
                    n, st, [&](int i) { return od[i]; },
                    [&](int i, double v) { return halved(i, -(double)Z * 4.0 * xcf::PI * r[i] * v); });
                if (lane == 0) S.ee = e * dr;
            } else if (q == 2 * norb + 1) {  // Hartree energy (HartreePotential.cpp:88-137)
                const double e = seq_sum(
                    n, st, [&](int i) { return make_double2(od[i], vh[i]); },
                    [&](int i, double2 v) { return halved(i, fourpi * r[i] * r[i] * v.x * v.y); });
                if (lane == 0) S.eh = 0.5 * e * dr;
            } else if (q == 2 * norb + 2) {
                const double e = seq_sum(
                    n, st, [&](int i) { return t4[i]; }, [&](int i, double v) { return halved(i, v); });
                if (lane == 0) S.exc = e * dr;
            } else {  // density differences (:414-485)
                const int w = (q - 2 * norb - 3) >> 1;
                const double* o = w == 0 ? rd : (w == 1 ? da : db);
                const double* nw = w == 0 ? od : (w == 1 ? oa : ob);
                const auto load = [&](int i) { return make_double2(nw[i], o[i]); };
                if ((q - 2 * norb - 3) & 1) {
                    const double n2 = seq_sum(n, st, load, [&](int i, double2 v) {
                        const double wt = 4.0 * xcf::PI * r[i] * r[i];
                        return v.x * v.x * wt;
                    });
                    if (lane == 0) S.dnorm[w] = n2;
                } else {
                    const double d2 = seq_sum(n, st, load, [&](int i, double2 v) {
                        const double wt = 4.0 * xcf::PI * r[i] * r[i];
                        const double d = v.x - v.y;
                        return d * d * wt;
                    });
                    if (lane == 0) S.dsum[w] = d2;
                }
            }
        }
        __syncthreads();
        if (tid == 0) {
            double T = 0.0, res = 0.0;
            for (int w = 0; w < 3; ++w) {
                const double dn = sqrt(S.dsum[w] * dr), nn = sqrt(S.dnorm[w] * dr);
                S.dsum[w] = nn <= EPS ? dn : dn / nn;
            }
            for (int q = 0; q < norb; ++q) {
                T += S.Tpart[q];
                res = fmax(res, S.respart[q]);
            }
            S.E[0] = T;
            S.E[1] = S.ee;
            S.E[2] = S.eh;
            S.E[3] = S.exc;
            S.E[4] = T + S.ee + S.eh + S.exc;
            S.effd = fmax(S.dsum[0], fmax(S.dsum[1], S.dsum[2]));
            S.resid = res;
            S.iter = it;
            const double dE = isfinite(S.prevE) ? fabs(S.E[4] - S.prevE) : INFINITY;
            S.conv = (S.effd < 1.0e-9 && dE < 1.0e-11 && res < 1.0e-7) ? 1 : 0;
            if (!S.conv) {
                if (isfinite(S.prevD)) {
                    if (S.effd > S.prevD * 1.05) S.mixing = fmax(0.10, S.mixing * 0.50);
                    else if (S.effd < S.prevD) S.mixing = fmin(0.50, S.mixing * 1.10);
                }
                S.prevD = S.effd;
                S.prevE = S.E[4];
            }
        }
        __syncthreads();
        if (S.conv) break;
        // mixDensity with the updated factor (SelfConsistentField.cpp:514-535, :766-776)
        const double m = S.mixing;
        for (int i = tid; i < n; i += RT) {
            da[i] = (1.0 - m) * da[i] + m * oa[i];
            db[i] = (1.0 - m) * db[i] + m * ob[i];
        }
        __syncthreads();
    }
    if (tid == 0 && rank == 0) {
        dft_atom_result& o = out[run];
        o.Z = Z;
        o.kind = kind;
        o.kinetic = S.E[0];
        o.external = S.E[1];
        o.hartree = S.E[2];
        o.exchange_correlation = S.E[3];
        o.total = S.E[4];
        o.iterations = S.iter;
        o.converged = S.conv;
        o.density_difference = S.effd;
        o.max_ks_residual = S.resid;
        o.n_orbitals = norb;
        o.status = S.status;
    }
    cluster.sync();  // no block leaves while another may still read its status
}

// The chains by themselves, for tests.
__global__ void radial_quotient_kernel(long long m, const double* __restrict__ a, const double* __restrict__ g,
                                       double* __restrict__ out) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (long long)gridDim.x * blockDim.x)
        out[i] = quotient(a[i], g[i]);
}
// block 0: the factors at `shift` and the solution for u; block 1 + b: counts at 32 values of E
__global__ void __launch_bounds__(32)
    radial_tridiagonal_kernel(int n, const double* __restrict__ diag, double off, double shift, const double* u, double* f,
                              double* w, double* x, double* zh, int m, const double* __restrict__ E,
                              int* __restrict__ counts, int* __restrict__ ok) {
    __shared__ __align__(16) double st[WARP_STAGE];
    const int lane = threadIdx.x;
    double top = 0.0;
    for (int i = lane; i < n; i += 32) top = fmax(top, fabs(diag[i]));
    for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (blockIdx.x > 0) {
        const int e = (blockIdx.x - 1) * 32 + lane;
        const int c = sturm_count(n, diag, off * off, top, E[min(e, m - 1)], st);
        if (e < m) counts[e] = c;
        return;
    }
    const bool good = factor(n, diag, off, top, shift, EPS, f, w, zh, st);
    __syncwarp();
    if (good) solve(n, u, f, w, zh, off, x, st);
    if (lane == 0) *ok = good;
}

// getAtomicConfiguration (ElectronicConfiguration.cpp:16-146) as (n,l,alpha,beta) rows
void configuration(int Z, std::vector<std::array<int, 4>>& rows) {
    rows.clear();
    auto add = [&](int n, int l, int e) {
        const int cap = 2 * l + 1;
        const int a = std::min(e, cap);
        rows.push_back({n, l, a, e - a});
    };
    add(1, 0, std::min(Z, 2));
    if (Z >= 3) add(2, 0, std::min(Z - 2, 2));
    if (Z >= 5) add(2, 1, std::min(Z - 4, 6));
    if (Z >= 11) add(3, 0, std::min(Z - 10, 2));
    if (Z >= 13) add(3, 1, std::min(Z - 12, 6));
    if (Z >= 19) {
        int s = Z >= 20 ? 2 : 1;
        if (Z == 24 || Z == 29) s = 1;
        add(4, 0, s);
    }
    if (Z >= 21) {
        int d = Z - 20;
        if (Z == 24) d = 5;
        else if (Z >= 29) d = 10;
        add(3, 2, d);
    }
}

}  // namespace

namespace {

constexpr long RADIAL_MAX_POINTS = 12000;
constexpr size_t radial_smem(long points) {  // at most 175 KB
    return sizeof(double) * ((size_t)(points + 1) / 2 * 2 + (size_t)RW * WARP_STAGE);
}

// Builds the run specs, launches the batch and leaves every run's arrays in the WS_RADIAL
// workspace (returned; per_run doubles per run: A_* per block, then at `orbitals` MAXORB x O_*).
double* run_batch(dft_context* ctx, int nruns, const int* Z, const int* kinds, long points, double rmax,
                  dft_atom_result* results, std::vector<RunSpec>& specs, long long& per_run,
                  long long& orbitals) {
    if (points < 2) fail(DFT_INVALID_ARGUMENT, "La malla radial debe contener al menos dos puntos.");
    if (points > RADIAL_MAX_POINTS) fail(DFT_INVALID_ARGUMENT, "at most %ld radial points per run", RADIAL_MAX_POINTS);
    if (!(rmax > 0.0)) fail(DFT_INVALID_ARGUMENT, "RMAX debe ser mayor que cero.");
    specs.assign(nruns, RunSpec{});
    for (int rr = 0; rr < nruns; ++rr) {
        if (Z[rr] < 1 || Z[rr] > 30) fail(DFT_INVALID_ARGUMENT, "Configuracion atomica no disponible para Z = %d", Z[rr]);
        if (kinds[rr] != 0 && kinds[rr] != 1) fail(DFT_INVALID_ARGUMENT, "unknown functional kind %d", kinds[rr]);
        std::vector<std::array<int, 4>> rows;
        configuration(Z[rr], rows);
        RunSpec& s = specs[rr];
        std::memset(&s, 0, sizeof s);
        s.Z = Z[rr];
        s.kind = kinds[rr];
        s.pivot_eps = ctx->radial_pivot_exp == -14 ? EPS : std::pow(10.0, (double)ctx->radial_pivot_exp);
        int q = 0;
        for (int spin = 0; spin < 2; ++spin) {
            int count_l[4] = {0, 0, 0, 0};
            for (auto& row : rows) {
                const int e = row[2 + spin];
                if (e <= 0) continue;
                s.n[q] = row[0];
                s.l[q] = row[1];
                s.spin[q] = spin;
                s.el[q] = e;
                s.idx[q] = count_l[row[1]]++;
                ++q;
            }
        }
        s.norb = q;
    }
    // blocks per run: four, or two, while all of them have an SM of their own
    const int cl = 4LL * nruns <= ctx->num_sms ? 4 : 2LL * nruns <= ctx->num_sms ? 2 : 1;
    orbitals = (long long)cl * A_COUNT * points;
    per_run = orbitals + (long long)MAXORB * O_COUNT * points;
    double* ws = (double*)ws_get(ctx, WS_RADIAL, sizeof(double) * (size_t)per_run * nruns);
    const size_t spec_bytes = ((sizeof(RunSpec) * nruns + 255) / 256) * 256;  // keep the results 256-B aligned
    char* dbuf = (char*)ws_get(ctx, WS_TMP2, spec_bytes + sizeof(dft_atom_result) * nruns);
    RunSpec* dspec = (RunSpec*)dbuf;
    dft_atom_result* dres = (dft_atom_result*)(dbuf + spec_bytes);
    DFT_CUDA(cudaMemcpyAsync(dspec, specs.data(), sizeof(RunSpec) * nruns, cudaMemcpyHostToDevice, ctx->stream));
    DFT_CUDA(cudaMemsetAsync(dres, 0, sizeof(dft_atom_result) * nruns, ctx->stream));
    // The limit is the process's, not the context's: the same value from every thread, so that none lowers it
    // between another's two calls.
    const size_t smem = radial_smem(points);
    DFT_CUDA(cudaFuncSetAttribute(radial_scf_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)radial_smem(RADIAL_MAX_POINTS)));
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = cl;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(nruns * cl);
    lc.blockDim = dim3(RT);
    lc.dynamicSmemBytes = smem;
    lc.stream = ctx->stream;
    lc.attrs = &at;
    lc.numAttrs = 1;
    DFT_CUDA(cudaLaunchKernelEx(&lc, radial_scf_kernel, (const RunSpec*)dspec, (int)points, rmax, ws, per_run, dres));
    count_launch(ctx);
    DFT_CUDA(cudaMemcpyAsync(results, dres, sizeof(dft_atom_result) * nruns, cudaMemcpyDeviceToHost, ctx->stream));
    sync(ctx);
    return ws;
}

}  // namespace

void solve_atoms(dft_context* ctx, int nruns, const int* Z, const int* kinds, long points, double rmax,
                 dft_atom_result* results) {
    std::vector<RunSpec> specs;
    long long per_run = 0, orbitals = 0;
    run_batch(ctx, nruns, Z, kinds, points, rmax, results, specs, per_run, orbitals);
}

void radial_quotients(dft_context* ctx, long long m, const double* a, const double* g, double* out) {
    radial_quotient_kernel<<<(unsigned)std::min<long long>((m + 255) / 256, 8LL * ctx->num_sms), 256, 0, ctx->stream>>>(
        m, a, g, out);
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
    sync(ctx);
}

void radial_tridiagonal(dft_context* ctx, long n, const double* diag, double off, double shift, const double* u,
                        double* f, double* w, double* x, int m, const double* E, int* counts) {
    if (n < 2 || n > RADIAL_MAX_POINTS) fail(DFT_INVALID_ARGUMENT, "2 to %ld points", RADIAL_MAX_POINTS);
    double* zh = (double*)ws_get(ctx, WS_RADIAL, sizeof(double) * (size_t)n);
    int* ok = (int*)ws_get(ctx, WS_TMP2, sizeof(int));
    radial_tridiagonal_kernel<<<1 + (m + 31) / 32, 32, 0, ctx->stream>>>((int)n, diag, off, shift, u, f, w, x, zh, m, E,
                                                                         counts, ok);
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
    int* h = (int*)pinned(ctx, 1);
    DFT_CUDA(cudaMemcpyAsync(h, ok, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    sync(ctx);
    if (!*h) fail(DFT_SINGULAR, "a pivot of the shifted radial Hamiltonian is below %g", EPS);
}

int atomic_orbital_count(int nnuc, const int* Z) {
    int n = 0;
    std::vector<std::array<int, 4>> rows;
    for (int a = 0; a < nnuc; ++a) {
        if (Z[a] < 1 || Z[a] > 30) continue;
        configuration(Z[a], rows);
        for (auto& row : rows)
            if (row[2] > 0 && row[1] <= 2) n += 2 * row[1] + 1;
    }
    return n;
}

void radial_atom_tables(dft_context* ctx, int nz, const int* Z, int kind, long points, double rmax, double* dens,
                        double* orbs, std::vector<std::vector<std::array<int, 2>>>& shells) {
    // elements not solved before on this context (for this functional and radial grid) are
    // solved in one batch and kept; every element is then copied from the kept tables
    long long rbits;
    std::memcpy(&rbits, &rmax, sizeof(rbits));
    auto key = [&](int z) { return std::array<long long, 4>{z, kind, points, rbits}; };
    std::vector<int> todo;
    for (int rr = 0; rr < nz; ++rr)
        if (!ctx->radial_tables.count(key(Z[rr])) && std::find(todo.begin(), todo.end(), Z[rr]) == todo.end())
            todo.push_back(Z[rr]);
    if (!todo.empty()) {
        const int nt = (int)todo.size();
        std::vector<int> kinds(nt, kind);
        std::vector<dft_atom_result> res(nt);
        std::vector<RunSpec> specs;
        long long per_run = 0, orbitals = 0;
        const double* ws =
            run_batch(ctx, nt, todo.data(), kinds.data(), points, rmax, res.data(), specs, per_run, orbitals);
        for (int rr = 0; rr < nt; ++rr) {
            if (res[rr].status != DFT_OK)
                fail((dft_status_t)res[rr].status, "radial atom Z = %d failed (status %d)", todo[rr], res[rr].status);
            RadialTable t;
            const RunSpec& sp = specs[rr];
            for (int q = 0; q < sp.norb; ++q)
                if (sp.spin[q] == 0) t.shells.push_back({sp.n[q], sp.l[q]});  // every occupied alpha (n, l)
            if ((int)t.shells.size() > RADIAL_MAX_SHELLS)
                fail(DFT_INVALID_ARGUMENT, "atom Z = %d has more than %d shells", todo[rr], RADIAL_MAX_SHELLS);
            DFT_CUDA(cudaMalloc(&t.dens, sizeof(double) * points * (1 + RADIAL_MAX_SHELLS)));
            t.orbs = t.dens + points;
            const double* base = ws + (long long)rr * per_run;
            DFT_CUDA(cudaMemcpyAsync(t.dens, base + (long long)A_OD * points, sizeof(double) * points,
                                     cudaMemcpyDeviceToDevice, ctx->stream));
            int k = 0;
            for (int q = 0; q < sp.norb; ++q) {
                if (sp.spin[q] != 0) continue;
                DFT_CUDA(cudaMemcpyAsync(t.orbs + (long long)k * points,
                                         base + orbitals + (long long)(q * O_COUNT + O_U) * points,
                                         sizeof(double) * points, cudaMemcpyDeviceToDevice, ctx->stream));
                ++k;
            }
            ctx->radial_tables[key(todo[rr])] = std::move(t);
        }
    }
    shells.assign(nz, {});
    for (int rr = 0; rr < nz; ++rr) {
        const RadialTable& t = ctx->radial_tables.at(key(Z[rr]));
        DFT_CUDA(cudaMemcpyAsync(dens + (long long)rr * points, t.dens, sizeof(double) * points,
                                 cudaMemcpyDeviceToDevice, ctx->stream));
        if (!t.shells.empty())
            DFT_CUDA(cudaMemcpyAsync(orbs + (long long)rr * RADIAL_MAX_SHELLS * points, t.orbs,
                                     sizeof(double) * points * t.shells.size(), cudaMemcpyDeviceToDevice,
                                     ctx->stream));
        shells[rr] = t.shells;
    }
}

}  // namespace dftb
