// Correctly rounded division by a loop-invariant divisor (bit-identical to __ddiv_rn).
//
// With zh = RN(1/b) and zl = RN(1/b - zh), q = RN(a zh + RN(a zl)) is a faithful quotient a/b
// (Brisebarre, Muller and Raina, "Accelerating correctly rounded floating-point division when the
// divisor is known in advance", IEEE Trans. Comput. 53, 2004); the remainder r = a - b q is then exact in
// one FMA and RN(q + r zh) is the correctly rounded quotient (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990).  Four dependent FP64
// operations instead of the 126 cycles measured for a general division.  Both theorems assume that
// nothing under- or overflows: numerators outside [2^-899, 2^900) take the general division, as does
// every numerator when the divisor is not in [2^-100, 2^100].
#pragma once

#include <cmath>

namespace dftb {

struct ExactDiv {
    double b, zh, zl;
    int general;  // 1: the divisor is out of range, always divide
};

#ifdef __CUDACC__
__host__ __device__
#endif
inline ExactDiv exact_div(double b) {
    ExactDiv d{b, 0.0, 0.0, 1};
    if (b >= 0x1p-100 && b <= 0x1p100) {
        d.zh = 1.0 / b;
        d.zl = fma(-b, d.zh, 1.0) / b;  // 1 - b zh is exact
        d.general = 0;
    }
    return d;
}

#ifdef __CUDACC__
// the quotient for zero and for numerators in range; bad: others (the value is then not used)
__device__ __forceinline__ double divide_fast(double a, const ExactDiv& d, bool& bad) {
    const unsigned hi = (unsigned)__double2hiint(a), e = (hi >> 20) & 0x7ffu;
    const bool zero = ((hi & 0x7fffffffu) | (unsigned)__double2loint(a)) == 0;
    bad = e - 124u >= 1800u && !zero;
    const double q = __fma_rn(a, d.zh, __dmul_rn(a, d.zl));
    const double r = __fma_rn(-d.b, q, a);
    return zero ? a : __fma_rn(r, d.zh, q);  // b is positive
}
__device__ __forceinline__ double divide(double a, const ExactDiv& d) {
    bool bad;
    const double q = divide_fast(a, d, bad);
    return bad || d.general ? __ddiv_rn(a, d.b) : q;
}
#endif

}  // namespace dftb
