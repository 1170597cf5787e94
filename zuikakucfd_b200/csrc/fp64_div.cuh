// FP64 division without branches, and several quotients over one denominator.
//
// The FP64 kernels divide up to 15 times per interface.  The compiler's divide
// carries a range test and a call on its slow path each time, so consecutive
// divisions cannot overlap, and every division starts from its own
// reciprocal.  Here the caller vouches for the operands' ranges -- tested once
// for a whole tile of cells (plain_value) or for a state's four values (num_ok),
// plus a test of the few denominators that differences form (in_range) -- and
// takes plain `/` elsewhere; inside the range the quotients are straight-line
// code.
//
// Reference-arithmetic build: quotients are correctly rounded, hence bit for
// bit those of `/`.  With y = RN(1/b) and q within one ulp of a/b,
// RN(q + y RN(a - b q)) = RN(a/b) (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34,
// 1990, Theorem 8.1's correction step; the remainder is exact).  y starts from
// the 20-bit hardware approximation y0: with e = 1 - b y0, the cubic step
// y0 + y0 (e + e^2) leaves a relative error below 2^-53 + 2^-57, and one
// Newton step from there rounds to RN(1/b) for every b but the all-ones
// significand (in_range sends those to `/`).  RN(a y) is within 1.5 ulp of
// a/b, so two correction steps follow: the first brings it within one ulp, the
// second rounds.
//
// FMA build (ZK_PREC_FP64_FMA): y within one ulp, quotients a y.
#pragma once

#include <cstdint>

namespace zk {

// |x| in [2^-500, 2^500): denominators for which neither the reciprocal nor a
// remainder leaves the normal range (false for NaN, inf, 0 and, by its low
// word alone, the all-ones significand).
__device__ __forceinline__ bool in_range(double x) {
    return (uint32_t)((__double2hiint(x) & 0x7fffffff) - 0x20b00000) < 0x3e800000u && __double2loint(x) != -1;
}

// a == +0 (the quotient of a -0 would lose its sign) or |a| in [2^-300, 2^100):
// conserved values whose quotients by a density in [1e-5, 2^100), and the
// fluxes' second-level quotients of those, stay above 2^-800 and below 2^700.
__device__ __forceinline__ bool num_ok(double a) {
    const int h = __double2hiint(a);
    return (uint32_t)((h & 0x7fffffff) - 0x2d300000) < 0x19000000u || (h | __double2loint(a)) == 0;
}

// Whether any of the values has a low word of all ones: the test that in_range
// makes, for denominators known to be within its bounds.
__device__ __forceinline__ bool ones_low(double a, double b) {
    return max((uint32_t)__double2loint(a), (uint32_t)__double2loint(b)) == 0xffffffffu;
}
__device__ __forceinline__ bool ones_low(double a, double b, double c) {
    return max(max((uint32_t)__double2loint(a), (uint32_t)__double2loint(b)), (uint32_t)__double2loint(c)) ==
           0xffffffffu;
}

// a == 0 or |a| in [2^-200, 2^60).
__device__ __forceinline__ bool plain_value(double a) {
    const uint32_t h = __double2hiint(a) & 0x7fffffff;
    return h - 0x33700000u < 0x10400000u || (h | __double2loint(a)) == 0;
}

// 1/b for in_range(b): RN (see above), or within one ulp when !EXACT.
template <bool EXACT>
__device__ __forceinline__ double recip(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    double e = __fma_rn(-b, y, 1.0);
    e = __fma_rn(e, e, e);
    y = __fma_rn(y, e, y);
    if constexpr (EXACT) y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
    return y;
}

// a/b, given y = recip<EXACT>(b).
template <bool EXACT>
__device__ __forceinline__ double quot(double a, double b, double y) {
    double q = __dmul_rn(a, y);
    if constexpr (EXACT) {
        q = __fma_rn(__fma_rn(-b, q, a), y, q);
        q = __fma_rn(__fma_rn(-b, q, a), y, q);
    }
    return q;
}

template <bool EXACT>
__device__ __forceinline__ double divide(double a, double b) {
    return quot<EXACT>(a, b, recip<EXACT>(b));
}

}  // namespace zk
