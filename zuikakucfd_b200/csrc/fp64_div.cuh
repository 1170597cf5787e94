// FP64 division without branches, and several quotients over one denominator.
//
// The FP64 kernels divide up to 15 times per interface, several times by the
// same value.  Here the caller vouches for the operands' ranges -- tested once
// for a whole tile of cells (plain_value) or for a state's four values (num_ok),
// plus a test of the few denominators that differences form (in_range) -- and
// takes plain `/` elsewhere; inside the range the quotients are straight-line
// code that overlaps, and those over one denominator share its reciprocal.
//
// Quotients are correctly rounded, hence bit for bit those of `/`, in the
// reference-arithmetic build and in the contracted one (ZK_PREC_FP64_FMA fuses
// multiply-adds and changes nothing else).  The method is P. Markstein's
// ("Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34, 1990): Newton's iteration
// y <- y + y (1 - b y) for the reciprocal, then the quotient corrected by its
// remainder, q <- q + y (a - b q), all with fused multiply-adds.
//   Reciprocal.  The hardware approximation is within 2^-19 of 1/b (measured
// for every significand it distinguishes, tests/test_fp64_div_gpu.py).  Two
// iterations leave half an ulp plus a relative 2^-75.  The third then adds an
// exact residual: before rounding it is (1/b)(1 - d^2) with |d| < b 2^-54 +
// 2^-75, b scaled to [1, 2).  It rounds as 1/b does unless a midpoint m of two
// neighbouring values lies between, 0 < 1 - b m <= d^2.  1 - b m is a positive
// multiple of 2^-106, so d^2 >= 2^-106 and b > 2 - 2^-20; with b = 2 - t 2^-52
// that needs t^2 - 1 to be a multiple of 2^53 - t, which of t < 2^33 only t =
// 1 is: the all-ones significand, which in_range sends to `/`.
//   Quotient.  RN(a y) is within 2 ulp of a/b; the first correction brings it
// within one, and from there RN(q + y (a - b q)) = RN(a/b) for y = RN(1/b)
// (Markstein's theorem; the remainder is exact).
#pragma once

#include <cstdint>

namespace zk {

// |x| in [2^-500, 2^500): denominators for which neither the reciprocal nor a
// remainder leaves the normal range (false for NaN, inf, 0 and, by its low
// word alone, the all-ones significand).
__device__ __forceinline__ bool in_range(double x) {
    return (uint32_t)((__double2hiint(x) & 0x7fffffff) - 0x20b00000) < 0x3e800000u && __double2loint(x) != -1;
}

// a == +0 (face and point values are sums that start from +0, never -0) or |a|
// in [2^-300, 2^100): conserved values whose quotients by a density in [1e-5, 2^100), and the
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

// RN(1/b) for in_range(b).
__device__ __forceinline__ double recip(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
#pragma unroll
    for (int k = 0; k < 3; ++k) y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
    return y;
}

// RN(a/b) for b > 0, given y = recip(b).  The remainder is formed as b q - a:
// for a = -0 that is +0, subtracting it keeps the quotient -0, and so with +0.
__device__ __forceinline__ double quot(double a, double b, double y) {
    double q = __dmul_rn(a, y);
#pragma unroll
    for (int k = 0; k < 2; ++k) q = __fma_rn(-__fma_rn(b, q, -a), y, q);
    return q;
}

// RN(a/b) for b of either sign and a other than -0 (with this sign of the
// remainder, +0 keeps its quotient's sign over a negative b).
__device__ __forceinline__ double divide(double a, double b) {
    const double y = recip(b);
    double q = __dmul_rn(a, y);
#pragma unroll
    for (int k = 0; k < 2; ++k) q = __fma_rn(__fma_rn(-b, q, a), y, q);
    return q;
}

}  // namespace zk
