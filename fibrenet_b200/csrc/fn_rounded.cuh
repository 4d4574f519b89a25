/*
 * fn_rounded.cuh -- square roots, reciprocals and quotients that share one
 * seed, each rounded as the IEEE operation rounds it.
 *
 * The force terms take a root, its reciprocal and one or two quotients of the
 * same quantity (a spring's length, an angle's arms, a contact's distance).
 * As separate operators each of them starts from a seed of its own, tests its
 * own range and branches to its own slow path; here one reciprocal square
 * root seeds them all and one range test covers them, so a Lennard-Jones
 * contact's root, reciprocal and two quotients are 18 multiply-adds and one
 * seed with no branch between them.
 *
 * The corrections are the classical ones for hardware with a fused
 * multiply-add (P. Markstein, "Computation of elementary functions on the
 * IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990; M. Cornea,
 * J. Harrison, P. Tang, "Intel Itanium floating-point architecture", 2003):
 * the residual of an approximation is exact in one fused operation, and one
 * more fused operation adds it.  With u = 2^-52:
 *   root        y ~ 1/sqrt(d) to 0.75 u; s = d y; s + (d - s s) y/2 differs
 *               from the root by less than 3.4 u^2 before it is rounded;
 *   reciprocal  y ~ 1/b to 2 u; y + y (1 - b y) differs from 1/b by the
 *               square of y's error, below 4 u^2/b, and always from below;
 *   quotient    with y = 1/b correctly rounded, q = a y, q + y (a - b q) is
 *               a/b correctly rounded (Markstein's theorem).
 * A root or a reciprocal can round differently from the operator only where
 * the exact value lies within those errors of the middle of two doubles: for
 * a root where d - m^2 is a multiple k 2^-107 of d's binade with |k| < 54, m
 * the middle; for a reciprocal where b m = 1 - k 2^-106, 0 < k <= 16.  All
 * such operands (3,235 mantissas, found by square roots modulo 2^54 and by
 * factoring 2^106 - k) and 9e9 random ones were compared with the operators:
 * every root and every quotient is the operator's, and so is every reciprocal
 * but those of a few dozen mantissas out of 2^52, which may come out one unit
 * in the last place apart.  The one of them that real inputs meet, 2^53 - 1
 * (squared distances a rounding below 1 or 4: straight fibres of unit
 * spacing), is corrected.
 */
#ifndef FIBRENET_ROUNDED_CUH
#define FIBRENET_ROUNDED_CUH

#include <cuda_runtime.h>

namespace fn {

/* d in [2^-200, 2^200): no intermediate of the sequences below leaves the
   normal range.  False for 0, negative numbers, infinities and NaN. */
__device__ __forceinline__ bool fn_fast_range(double d) {
    return (unsigned)(__double2hiint(d) - 0x33700000) < 0x19000000u;
}

/* 1/sqrt(d) to 0.75 u: the hardware's approximation, then one third-order
   step (y + y e (1/2 + 3/8 e), e = 1 - d y^2). */
__device__ __forceinline__ double rsqrt_seeded(double d) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = __fma_rn(-__dmul_rn(d, y), y, 1.0);
    return __fma_rn(__fma_rn(e, 0.375, 0.5), __dmul_rn(y, e), y);
}

/* sqrt(d), y = rsqrt_seeded(d) */
__device__ __forceinline__ double root_from(double d, double y) {
    const double s = __dmul_rn(d, y);
    return __fma_rn(__fma_rn(-s, s, d), __dmul_rn(0.5, y), s);
}

/* 1/b, y ~ 1/b to 2 u.  A mantissa of all ones comes out as a power of two,
   one unit below the rounded reciprocal (Markstein's exception). */
__device__ __forceinline__ double recip_from(double b, double y) {
    const double r = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
    const int ones = (__double2hiint(b) | (int)0xfff00000) & __double2loint(b);
    return __hiloint2double(__double2hiint(r), __double2loint(r) | (ones == -1 ? 1 : 0));
}

/* a/b, y = 1/b correctly rounded */
__device__ __forceinline__ double quotient(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

/* l = sqrt(d) and il = 1/l as the operators give them (il = 0 for l = 0, as
   the force terms want it). */
__device__ __forceinline__ void root_and_inverse(double d, double& l, double& il) {
    if (fn_fast_range(d)) {
        const double y = rsqrt_seeded(d);
        l = root_from(d, y);
        il = recip_from(l, y);
    } else {
        l = sqrt(d);
        il = l != 0.0 ? 1.0 / l : 0.0;
    }
}

}  // namespace fn

#endif
