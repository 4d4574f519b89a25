/*
 * fn_rounded.cuh -- square roots, reciprocals and quotients that share one
 * seed, each rounded as the IEEE operation rounds it.
 *
 * The force terms take a root, its reciprocal and one or two quotients of the
 * same quantity (a spring's length, an angle's arms, a contact's distance).
 * As separate operators each of them starts from a seed of its own, tests its
 * own range and branches to its own slow path; here one reciprocal square
 * root seeds them all and one range test covers them, so a Lennard-Jones
 * contact's root, its reciprocal and two quotients are 22 multiplications and
 * multiply-adds and one seed with no branch between them.
 *
 * The corrections are the classical ones for hardware with a fused
 * multiply-add (P. Markstein, "Computation of elementary functions on the
 * IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990; M. Cornea,
 * J. Harrison, P. Tang, "Intel Itanium floating-point architecture", 2003):
 * the residual of an approximation is exact in one fused operation, and one
 * more fused operation adds it.  With u = 2^-52:
 *   root        y ~ 1/sqrt(d) to 0.75 u; s = d y; s + (d - s s) y/2 differs
 *               from the root by less than 3.4 u^2 before it is rounded;
 *   reciprocal  y ~ 1/b to 2 u; r = y + y (1 - b y) differs from 1/b by less
 *               than 4 u^2/b before it is rounded, so r is one of the two
 *               doubles around 1/b; r + r (1 - b r) is then below 1/b by
 *               b 2^-108 at most (b in [1, 2)), while the middle of two
 *               doubles that lies below 1/b lies k 2^-106/b below it for a
 *               whole k > 0.  b^2 < 4: no middle is between, the result is
 *               rounded as 1/b is, but for b = 2 - u, where the two meet;
 *   quotient    with y = 1/b, q = a y, q + y (a - b q) is a/b correctly
 *               rounded (Markstein's theorem; where a/b is next to a middle, q
 *               is one of the two doubles around it).  y may also be the
 *               double on the other side of a middle next to 1/b: the error of
 *               the last operation, half a unit of q times b times y's error,
 *               reaches a middle only for mantissas b = 2 - j u with k = j^2
 *               >= 2 j, k <= 16, i.e. j = 3, of whose few quotients next to a
 *               middle none rounds wrongly.  So the reciprocals that only
 *               quotients use take one correction.
 * A root can round differently from the operator only where d - m^2 is a
 * multiple k 2^-107 of d's binade with |k| < 54, m the middle of two doubles.
 * Those operands (found by square roots modulo 2^54), the mantissas whose
 * reciprocals lie closest to a middle (the divisors of 2^106 - k, k <= 16),
 * quotients next to a middle and random operands are compared with the IEEE
 * operations by the GPU tests: every bit is the same.  (With one correction of
 * the reciprocal instead of two, some dozens of mantissas came out one unit
 * in the last place apart; the second, with the quotients' test of the
 * numerator, costs 0.5-0.9 % of a run: 100 steps of the 1M-bead tensile network
 * 14.95 -> 15.02 ms, the dense mat's 24 of 4M beads 15.63 -> 15.72.)
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

/* 1/b, y ~ 1/b to 2 u, or for some dozens of mantissas the double on the other
   side of the middle next to it: what quotient needs.  A mantissa of all ones
   comes out as a power of two, one unit below the rounded reciprocal
   (Markstein's exception). */
__device__ __forceinline__ double recip_near(double b, double y) {
    const double r = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
    const int ones = (__double2hiint(b) | (int)0xfff00000) & __double2loint(b);
    return __hiloint2double(__double2hiint(r), __double2loint(r) | (ones == -1 ? 1 : 0));
}

/* 1/b, y ~ 1/b to 2 u */
__device__ __forceinline__ double recip_from(double b, double y) {
    const double r = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
    return recip_near(b, r);
}

/* a/b, y = 1/b as recip_near or recip_from gives it, neither a nor a/b near the ends of the
   normal range */
__device__ __forceinline__ double quotient(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

/* |a| in [2^-400, 2^400): the residual of a/b is exact and the quotient normal
   for every b that is a root above 0 (2^-537 .. 2^512).  False for zeros,
   infinities (whose residual is NaN) and NaN. */
__device__ __forceinline__ bool fn_quotient_range(double a) {
    return ((unsigned)__double2hiint(a) & 0x7fffffffu) - 0x26f00000u < 0x32000000u;
}

/* a/b for any a, b a finite root above 0.  A zero, as most tangents of an
   adjoint sweep's first steps are, keeps its sign. */
__device__ __forceinline__ double quotient_any(double a, double b, double y) {
    if (fn_quotient_range(a)) return quotient(a, b, y);
    return a == 0.0 ? __dmul_rn(a, y) : a / b;
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
