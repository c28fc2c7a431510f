// Correctly rounded double division by a shared divisor, after P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34(1), 1990 (the reciprocal and quotient correction
// theorems), as also presented in Cornea, Harrison & Tang, "Scientific
// Computing on Itanium-based Systems", 2002, ch. 8.
//
//   quot_rn(a, b, y):  with y = RN(1/b): q0 = RN(a y), r = a - q0 b (exact by
//                 fused multiply-add), q = RN(q0 + r y) = RN(a / b).
//
// The reciprocal of an undeformed length is an IEEE division on the host (the bond
// dictionary), that of a deformed length comes with its square root
// (sqrt_recip_rn).
//
// Preconditions (no underflow or overflow in any step): b and a / b normal and
// well inside the exponent range, a not -0. The kernels use this only when
// every coordinate is +0 or of magnitude in [2^-100, 2^100] and L0 lies in the
// same range; outside it they fall back to IEEE division. bbpd_selftest_division
// compares it, with both kinds of reciprocal, against IEEE `/` bit for bit on the
// device.
#pragma once

namespace bbpd {

// RN(a / b) given y = RN(1/b), for a = +0 or |a / b| normal (see
// preconditions). An exact q0 leaves r = +0 and q0 unchanged.
__device__ __forceinline__ double quot_rn(double a, double b, double y)
{
    const double q0 = __dmul_rn(a, y);
    const double r = __fma_rn(-q0, b, a);
    return __fma_rn(r, y, q0);
}

// Correctly rounded square root and reciprocal of it from one hardware
// reciprocal-square-root approximation, without a branch: P. Markstein,
// "Software division and square root using Goldschmidt's algorithms", Proc.
// RNC'6, 2004. With y0 ~ 1/sqrt(x), g = x y0 and h = y0/2 converge together to
// sqrt(x) and 1/(2 sqrt(x)): r = 1/2 - g h, g <- g + g r, h <- h + h r. Two
// rounds leave g and h a few units of 2^-53 off, whatever the seed's last bits
// are; then d = x - g^2 and L = RN(g + d h) is the square root. Two Newton-Raphson
// steps y <- y + y (1 - L y) from y = 2h give RN(1/L) for every L whose significand
// is not all ones (the reciprocal theorem).
//
// Error of g + d h before its rounding, relative, with g and h within
// 2.5 2^-53: second order 3.1 2^-106, h's error on d h 6.2 2^-106, rounding of
// d 2 2^-106; below 2^-102 in all. sqrt(x) of a double that is no perfect
// square is |c| 2^-108 or more away from the next rounding midpoint, c the odd
// integer M^2 - x scaled by the midpoint's last place (c = 1 mod 8), so only
// the few hundred significands with |c| < 2^7 could round another way.
// bbpd_selftest_sqrt compares every significand with |c| < 2^13, the seed of
// every high word, and seeded samples with IEEE sqrt and division bit for bit.
//
// The compiler's double sqrt carries a branch for its rare operands, which kept
// the four entries of a group from interleaving, and its result had to be ready
// before the reciprocal's own seed: together they took 15 to 16 FP64 operations
// and two seeds an entry, here 13 and one. Step kernel, B200, before and after:
// 720 nodes 38.8 -> 30.6 us, 20 000 nodes 49.7 -> 46.1 us, 128 000 nodes 131.8 ->
// 121.7 us, 1.28M nodes 865 -> 818 us, eight beams in a batch 270 -> 262 us.
//
// ok = false where x is zero, negative, infinite, NaN or outside
// [2^-700, 2^700), and where the low 32 bits of L are all ones, which includes the
// significand that the last step does not cover: the caller takes IEEE operations
// then.
__device__ __forceinline__ double rsqrt_approx(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}

__device__ __forceinline__ void sqrt_recip_rn(double x, double &L, double &rL, bool &ok)
{
    const double y0 = rsqrt_approx(x);
    double g = __dmul_rn(x, y0);
    double h = __hiloint2double(__double2hiint(y0) - (1 << 20), __double2loint(y0));   // y0 / 2
    double r = __fma_rn(-g, h, 0.5);
    g = __fma_rn(g, r, g);
    h = __fma_rn(h, r, h);
    r = __fma_rn(-g, h, 0.5);
    g = __fma_rn(g, r, g);
    h = __fma_rn(h, r, h);
    const double d = __fma_rn(-g, g, x);
    L = __fma_rn(d, h, g);
    double y = __hiloint2double(__double2hiint(h) + (1 << 20), __double2loint(h));     // 2 h
    double e = __fma_rn(-L, y, 1.0);
    y = __fma_rn(y, e, y);
    e = __fma_rn(-L, y, 1.0);
    rL = __fma_rn(y, e, y);
    const unsigned lo = (unsigned)(1023 - 700) << 20, span = (unsigned)1400 << 20;
    ok = ((unsigned)__double2hiint(x) - lo) < span && __double2loint(L) != -1;
}

}  // namespace bbpd
