// mph_exact.cuh — correctly rounded FP64 arithmetic helpers for the
// bit-exact FP64 form.
#pragma once

namespace mph {

// Round-to-nearest quotient x/y from yi = RN(1/y), by Markstein's method
// (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34(1), 1990; see also Muller et
// al., Handbook of Floating-Point Arithmetic, the FMA-based division
// chapter): start from q0 = RN(x*yi), then twice form the exact remainder
// r = x - q*y with one FMA and correct q += r*yi.  The first correction
// brings q within half an ulp plus a tiny term, the second (Markstein's
// step) yields RN(x/y).  Valid for finite, normal operands without overflow
// or underflow of the intermediates, which is the range the pair kernels use
// (lengths between ~1e-9 and ~1e3 m, forces far from the double limits); a
// zero numerator returns x*yi, i.e. a zero with the IEEE sign.  The FP64
// kernels call this where the reference divides, and
// mph_check_exact_division() compares it bit for bit with the hardware
// IEEE division on random and adversarial operands.
__device__ __forceinline__ double div_rn(double x, double y, double yi) {
    double q = x * yi;
    double r = __fma_rn(-q, y, x);
    q = __fma_rn(r, yi, q);
    r = __fma_rn(-q, y, x);
    q = __fma_rn(r, yi, q);
    return x == 0.0 ? x * yi : q;
}

// A divisor's reciprocal for div_q: y + l = 1/divisor to about 2^-102 relative
// (l a small correction of y), h = the same rounded to FP64.
struct Recip {
    double y, l, h;
};

// The Recip of a constant divisor d from h = RN(1/d) and l = (1 - d h) h, both
// evaluated on the host with one fused multiply-add (make_simconst).
__device__ __forceinline__ Recip recip_const(double h, double l) { return {h, l, h}; }

// RN(x/d) in four operations: q = x y + x l is x/d rounded once, but for an
// error of 2^-49 ulp, hence faithful; its remainder m = x - q d is then exact, and
// q + m h rounds to RN(x/d) by Markstein's theorem (as in div_rn, whose first
// correction this replaces).  The theorem's bound holds with that 2^-49 for
// every divisor whose significand is below 2^53 - 8 units, and for the larger
// ones when h is RN(1/d) and l its remainder, as recip_const and sqrt_recip_any
// give them.  mph_check_exact_division() compares it with the hardware division
// on the (x, d) whose quotient is nearest to the middle of two doubles and on
// random operands.  A zero numerator gives a zero of either sign, and every such
// quotient reaches the state only through products and sums that start at +0.0
// and can never hold -0.0 (+0 + -0 = +0, and an exact cancellation rounds to
// +0), so adding a zero of either sign leaves them unchanged.
__device__ __forceinline__ double div_q(double x, double d, const Recip& c) {
    const double q = __fma_rn(x, c.y, x * c.l);
    const double m = __fma_rn(-q, d, x);
    return __fma_rn(m, c.h, q);
}

// r = RN(sqrt(a)) and the Recip of r together, for an a that plain_root() takes.  The
// hardware's approximation of 1/sqrt(a) takes one third-order step of the
// Householder family, y (1 + e/2 + 3/8 e^2) with e = 1 - a y^2 (from 2^-20 to about
// 2^-52.4), g = a y is within three ulps of sqrt(a), and Markstein's
// correction g + (a - g^2) y/2 rounds it: its error before rounding is below
// 2^-49 ulp, so only an a whose root lies that close to the middle of two
// doubles could round wrongly; those (a 2^54 = M^2 - k for an odd M and |k| < 80, 40
// significands) are compared with the hardware square root by
// mph_check_exact_division(), with random ones.  The same y then serves 1/r,
// which the separate square root and reciprocal would compute anew: with div_q's
// shorter division the force sweep's FP64 operations per list entry went from about
// 100 to 84, 2.90 -> 2.60 ms on the 2,779,256-particle dam break.
__device__ __forceinline__ void sqrt_recip(double a, double& r, Recip& c) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = __fma_rn(-(a * y), y, 1.0);
    y = __fma_rn(y, e * __fma_rn(e, 0.375, 0.5), y);
    const double g = a * y;
    const double half_y = __hiloint2double(__double2hiint(y) - 0x100000, __double2loint(y));
    r = __fma_rn(__fma_rn(-g, g, a), half_y, g);
    const double f = __fma_rn(-r, y, 1.0);
    c.y = y;
    c.l = y * f;
    c.h = __fma_rn(y, f, y);
}
// The same for any other a (coincident particles among them), by the hardware
// operations; a = 0 gives an infinite reciprocal and NaN quotients, as the
// reference's 0/0.
__device__ __forceinline__ void sqrt_recip_any(double a, double& r, Recip& c) {
    r = sqrt(a);
    c.y = c.h = __drcp_rn(r);
    c.l = __fma_rn(-r, c.h, 1.0) * c.h;
}
// a >= 2^-400 (squared distances are below 2^400), and the upper 20 bits of
// its significand not all ones: then the root's significand is below 2^53 - 8.
__device__ __forceinline__ bool plain_root(double a) {
    const int hi = __double2hiint(a);
    return hi >= ((1023 - 400) << 20) && (hi & 0xFFFFF) != 0xFFFFF;
}

}  // namespace mph
