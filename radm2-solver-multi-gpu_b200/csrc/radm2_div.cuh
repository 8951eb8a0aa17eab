// Divisions of the wide solver: by a number that divides many times over, and four at a time.
#pragma once

#include <cmath>
#include <cstring>

namespace radm2 {

static __device__ __noinline__ double div_exact(double a, double u) { return a / u; }

// Division by a number that divides many times over (the LU's pivots in reference arithmetic).
//
// With r = 1 / u rounded to nearest, formed once (CUDA's __drcp_rn), the quotient a / u takes one
// product and two fused multiply-adds: q0 = a r, then q0 + (a - u q0) r.  The result is the
// correctly rounded quotient, so the bits are those of a / u: P. W. Markstein, Computation of
// elementary functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34 (1990);
// N. Brisebarre, J.-M. Muller and S. K. Raina, Accelerating correctly rounded floating-point
// division when the divisor is known in advance, IEEE Trans. Computers 53 (2004).  That needs an
// exact remainder, hence operands and quotient away from the ends of the exponent range.
//
// Operands: any.  Zeros keep their sign; what could leave the range is divided plainly.  The wide
// solver in reference arithmetic, 8,191 cells of one step: 12.1 ms, 19.5 with a / u throughout.

// The reciprocal for div_pivot: NaN for a pivot that is negative (backward integration, negative
// states) or outside 2^-100 .. 2^100; its quotients are divided plainly.
__device__ __forceinline__ double rcp_pivot(double u)
{
    const unsigned h = (unsigned)__double2hiint(u);
    return h - 0x39b00000u <= 0x46300000u - 0x39b00000u ? __drcp_rn(u) : __hiloint2double(0x7ff80000, 0);
}

// A double's upper half as a float: magnitudes compare as the doubles' exponents do, sign off by the
// operand's own modifier (the halves of NaN and of anything beyond 2^1017 compare as too large).
__device__ __forceinline__ float upper(double a)
{
    const int h = __double2hiint(a);
    float f;
    memcpy(&f, &h, sizeof f);
    return f;
}

constexpr float PIVOT_MAX = 0x1.6p88f, PIVOT_MIN = 0x1.6p-87f;  // uppers of 2^700 and 2^-700

// a / u with r = rcp_pivot(u), called by all lanes of a warp together; limit: PIVOT_MAX, or -1 to
// divide plainly.  A numerator outside 2^-700 .. 2^700 (its quotient may leave 2^-800 .. 2^800) is
// divided plainly too, and the whole warp takes that branch, for the warp-collective instructions
// that follow it.  The check looks at the numerator, not at the quotient, so it is done by the time
// the quotient is (64 cells, one step: 11.57 ms, 11.70 otherwise), and is three comparisons that
// pass one predicate on (65,536 cells 50.7 ms, 52.2 with integer operations on the upper half).
// Zero multipliers are common (a rate that is zero at night) and stay on the short path: the
// remainder is taken as u q0 - a, a +0 then, so that the correction is -0 and a zero q0 keeps its
// sign.
__device__ __forceinline__ double div_pivot(double a, double u, double r, float limit)
{
    const double q0 = a * r;
    double q = fma(-fma(u, q0, -a), r, q0);
    const float f = fabsf(upper(a));
    const bool plain = (f < PIVOT_MIN && a != 0.0) || !(f <= limit);
    if (__any_sync(0xffffffffu, plain)) {
        const double e = div_exact(a, u);
        if (plain) q = e;
    }
    return q;
}
__device__ __forceinline__ double div_pivot(double a, double u, double r)
{
    return div_pivot(a, u, r, r != r ? -1.0f : PIVOT_MAX);
}

// Four quotients of non-negative numbers with one division: the reciprocal of the denominators'
// product, times the other denominators, is each one's own (simultaneous inversion: P. L.
// Montgomery, Speeding the Pollard and elliptic curve methods of factorization, Math. Comp. 48
// (1987)).  It is six roundings off at most, so a product with it is seven off; the remainder corrects
// the quotient to within 2^-47 ulp before its last rounding.  So the bits are those of a / u unless
// the quotient lies that close to the middle of two neighbours.  Denominators outside 2^-200 .. 2^200
// and numerators outside 2^-700 .. 2^700 (but zero) are divided plainly.
__device__ __forceinline__ void div_four(const double (&a)[4], const double (&u)[4], double (&q)[4])
{
    const double u01 = u[0] * u[1], u23 = u[2] * u[3];
    const double r = 1.0 / (u01 * u23);
    const double r01 = r * u23, r23 = r * u01;
    const double rj[4] = {r01 * u[1], r01 * u[0], r23 * u[3], r23 * u[2]};
    bool plain = false;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        q[j] = a[j] * rj[j];
        q[j] = fma(fma(-u[j], q[j], a[j]), rj[j], q[j]);
        const unsigned ha = (unsigned)__double2hiint(a[j]), hu = (unsigned)__double2hiint(u[j]);
        plain = plain || hu - 0x33700000u > 0x4c700000u - 0x33700000u ||
                (ha - 0x14300000u > 0x6bb00000u - 0x14300000u && a[j] != 0.0);
    }
    if (plain) {
#pragma unroll
        for (int j = 0; j < 4; j++) q[j] = div_exact(a[j], u[j]);
    }
}

}  // namespace radm2
