/*
 * The divisions of the plain-FP64 gradients, for device code and for host-side
 * tests of the same source: a quotient by a stored reciprocal (sfx_div_by) and
 * the slope limiter's quotients.
 *
 * The slope limiter's quotient for one face, plain-FP64 gradients
 * (VorCell::estimate_gradient, src/VorCell.cpp:486-530).
 *
 * The reference forms q1 = a / dp and q2 = b / dp with a = W_max - W and
 * b = W_min - W (q1 = q2 = 1 where dp == 0) and keeps mx = (q1 < q2) ? q2 : q1.
 * sfx_limiter_ratio returns the same value bit for bit with one division
 * where the signs decide the select: for finite a >= 0 >= b and finite
 * dp > 0, q1 >= +0 >= q2 (b = +0 gives q2 = +0, which does not compare below
 * q1), so mx = q1; for finite dp < 0, q1 <= -0 and q2 >= -0, so mx = q2
 * unless q2 is zero, where q1 is zero too and the select keeps q1.  Any
 * other input (dp == 0, a non-finite or misordered operand) takes the
 * reference's two divisions.
 */
#pragma once

#include <math.h>

#if defined(__CUDACC__)
#define SFX_LIM_HD __host__ __device__ __forceinline__
#else
#define SFX_LIM_HD static inline
#endif

/* a / b from y = 1 / b (rounded to nearest): two corrections of a y, the
 * second of them with an exact residual of a quotient within an ulp, give the
 * correctly rounded quotient (P. Markstein, "Computation of elementary
 * functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990)
 * where nothing under- or overflows; a zero quotient may lose its sign */
SFX_LIM_HD double sfx_div_by(double a, double b, double y) {
    double q = a * y;
    q = fma(fma(-q, b, a), y, q);
    return fma(fma(-q, b, a), y, q);
}

/* the reference's two divisions and select */
SFX_LIM_HD double sfx_limiter_ratio_ref(double a, double b, double dp) {
    double q1 = a, q2 = b;
    if(dp != 0.) {
        q1 = q1 / dp;
        q2 = q2 / dp;
    } else {
        q1 = 1.;
        q2 = 1.;
    }
    return (q1 < q2) ? q2 : q1;
}

SFX_LIM_HD double sfx_limiter_ratio(double a, double b, double dp) {
    const double big = 1.7976931348623157e308;
    const bool fin = a >= 0. && a <= big && b <= 0. && b >= -big && fabs(dp) <= big;
    if(fin && dp > 0.) return a / dp;
    if(fin && dp < 0.) {
        const double q2 = b / dp;
        if(q2 != 0.) return q2;
        const double q1 = a / dp;
        return (q1 < q2) ? q2 : q1;
    }
    return sfx_limiter_ratio_ref(a, b, dp);
}

/*
 * The minimum over a cell's faces of 1 and those quotients, with two
 * divisions.  For dp > 0 the quotient is a / dp, smallest where dp is
 * largest, and rounding is monotonic, so the minimum over those faces is
 * a / dmax rounded; for dp < 0 it is b / dp, smallest at dmin.  dmax and dmin
 * are the largest positive and smallest negative dp (0: none), `first` the sign
 * of the first dp that is neither 0 nor NaN in the reference's face order
 * (which of a +0 and a -0 quotient it keeps: the first).  For a, b, dmax and
 * dmin finite and far from under- and overflow.
 */
SFX_LIM_HD double sfx_limiter_min(double a, double b, double dmax, double dmin, int first) {
    double alpha = 1.;
    if(dmax > 0.) {
        const double q = a / dmax;
        alpha = (q < alpha) ? q : alpha;
    }
    if(dmin < 0.) {
        const double q = b / dmin;
        alpha = (q < alpha) ? q : alpha;
        if(b == 0. && (a != 0. || first < 0)) alpha = q; /* -0 */
    }
    return alpha;
}
