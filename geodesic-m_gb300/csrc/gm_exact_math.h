/* gm_exact_math.h — exact-rounding helpers shared by the kernels and by the
 * CPU test that checks them (tests/test_exact_arithmetic.py compiles this
 * header as C11 with gcc).
 *
 * gm_f2fix:  round(v * 2^40) to the nearest integer, ties to even, for
 *            |v| < 2^22: the value of __float2ll_rn(v * 2^40), whose 64-bit
 *            conversion runs on the FP64 pipe of this part, from two 32-bit
 *            conversions (8 instructions; shifting the bits of v took ~25).
 * gm_div_by_dt: num / dt correctly rounded from y = RN(1 / dt), computed once:
 *            Markstein's correction (P. Markstein, "IA-64 and Elementary
 *            Functions", 2000): q = RN(num y), r = num - q dt is exact in one
 *            FMA, and RN(q + r y) is the correctly rounded quotient when y is
 *            the correctly rounded reciprocal (away from overflow and
 *            underflow).  Three FP64 operations instead of a division.
 * gm_div_rcp: num / den correctly rounded from y = RN(1 / den), the same
 *            correction for any den of ordinary size (2^-200 to 2^200, the
 *            caller's to see); a numerator that is zero, tiny or huge takes
 *            the division.
 * gm_rsqrt_step: 1 / sqrt(x) from a seed y within 2^-22 of it: one step of
 *            Chebyshev's third-order method (J. F. Traub, "Iterative Methods for
 *            the Solution of Equations", 1964) for y^-2 - x, which is
 *            y (1 + e/2 + 3 e^2/8) with e = 1 - x y^2.  |e| < 2^-20.9, so the
 *            next term of the series, 5/16 e^3, is below 2^-64; the rounding of
 *            x y moves the result by half an ulp at most, its own rounding by
 *            another half.
 * gm_abs_ge: |v| >= t for a positive finite t, by integer comparison of the
 *            bits (an FP64 comparison occupies the FP64 pipe like any other
 *            FP64 instruction); false for a NaN.
 * gm_moved_far: d2 >= far_sq for a squared distance d2 >= 0 and far_sq >= 0,
 *            rounded towards yes (the high words, no FP64 comparison); a NaN of
 *            either sign counts as far.
 * gm_min_image: d - L round(d / L), round half away from zero, each operation
 *            rounded on its own: the reference's min_image
 *            (neighbor.rs:74-76).  Away from |d| = L/2 the rounded quotient
 *            is known without the division: 0 below it, +-1 between L/2 and
 *            1.4 L, so the value is d, or d -+ L rounded once; both tests
 *            are integer comparisons of the high words, 0.4 % clear of L/2.
 *            An FP64 division and round are ~20 operations of a pipe with
 *            1/64 of the FP32 rate (the divisions were a third of the FP64
 *            pair kernel in a periodic box).  The value is the general
 *            expression's for every d (a zero may differ in its sign).
 */
#ifndef GM_EXACT_MATH_H
#define GM_EXACT_MATH_H

#include <math.h>
#include <string.h>

#ifdef __CUDACC__
#define GM_HD __host__ __device__ __forceinline__
#else
#define GM_HD static inline
#endif

GM_HD long long gm_f2fix(float v) {
    /* k1 = round(v 2^9) and r = v - k1 2^-9 exactly: below 2^24 k1 is an FP32
     * number, from there on v 2^9 is an integer and r is 0.  |r 2^40| <= 2^30,
     * and k1 2^31 is even, so a tie of r is the tie of v. */
#ifdef __CUDA_ARCH__
    const int k1 = __float2int_rn(__fmul_rn(v, 512.f));
    const float r = __fmaf_rn((float)k1, -1.f / 512.f, v);
    const int k2 = __float2int_rn(__fmul_rn(r, 1099511627776.f));
#else
    const int k1 = (int)nearbyintf(v * 512.f);
    const float r = fmaf((float)k1, -1.f / 512.f, v);
    const int k2 = (int)nearbyintf(r * 1099511627776.f);
#endif
    return ((long long)k1 << 31) + k2;
}

GM_HD int gm_hi_word(double v) {
#ifdef __CUDA_ARCH__
    return __double2hiint(v);
#else
    unsigned long long b;
    memcpy(&b, &v, sizeof b);
    return (int)(unsigned)(b >> 32);
#endif
}

GM_HD double gm_div_by_dt(double num, double dt, double y) {
    const double q = num * y;
    const double r = fma(-q, dt, num);
    return fma(r, y, q);
}

GM_HD int gm_ordinary(double v) { /* 2^-200 to 2^200 */
    return (unsigned)((gm_hi_word(v) & 0x7fffffff) - ((1023 - 200) << 20)) < (unsigned)(400 << 20);
}

GM_HD double gm_div_rcp(double num, double den, double y) {
    /* |num| in [2^-700, 2^700) */
    if ((unsigned)((gm_hi_word(num) & 0x7fffffff) - ((1023 - 700) << 20)) >= (unsigned)(1400 << 20)) return num / den;
    return gm_div_by_dt(num, den, y);
}

GM_HD double gm_rsqrt_step(double x, double y) {
    const double e = fma(-(x * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

GM_HD int gm_abs_ge(double v, double t) {
#ifdef __CUDA_ARCH__
    const unsigned long long b = (unsigned long long)__double_as_longlong(v), tb = (unsigned long long)__double_as_longlong(t);
#else
    unsigned long long b, tb;
    memcpy(&b, &v, sizeof b);
    memcpy(&tb, &t, sizeof tb);
#endif
    const unsigned long long a = b & 0x7fffffffffffffffull;
    return a >= tb && a <= 0x7ff0000000000000ull;
}

GM_HD int gm_moved_far(double d2, double far_sq) {
    return (unsigned)gm_hi_word(d2) >= (unsigned)gm_hi_word(far_sq);
}

GM_HD double gm_min_image(double d, double L) {
    const int hd = gm_hi_word(d) & 0x7fffffff, hl = gm_hi_word(L);
    if (hd < hl - 0x101000) return d; /* |d| < L/2 (1 - 2^-8) */
#ifdef __CUDA_ARCH__
    if (hd > hl - 0xff000 && hd < hl + 0x70000) return __dsub_rn(d, copysign(L, d));
    return __dsub_rn(d, __dmul_rn(L, round(__ddiv_rn(d, L))));
#else
    if (hd > hl - 0xff000 && hd < hl + 0x70000) return d - copysign(L, d);
    return d - L * round(d / L);
#endif
}

#endif
