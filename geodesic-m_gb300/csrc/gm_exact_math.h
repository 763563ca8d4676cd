/* gm_exact_math.h — exact-rounding helpers shared by the kernels and by the
 * CPU test that checks them (tests/test_exact_arithmetic.py compiles this
 * header as C11 with gcc).
 *
 * gm_f2fix:  round(v * 2^40) to the nearest integer, ties to even, for
 *            |v| < 2^22, from the bits of v with integer operations only (the
 *            value of __float2ll_rn(v * 2^40); the 64-bit conversion
 *            instruction is slow on this part).
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
 * gm_abs_ge: |v| >= t for a positive finite t, by integer comparison of the
 *            bits (an FP64 comparison occupies the FP64 pipe like any other
 *            FP64 instruction); false for a NaN.
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
#ifdef __CUDA_ARCH__
    const unsigned int b = __float_as_uint(v);
#else
    unsigned int b;
    memcpy(&b, &v, sizeof b);
#endif
    const int e = (int)((b >> 23) & 0xffu);
    const long long m = (long long)((b & 0x7fffffu) | 0x800000u);
    const int sh = e - 150 + 40; /* |v| * 2^40 = m * 2^sh for normal v */
    long long r;
    if (e == 0 || sh < -25) {
        r = 0; /* below 2^-41: rounds to zero */
    } else if (sh >= 0) {
        r = m << sh;
    } else {
        const int s = -sh;
        const long long q = m >> s, rem = m & ((1ll << s) - 1), half = 1ll << (s - 1);
        r = q + ((rem > half || (rem == half && (q & 1))) ? 1 : 0);
    }
    return (b >> 31) ? -r : r;
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
