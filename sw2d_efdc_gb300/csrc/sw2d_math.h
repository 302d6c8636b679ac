/* Device-side FP64 helpers of the SW2D step, shared verbatim by the CUDA
 * kernels and by the CPU oracle's "device math" flavour so that the two
 * perform the same IEEE operations in the same order (compile without FMA
 * contraction on both sides: nvcc --fmad=false, gcc -ffp-contract=off).
 *
 * Only +, -, *, /, sqrt and fma appear here; all are correctly rounded in
 * IEEE binary64/binary32 on the host and on the GPU, so results are
 * bit-identical across the two.
 *
 * The reference evaluates the Manning friction factor as
 *     ram = gg*rn*rn*sqx / pow(hm, 1.3333330)        (SW2D-EFDC.cu:193-195, :310-312)
 * On GB300 the FP64 pipe is ~1/64 of the FP32 rate, so the library pow
 * (an extended-precision log/exp) dominates the FP64 step.  sw2d_rpow_manning()
 * returns hm^-1.333333 to a few ulp from a short published construction,
 * evaluated in pairs of binary32 numbers (only two binary64 additions):
 *   - x^(-1/3) by Newton's iteration for f(r) = x r^3 - 1 in binary32, seeded
 *     by the exponent-scaling bit trick (Blinn, "Floating-point tricks",
 *     IEEE CG&A 1997);
 *   - x^(-4/3) = r^4 (1 - e)^(-4/3), e = 1 - x r^3, by its binomial series
 *     to second order in binary64;
 *   - the residual exponent d = 1.333333 - 4/3 (|d| = 3.3e-7) as
 *     x^(-d) = exp(-d ln x) ~ 1 + t + t^2/2, t = -d ln x, with ln x from the
 *     atanh series ln m = 2 atanh((m-1)/(m+1)) on m in [sqrt(1/2), sqrt(2))
 *     in binary32 (t needs ln x to 1e-6 only).
 * The result is within 3e-13 relative of libm pow, far inside what the step's
 * 1e-9 m agreement with the reference needs; the test suite checks both.
 */
#ifndef SW2D_MATH_H
#define SW2D_MATH_H

#include <stdint.h>
#include <string.h>
#include <math.h>

#if defined(__CUDACC__)
#define SW2D_HD __host__ __device__ __forceinline__
#else
#define SW2D_HD static inline
#endif

/* Index of the series entry in force at `time` (one entry every dts
 * seconds), clamped to n, the first entry of the series' zero tail, and to
 * the first entry (a clock that starts before time 0): the reference's
 * int(time / dts) (SW2D-EFDC.cu:537, :550) without reading outside the
 * series.  The clamps are decided on the quotient f = time / dts, so one
 * beyond the int range (a long run with a short series interval) clamps
 * instead of converting out of range. */
SW2D_HD int sw2d_series_entry(double f, int n) {
#if defined(__CUDA_ARCH__)
    /* the conversion saturates, and of NaN gives 0 or the least int; the clamps
     * are integer ones (10.0 us an iteration at 33 x 41, 10.1 with one in
     * binary64) */
    const int it = (int)f;
    return it >= n ? n : it > 0 ? it : 0;
#else
    return f >= (double)n ? n : f > 0.0 ? (int)f : 0;
#endif
}
SW2D_HD int sw2d_series_index(double time, double dts, int n) { return sw2d_series_entry(time / dts, n); }

/* 1.3333330 - 4/3 evaluated exactly (binary64 value of 1.3333330 minus the
 * real 4/3), then rounded to binary64. */
#define SW2D_POW_RESIDUAL (-3.3333333323189623e-07)

SW2D_HD uint32_t sw2d_f32_bits(float f) {
#if defined(__CUDA_ARCH__)
    return (uint32_t)__float_as_uint(f);
#else
    uint32_t u;
    memcpy(&u, &f, sizeof u);
    return u;
#endif
}

SW2D_HD float sw2d_f32_from_bits(uint32_t u) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float f;
    memcpy(&f, &u, sizeof f);
    return f;
#endif
}

/* On the device the bits pass through an instruction the optimiser does not
 * look into: it otherwise recognises integer comparisons and zero tests of
 * them as binary64 ones (and "zero ? 0 : x" as x + 0) and puts them back on
 * the FP64 pipe. */
SW2D_HD uint64_t sw2d_f64_bits(double d) {
#if defined(__CUDA_ARCH__)
    uint64_t u;
    asm("mov.b64 %0, %1;" : "=l"(u) : "d"(d));
    return u;
#else
    uint64_t u;
    memcpy(&u, &d, sizeof u);
    return u;
#endif
}

SW2D_HD double sw2d_f64_from_bits(uint64_t u) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)u);
#else
    double d;
    memcpy(&d, &u, sizeof d);
    return d;
#endif
}

/* ---- exact binary64 comparisons and power-of-two scalings on the bits ----
 * GB300 executes binary64 arithmetic at 1/64 of the binary32 rate, so the
 * FP64 step moves every comparison, zero test, maximum with zero and
 * multiplication by 1/2 or 1/4 off the FP64 pipe into integer operations on
 * the bit patterns.  Each helper returns the IEEE result for every non-NaN
 * operand (subnormals, signed zeros and infinities included). */

/* a signed integer with the order of the doubles (-0 and +0 map to 0) */
SW2D_HD int64_t sw2d_ord(double x) {
    const int64_t s = (int64_t)sw2d_f64_bits(x);
    return s >= 0 ? s : -(s & INT64_MAX);
}
/* the double of sw2d_ord's value (+0 for both zeros) */
SW2D_HD double sw2d_f64_of_ord(int64_t o) {
    return sw2d_f64_from_bits(o >= 0 ? (uint64_t)o : ((uint64_t)0 - (uint64_t)o) | 0x8000000000000000ULL);
}
SW2D_HD int sw2d_lt(double a, double b) { return sw2d_ord(a) < sw2d_ord(b); }
SW2D_HD int sw2d_gt(double a, double b) { return sw2d_ord(a) > sw2d_ord(b); }
SW2D_HD int sw2d_le(double a, double b) { return sw2d_ord(a) <= sw2d_ord(b); }
SW2D_HD int sw2d_ge(double a, double b) { return sw2d_ord(a) >= sw2d_ord(b); }
SW2D_HD int sw2d_gt0(double x) { return (int64_t)sw2d_f64_bits(x) > 0; }                 /* x > 0 */
SW2D_HD int sw2d_lt0(double x) { return sw2d_f64_bits(x) > 0x8000000000000000ULL; }       /* x < 0 */
SW2D_HD int sw2d_is0(double x) { return (sw2d_f64_bits(x) << 1) == 0; }                   /* x == 0 */
/* max(x, 0) with +0 for every x <= 0 */
SW2D_HD double sw2d_max0(double x) { return (int64_t)sw2d_f64_bits(x) > 0 ? x : 0.0; }

/* x * 2^-k for 1 <= k <= 31, correctly rounded: an exponent decrement while the
 * result stays normal, else the magnitude shifted right with
 * round-half-to-even (the subnormal result of the IEEE product). */
SW2D_HD double sw2d_scale_down(double x, int k) {
    const uint64_t b = sw2d_f64_bits(x);
    const uint64_t sign = b & 0x8000000000000000ULL, mag = b & 0x7fffffffffffffffULL;
    const uint64_t e = mag >> 52;
    if (e == 0x7ff) return x;                                   /* inf, NaN */
    if (e > (uint64_t)k) return sw2d_f64_from_bits(b - ((uint64_t)k << 52));
    /* result subnormal (or zero): the significand m counts units of 2^-1074
     * (of 2^(e - 1 - 1074) for e >= 1), so the result is m / 2^s rounded */
    uint64_t m = (e == 0) ? mag : (mag & 0x000fffffffffffffULL) | 0x0010000000000000ULL;
    uint32_t s = (uint32_t)k;
    if (e != 0) {
        if (k <= 2) m <<= e - 1; /* shorter where k is known (a step at 33 x 41 10.0 us, 10.2 without) */
        else s = (uint32_t)k + 1u - (uint32_t)e;
    }
    const uint64_t q = m >> s, rem = m & ((1ULL << s) - 1), halfw = 1ULL << (s - 1);
    const uint64_t r = q + ((rem > halfw || (rem == halfw && (q & 1))) ? 1 : 0);
    return sw2d_f64_from_bits(sign | r);
}
/* x/2 and x/4 as used by the step.  On the device an exponent decrement
 * when the result stays normal, x itself when it is zero, and the shift of
 * sw2d_scale_down for the rest (all exact; no binary64 instruction on any
 * path: one that is predicated off still takes its 71 cycles); the host
 * evaluates the product. */
#if defined(__CUDACC__)
__device__ __forceinline__ double sw2d_pow2_down(double x, int k, double m) { /* m = 2^-k, k >= 1 */
#if defined(__CUDA_ARCH__)
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    const uint32_t e = hi & 0x7ff00000u, kk = (uint32_t)k << 20;
    if (e - (kk + 0x00100000u) < 0x7fe00000u - kk) return __hiloint2double((int)(hi - kk), (int)lo);
    if (((hi << 1) | lo) == 0u) return x;
    return sw2d_scale_down(x, k);
#else
    return x * m;
#endif
}
__device__ __forceinline__ double sw2d_half(double x) { return sw2d_pow2_down(x, 1, 0.5); }
__device__ __forceinline__ double sw2d_quarter(double x) { return sw2d_pow2_down(x, 2, 0.25); }
#else
static inline double sw2d_half(double x) { return x * 0.5; }
static inline double sw2d_quarter(double x) { return x * 0.25; }
#endif
/* x > t for a positive threshold t (non-NaN x): one integer comparison */
SW2D_HD int sw2d_gt_pos(double x, double t) { return (int64_t)sw2d_f64_bits(x) > (int64_t)sw2d_f64_bits(t); }
SW2D_HD int sw2d_lt_pos(double x, double t) { return (int64_t)sw2d_f64_bits(x) < (int64_t)sw2d_f64_bits(t); }
SW2D_HD int sw2d_ge_pos(double x, double t) { return (int64_t)sw2d_f64_bits(x) >= (int64_t)sw2d_f64_bits(t); }
SW2D_HD int sw2d_le_pos(double x, double t) { return (int64_t)sw2d_f64_bits(x) <= (int64_t)sw2d_f64_bits(t); }

SW2D_HD double sw2d_fma(double a, double b, double c) { return fma(a, b, c); }
SW2D_HD float sw2d_fmaf(float a, float b, float c) { return fmaf(a, b, c); }

/* ---- conversions between binary32 and binary64 on the integer pipes ----
 * On GB300 a conversion between binary32 and binary64, or between a 64-bit
 * integer and binary32, runs on the FP64 pipe at the binary64 rate (a
 * micro-benchmark: about one binary64 addition each).  These build the
 * result from the bit pattern instead. */

/* (double)f, exact, by integer operations and, for a subnormal, an exact
 * binary32 scaling by 2^64 */
SW2D_HD double sw2d_f64_of_f32(float f) {
    const uint32_t b = sw2d_f32_bits(f);
    const uint32_t e = (b >> 23) & 0xffu;
    const uint64_t sign = (uint64_t)(b & 0x80000000u) << 32;
    if (e - 1u < 0xfeu)
        return sw2d_f64_from_bits(sign | ((uint64_t)(e + 896u) << 52) | ((uint64_t)(b & 0x7fffffu) << 29));
    if ((b & 0x7fffffffu) == 0u) return sw2d_f64_from_bits(sign);
    if (e == 0xffu) return sw2d_f64_from_bits(sign | 0x7ff0000000000000ULL | ((uint64_t)(b & 0x7fffffu) << 29));
    const uint32_t n = sw2d_f32_bits(f * 18446744073709551616.0f);
    return sw2d_f64_from_bits(sign | ((uint64_t)(((n >> 23) & 0xffu) + 832u) << 52) | ((uint64_t)(n & 0x7fffffu) << 29));
}

/* an estimate of (float)x for the binary32 prefilters: the significand
 * truncated to 24 bits (relative error below 2^-23); magnitudes below the
 * binary32 normal range give 0, above it infinity.  No path holds a hardware
 * conversion: predicated off, it would still take its 71 cycles of the FP64
 * pipe. */
SW2D_HD float sw2d_f32_est_of_f64(double x) {
    const uint64_t b = sw2d_f64_bits(x);
    const uint32_t hi = (uint32_t)(b >> 32), lo = (uint32_t)b;
    const uint32_t e = (hi >> 20) & 0x7ffu;
    uint32_t r = (hi & 0x80000000u) | ((e - 896u) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29);
    if (e < 897u) r = 0u;
    if (e > 1150u) r = (hi & 0x80000000u) | ((b << 1) > 0xffe0000000000000ULL ? 0x7fc00000u : 0x7f800000u);
    return sw2d_f32_from_bits(r);
}

/* The same from the high word alone, for the prefilters that run on every
 * cell: the significand truncated to 21 bits (relative error below 2^-20),
 * magnitudes below 2^-126 within 2^-126, 2^128 and above (infinities and NaN
 * too) infinity. */
SW2D_HD float sw2d_f32_est_hi(double x) {
    const uint32_t hi = (uint32_t)(sw2d_f64_bits(x) >> 32);
    uint32_t a = hi & 0x7fffffffu;
    a = a < 0x47f00000u ? a : 0x47f00000u;
    a = a > 0x38000000u ? a : 0x38000000u;
    return sw2d_f32_from_bits((hi & 0x80000000u) | (a - 0x38000000u) << 3);
}

/* The estimates hold for parameters of a run (threshold, gravity,
 * spacings) in this range; with others every value is evaluated in binary64. */
SW2D_HD int sw2d_est_range(double x) { return x >= 1e-30 && x <= 1e30; }
#define SW2D_EST_MOST 1e30f /* speeds up to here are compared by their estimates */

/* "depth h - dt2 ((qs - qn) rdx + (qe - qw) rdy - src), or 0 if that is
 * negative, < th" from sw2d_f32_est_hi of the binary64 values (src, dt2 and
 * the spacings truncated or rounded to binary32; srcmag: the magnitudes that
 * src is the sum of): 0 or 1, or 2 where th lies within the estimate's error
 * (2^-17 of the magnitudes that enter it; their truncation to 21 bits and the
 * estimate's own rounding stay below 2^-18 of them) or an infinity or NaN
 * takes part.  For values of sw2d_est_range's parameters; with others pass a NaN th. */
SW2D_HD int sw2d_dry_est(float h, float qn, float qs, float qw, float qe, float src, float srcmag, float dt2, float rdx,
                         float rdy, float th) {
    const float hs = h - dt2 * ((qs - qn) * rdx + (qe - qw) * rdy - src);
    const float mag =
        fabsf(h) + dt2 * ((fabsf(qs) + fabsf(qn)) * rdx + (fabsf(qe) + fabsf(qw)) * rdy + srcmag) + th;
    const float d = hs - th;
    if (!(fabsf(d) > 7.6293945e-6f * mag + 1e-35f) || !(mag < 1e37f)) return 2;
    return d < 0.f ? 1 : 0;
}

/* A depth's estimate for a sum with another's: as above for depths that are
 * not negative, infinity for all others (an estimate of the mean of two depths
 * of opposite sign would have no relative error; NaN counts with them) and
 * from 2^128. */
SW2D_HD float sw2d_f32_est_depth(double x) {
    uint32_t a = (uint32_t)(sw2d_f64_bits(x) >> 32);
    a = a < 0x47f00000u ? a : 0x47f00000u;
    a = a > 0x38000000u ? a : 0x38000000u;
    return sw2d_f32_from_bits((a - 0x38000000u) << 3);
}

/* an estimate of (float)v for a 32-bit unsigned v (relative error below
 * 2^-22): v = hi 2^16 + lo, each half exact in binary32 by the 2^23
 * magic-number construction */
SW2D_HD float sw2d_f32_est_of_u32(uint32_t v) {
    const float h = sw2d_f32_from_bits(0x4b000000u | (v >> 16)) - 8388608.0f;
    const float l = sw2d_f32_from_bits(0x4b000000u | (v & 0xffffu)) - 8388608.0f;
    return sw2d_fmaf(h, 65536.0f, l);
}

/* nearest integer to x for |x| < 2^22, by the 1.5 2^23 magic number */
SW2D_HD int32_t sw2d_i32_near_f32(float x) {
    return (int32_t)(sw2d_f32_bits(x + 12582912.0f) - 0x4b400000u);
}


/* a / d for a constant divisor d with rd = RN(1/d): one product and one
 * fma-based residual correction (Markstein's theorem: with rd = RN(1/d) the
 * corrected quotient is the correctly rounded a/d). */
SW2D_HD double sw2d_div_const(double a, double d, double rd) {
    if (sw2d_is0(a)) return 0.0; /* what the sequence below yields for +0 and -0 */
    double q = a * rd;
    double e = sw2d_fma(-q, d, a);
    return sw2d_fma(e, rd, q);
}

/* The same quotient on the integer pipes (the sequence above is three
 * binary64 operations, each 71 issue cycles of a GB300 warp): with md the
 * 53-bit significand of d, ed its biased exponent and rc = floor(2^115 / md),
 * the high half of (ma 2^11) rc is ma 2^62 / md less at most 2, so its top 56
 * bits are the 55 or 56 quotient bits or one less; the exact remainder
 * completes them and rounds.  Operands or quotients that are not normal take
 * the sequence above. */
typedef struct {
    double d, rd;
    uint64_t md, rc;
    uint32_t ed;
} sw2d_divisor;

static inline sw2d_divisor sw2d_divisor_of(double d) { /* d > 0, on the host */
    sw2d_divisor c;
    const uint64_t u = sw2d_f64_bits(d);
    c.d = d;
    c.rd = 1.0 / d;
    c.ed = (uint32_t)(u >> 52) & 0x7ffu;
    c.md = (u & ((1ull << 52) - 1ull)) | (1ull << 52);
    c.rc = (uint64_t)(((unsigned __int128)1 << 115) / c.md);
    if (c.ed == 0u || c.ed == 0x7ffu) c.ed = 0u; /* not normal: always the plain sequence */
    return c;
}

/* binary32 seed r ~ x^(-1/3) (relative error ~1e-7): exponent-halving bit
 * trick followed by four binary32 Newton steps r <- r + r (1 - x r^3) / 3. */
SW2D_HD float sw2d_rcbrt_seed(float xf) {
    float r = sw2d_f32_from_bits(0x54aaaaaau - sw2d_f32_bits(xf) / 3u);
    for (int i = 0; i < 4; i++) {
        float r3 = (r * r) * r;
        float e = sw2d_fmaf(-xf, r3, 1.0f);
        r = sw2d_fmaf(r * e, 1.0f / 3.0f, r);
    }
    return r;
}

/* ln(x) in binary32 for a positive normal binary64 x, absolute error below
 * 6e-7 for x in [1e-6, 1e6] and 4e-6 in [1e-30, 1e30] (half an ulp of the
 * binary32 result): the exponent k and the mantissa folded to
 * m in [sqrt(1/2), sqrt(2)) (truncated to 24 bits) by integer operations,
 * ln m = 2 atanh(s) with s = (m - 1)/(m + 1) to the s^9 term, and k ln 2 with
 * ln 2 split so that k ln2_hi is exact.  Only IEEE binary32 +, -, *, / and
 * fma appear, so host and device agree bit for bit. */
SW2D_HD float sw2d_ln_f32(double x) {
    const uint64_t b = sw2d_f64_bits(x);
    int k = (int)((b >> 52) & 0x7ff) - 1023;
    const uint32_t mant = (uint32_t)((b >> 29) & 0x7fffffu); /* top 23 mantissa bits */
    uint32_t mb;
    if (mant > 0x3504f3u) { /* m > sqrt(2): use m/2 in [0.707, 1) */
        k += 1;
        mb = mant | 0x3f000000u;
    } else {
        mb = mant | 0x3f800000u;
    }
    const float m = sw2d_f32_from_bits(mb);
    const float s = (m - 1.0f) / (m + 1.0f);
    const float z = s * s;
    float p = sw2d_fmaf(z, 1.0f / 9.0f, 1.0f / 7.0f);
    p = sw2d_fmaf(z, p, 1.0f / 5.0f);
    p = sw2d_fmaf(z, p, 1.0f / 3.0f);
    p = sw2d_fmaf(z, p, 1.0f);
    const float lnm = (2.0f * s) * p;
    const float kf = (float)k;
    return sw2d_fmaf(kf, 0.693145751953125f, sw2d_fmaf(kf, 1.428606820309417e-06f, lnm));
}

/* hm^(-1.3333330), the reciprocal of the reference's pow(hm, 1.3333330),
 * binary64 throughout: the form used outside the range of
 * sw2d_rpow_manning below.
 * With r0 the binary32 seed (exact in binary64, so r0^2 is exact) and
 * e = 1 - x r0^3, x^(-4/3) = r0^4 (1 - e)^(-4/3) = r0^4 (1 + 4e/3 + 14e^2/9 + O(e^3));
 * the residual exponent contributes x^(-d) = (1 + t + t^2/2), t = -d ln x,
 * |t| < 4e-6, with ln x from sw2d_ln_f32 (its 6e-7 error moves t by 2e-13);
 * both corrections are folded into one fma.  Relative error < 3e-13. */
SW2D_HD double sw2d_rpow_manning_f64(double x) {
    double r0 = (double)sw2d_rcbrt_seed((float)x);
    double r2 = r0 * r0;
    double w0 = r2 * r2;
    double e = sw2d_fma(-x, r2 * r0, 1.0);
    double a4 = e * sw2d_fma(e, 14.0 / 9.0, 4.0 / 3.0);
    double t = (-SW2D_POW_RESIDUAL) * (double)sw2d_ln_f32(x);
    double ft = t * sw2d_fma(t, 0.5, 1.0);
    double u = sw2d_fma(a4, ft, a4 + ft);
    return sw2d_fma(w0, u, w0);
}

/* hm^(-1.3333330) with the same construction carried in pairs of binary32
 * numbers (a value and its rounding error, Dekker's products by fma and
 * Knuth's TwoSum), so that only the last two additions run on the binary64
 * pipe (GB300: 1/64 of the binary32 rate):
 *   x = xh + xl split by integer operations (xh its leading 24 significand
 *   bits, exact in binary32);
 *   r0^2 = r2h + r2l and r0^4 exact or to 2^-48 relative by fma products;
 *   e = 1 - x r0^3 in one binary32 (|e| ~ 2^-21, absolute error ~2^-46);
 *   t = c ln x as a pair, c = 1.3333330 - 4/3 split into two binary32;
 *   u = (1 + 4e/3 + 14e^2/9)(1 + t + t^2/2) - 1 as the pair (s, ul);
 *   result w0 (1 + u) assembled in binary64 from three binary32 terms.
 * Relative error < 3e-13 of pow (the CPU test bounds it on 1e-4 <= x <=
 * 1e3); outside 2^-60 <= x < 2^61 the binary64 form above is used.  Only
 * IEEE binary32 +, -, *, fma, integer operations and exact conversions
 * appear, so host and device agree bit for bit. */
SW2D_HD double sw2d_rpow_manning(double x) {
    const uint64_t b = sw2d_f64_bits(x);
    const int ex = (int)((b >> 52) & 0x7ff);
    if (ex < 1023 - 60 || ex > 1023 + 60) return sw2d_rpow_manning_f64(x);
    const float xh = sw2d_f32_from_bits((uint32_t)((ex - 896) << 23) | (uint32_t)((b >> 29) & 0x7fffffu));
    const float xl = (float)(uint32_t)(b & 0x1fffffffu) * sw2d_f32_from_bits((uint32_t)(ex - 1075 + 127) << 23);
    const float r0 = sw2d_rcbrt_seed(xh);
    const float r2h = r0 * r0, r2l = sw2d_fmaf(r0, r0, -r2h);
    const float r3h = r2h * r0, r3l = sw2d_fmaf(r2h, r0, -r3h) + r2l * r0;
    const float P = xh * r3h;
    const float Pe = sw2d_fmaf(xh, r3h, -P);
    const float e = (1.0f - P) - (Pe + (xh * r3l + xl * r3h)); /* 1 - P is exact: P is within 2^-21 of 1 */
    const float a4 = e * sw2d_fmaf(e, 1.5555556f, 1.3333334f);
    const float ln = sw2d_ln_f32(x);
    const float th = 3.3333333249174757e-07f * ln;
    const float tl = sw2d_fmaf(3.3333333249174757e-07f, ln, -th) + 7.40148665436918e-16f * ln;
    const float fl = tl + 0.5f * th * th;
    const float s = th + a4; /* TwoSum(th, a4) */
    const float bb = s - th;
    const float ul = ((th - (s - bb)) + (a4 - bb)) + fl + a4 * th;
    const float w0h = r2h * r2h;
    const float w0l = sw2d_fmaf(r2h, r2h, -w0h) + 2.0f * r2h * r2l;
    const float ph = w0h * s;
    const float pl = sw2d_fmaf(w0h, s, -ph);
    const float rest = pl + w0l + w0h * ul + w0l * s;
    return sw2d_f64_of_f32(w0h) + (sw2d_f64_of_f32(ph) + sw2d_f64_of_f32(rest));
}

/* ------------------------------------------------------------------------
 * a / b correctly rounded (round to nearest even) with integer and binary32
 * operations only, for the GB300's FP64 pipe, which runs at 1/64 of the
 * binary32 rate: a binary64 division there costs about as much as fifteen
 * binary64 multiplies, while this long division runs on the integer and
 * binary32 pipes beside the step's other binary64 work.  For a and b normal
 * and a normal quotient (a zero dividend returns the signed zero, every other
 * case the hardware a / b), with ma, mb the 53-bit significands:
 *   - the digits of (ma - mb) 2^55 / mb in steps of 22, 22 and 11 bits, each
 *     estimated from the leading 32 bits of the signed running remainder
 *     times a binary32 reciprocal of mb and subtracted exactly (the remainder
 *     modulo 2^64).  Nothing corrects a digit but the next one: digits and
 *     remainders carry signs, so an estimate that is off leaves a remainder
 *     a few mb larger that the next digit takes up.  With the reciprocal off
 *     by up to 2^-19 (the tests force 2^-20) the first digit is within 10 of
 *     its value, the second within 100, the third within 0.3, |R| < 2^60;
 *   - the third digit is biased by 0.35 and rounded down, so it is at most
 *     the true one and less than 2 below it: one conditional subtraction
 *     makes Q = floor(ma 2^55 / mb), 55 or 56 bits, and the sticky bit
 *     R != 0 completes the rounding to 53 bits.
 * The signed digits leave no data-dependent loop: on a GB300 one warp issues
 * it in 127 cycles against 492 for a form that corrected every digit by
 * steps of mb, and its latency is a fifth.  Being the correctly rounded
 * quotient, the result is bit-identical to the IEEE division on any machine
 * (the CPU tests compare it with the host's division over every class of
 * operands). */
SW2D_HD float sw2d_rcp_est(float x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
#if defined(SW2D_TEST_EST_SCALE) /* tests: a seed as far off as the hardware approximation may be */
    return (1.0f / x) * (float)(SW2D_TEST_EST_SCALE);
#else
    return 1.0f / x;
#endif
#endif
}

SW2D_HD uint64_t sw2d_umulhi(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

/* floor(x) as an integer, |x| < 2^31 */
SW2D_HD int32_t sw2d_i32_floor_f32(float x) {
#if defined(__CUDA_ARCH__)
    return __float2int_rd(x);
#else
    return (int32_t)floorf(x);
#endif
}

/* the significand q 2^-(2+n) of a result whose leading bit sits at 2^(54+n),
 * rounded to 53 bits (nearest even; the sticky bit already or-ed into bit 0),
 * with the biased exponent e of the case n = 0 */
SW2D_HD double sw2d_round_pack(uint64_t q, uint32_t n, uint32_t e, uint64_t sign) {
    const uint32_t sh = 2u + n;
    const uint32_t rc = (2u << n) - 1u + ((uint32_t)(q >> sh) & 1u);
    /* the significand's leading bit carries into the exponent field; a
     * significand rounded up to 2^53 carries once more */
    return sw2d_f64_from_bits(sign + ((uint64_t)(e + n - 1u) << 52) + ((q + rc) >> sh));
}

SW2D_HD double sw2d_div_by(double a, const sw2d_divisor* c) {
    const uint64_t ua = sw2d_f64_bits(a);
    const uint32_t ea = (uint32_t)(ua >> 52) & 0x7ffu;
    const uint32_t e = ea - c->ed + 1022u;
    if (ea - 1u >= 0x7feu || c->ed == 0u || e - 1u >= 0x7fdu) return sw2d_div_const(a, c->d, c->rd);
    const uint64_t ma = (ua & ((1ull << 52) - 1ull)) | (1ull << 52);
    uint64_t Q = sw2d_umulhi(ma << 11, c->rc) >> 7;
    uint64_t R = (ma << 55) - Q * c->md;
    if (R >= c->md) {
        R -= c->md;
        Q += 1ull;
    }
    return sw2d_round_pack(Q | (R != 0 ? 1ull : 0ull), (uint32_t)(Q >> 55), e, ua & (1ull << 63));
}

SW2D_HD double sw2d_div_rn(double a, double b) {
    const uint64_t ua = sw2d_f64_bits(a), ub = sw2d_f64_bits(b);
    const uint32_t ea = (uint32_t)(ua >> 52) & 0x7ffu, eb = (uint32_t)(ub >> 52) & 0x7ffu;
    const uint64_t sign = (ua ^ ub) & (1ull << 63);
    const uint32_t e = ea - eb + 1022u; /* biased exponent of a quotient below 1 (ma < mb) */
    if (ea - 1u >= 0x7feu || eb - 1u >= 0x7feu || e - 1u >= 0x7fdu) {
        if ((ua << 1) == 0 && eb - 1u < 0x7feu) return sw2d_f64_from_bits(sign); /* 0 / b */
        return a / b; /* subnormal, inf, NaN; a quotient that is or may be subnormal or overflow */
    }
    const uint64_t M = (1ull << 52) - 1ull, H = 1ull << 52;
    const uint64_t ma = (ua & M) | H, mb = (ub & M) | H;
    const float rf = sw2d_rcp_est((float)(int32_t)(mb >> 29)); /* 2^29 / mb */
    int64_t R = (int64_t)(ma - mb);
    const int32_t d1 = (int32_t)((float)(int32_t)(R >> 22) * (rf * 32768.0f));
    R = (int64_t)(((uint64_t)R << 22) - (uint64_t)(int64_t)d1 * mb);
    const int32_t d2 = (int32_t)((float)(int32_t)(R >> 26) * (rf * 524288.0f));
    R = (int64_t)(((uint64_t)R << 22) - (uint64_t)(int64_t)d2 * mb);
    const int32_t d3 = sw2d_i32_floor_f32(sw2d_fmaf((float)(int32_t)(R >> 29), rf * 2048.0f, -0.35f));
    R = (int64_t)(((uint64_t)R << 11) - (uint64_t)(int64_t)d3 * mb);
    uint64_t Q = (1ull << 55) + ((uint64_t)(int64_t)d1 << 33) + ((uint64_t)(int64_t)d2 << 11) + (uint64_t)(int64_t)d3;
    if (R >= (int64_t)mb) {
        R -= (int64_t)mb;
        Q += 1ull;
    }
    return sw2d_round_pack(Q | (R != 0 ? 1ull : 0ull), (uint32_t)(Q >> 55), e, sign);
}

/* ------------------------------------------------------------------------
 * sqrt(x) correctly rounded with integer and binary32 operations only (the
 * companion of sw2d_div_rn), for x positive and normal (a zero returns
 * itself, every other x the hardware sqrt).  With x = m 2^E, E even, m in [2^52, 2^54),
 * S = floor(sqrt(m 2^54)) (54 bits) is built from its leading 24 bits, a
 * binary32 square root, and two signed digits of 15 bits, each the exact
 * remainder over twice the root so far, estimated with a binary32
 * reciprocal; the next digit takes up what an estimate is off by, the last
 * one is biased by 0.2 and rounded down, so one comparison with the exact
 * remainder completes it.  A 54-bit S decides the rounding by itself: its
 * last bit is the half bit, and m 2^54 is never an odd square.
 * Issue 72 cycles a warp on a GB300 against 185 for a form that corrected a
 * 46-bit estimate on its 128-bit remainder by single steps.
 * Bit-identical to the IEEE square root (the CPU tests compare it with the
 * host's sqrt). */
SW2D_HD float sw2d_sqrt_est(float x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
#if defined(SW2D_TEST_EST_SCALE)
    return sqrtf(x) * (float)(SW2D_TEST_EST_SCALE);
#else
    return sqrtf(x);
#endif
#endif
}

SW2D_HD double sw2d_sqrt_rn(double x) {
    const uint64_t ux = sw2d_f64_bits(x);
    const uint32_t ex = (uint32_t)(ux >> 52);
    if (ex - 1u >= 0x7feu) {
        if ((ux << 1) == 0) return x;
        return sqrt(x); /* negative, subnormal, inf, NaN */
    }
    const uint64_t H = 1ull << 52;
    const uint32_t odd = (ex + 1u) & 1u; /* E = ex - 1075 odd */
    const uint64_t m = ((ux & (H - 1ull)) | H) << odd;
    /* f = m / 2^52 in [1, 4) truncated to 23 bits, its root in [1, 2) */
    const float f = (float)(int32_t)(m >> 30) * 2.384185791015625e-07f;
    const float sh = sw2d_sqrt_est(f);
    const float rs = sw2d_rcp_est(sh) * 5.9604644775390625e-08f; /* 1 / (2 s0), s0 = sh 2^23 */
    const int32_t s0 = (int32_t)(sh * 8388608.0f);
    int64_t R = (int64_t)(m - ((uint64_t)s0 * (uint64_t)s0 << 6)); /* m - (s0 2^3)^2 */
    /* S1 = s0 2^15 + c1, remainder m 2^24 - S1^2 */
    const int32_t c1 = (int32_t)((float)(int32_t)(R >> 6) * (rs * 32768.0f));
    const uint64_t S1 = ((uint64_t)s0 << 15) + (uint64_t)(int64_t)c1;
    R = (int64_t)(((uint64_t)R << 24) - (uint64_t)(int64_t)c1 * (((uint64_t)s0 << 16) + (uint64_t)(int64_t)c1));
    /* S = S1 2^15 + c2, remainder m 2^54 - S^2 */
    const int32_t c2 = sw2d_i32_floor_f32(sw2d_fmaf((float)(int32_t)(R >> 15), rs * 32768.0f, -0.2f));
    uint64_t S = (S1 << 15) + (uint64_t)(int64_t)c2;
    R = (int64_t)(((uint64_t)R << 30) - (uint64_t)(int64_t)c2 * ((S1 << 16) + (uint64_t)(int64_t)c2));
    if (R > (int64_t)(2 * S)) S++;
    return sw2d_f64_from_bits(((uint64_t)((ex - odd + 1021u) >> 1) << 52) + ((S + 1ull) >> 1));
}

#endif /* SW2D_MATH_H */
