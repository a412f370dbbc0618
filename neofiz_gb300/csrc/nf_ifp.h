/*
 * nf_ifp.h -- IEEE double division and square root in 32-bit integer arithmetic.
 *
 * GB300 issues one FP64 warp instruction per 64 cycles on each quarter of an SM, and a division
 * or a square root is a sequence of about nine of them. The integer units issue a 32-bit
 * multiply every two cycles, so the same correctly rounded quotient costs less as some sixty
 * integer instructions, and it leaves the FP64 pipe to the additions and multiplications.
 *
 * Method: schoolbook long division and square root (Knuth, TAOCP vol. 2, 4.3.1, Algorithm D) on
 * the 53-bit significands, in digits of 26 to 30 bits. Each digit is the running remainder's
 * head times a 31-bit reciprocal (or reciprocal root) kept slightly too small, so every digit
 * is too small by a few units and every remainder stays positive and exact modulo 2^64. The
 * reciprocal starts from the FP32 approximation, whose documented error is at most 2^-23
 * (2^-22.9 for the root), and one Newton step in integers. Three digits give about 84 bits of
 * the quotient (root), at most 16 units too small in the last place kept; no quotient or root
 * of two 53-bit significands lies exactly halfway between two doubles, so those bits round
 * correctly unless they end within 32 units below a halfway point, where the machine operation
 * decides (one value in 2^27). Zeros, subnormals, infinities, NaN and exponents outside
 * 2^+-511 take the machine operation too.
 *
 * Bit-identical to the machine operations by construction; tests/test_ifp.py compares them on
 * the host (this header compiles there, with the approximations' error range played through)
 * and on the device.
 */
#ifndef NF_IFP_H
#define NF_IFP_H

#include <stdint.h>
#include <string.h>
#include <math.h>

#if defined(__CUDACC__)
#define NF_IFP static __host__ __device__ __forceinline__
#else
#define NF_IFP static inline
#endif

/* The host has no approximate reciprocal: it rounds the true value to float and, for tests,
 * moves it by nf_ifp_off units in the last place. */
#if !defined(__CUDA_ARCH__)
static int nf_ifp_off = 0;
#endif

NF_IFP uint32_t nf_ifp_hi(double x) {
#if defined(__CUDA_ARCH__)
    return (uint32_t)__double2hiint(x);
#else
    uint64_t u; memcpy(&u, &x, 8); return (uint32_t)(u >> 32);
#endif
}
NF_IFP uint32_t nf_ifp_lo(double x) {
#if defined(__CUDA_ARCH__)
    return (uint32_t)__double2loint(x);
#else
    uint64_t u; memcpy(&u, &x, 8); return (uint32_t)u;
#endif
}
NF_IFP double nf_ifp_make(uint32_t hi, uint32_t lo) {
#if defined(__CUDA_ARCH__)
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t u = ((uint64_t)hi << 32) | lo; double x; memcpy(&x, &u, 8); return x;
#endif
}
NF_IFP uint32_t nf_ifp_mulhi(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
NF_IFP int32_t nf_ifp_mulhi_s(int32_t a, int32_t b) {
#if defined(__CUDA_ARCH__)
    return __mulhi(a, b);
#else
    return (int32_t)(((int64_t)a * b) >> 32);
#endif
}
/* The low word of (hi:lo) << s and of (hi:lo) >> s, 0 < s < 32. */
NF_IFP uint32_t nf_ifp_shl(uint32_t hi, uint32_t lo, int s) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_l(lo, hi, s);
#else
    return (hi << s) | (lo >> (32 - s));
#endif
}
NF_IFP uint32_t nf_ifp_shr(uint32_t hi, uint32_t lo, int s) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(lo, hi, s);
#else
    return (hi << (32 - s)) | (lo >> s);
#endif
}
/* The bits of 1 / f for f in [1, 2) and of 1 / sqrt(f) for f in [1, 4), f given by its bits. */
NF_IFP uint32_t nf_ifp_rcp(uint32_t f) {
#if defined(__CUDA_ARCH__)
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(f)));
    return __float_as_uint(y);
#else
    float x, y; uint32_t r; memcpy(&x, &f, 4); y = 1.0f / x; memcpy(&r, &y, 4);
    return r + (uint32_t)nf_ifp_off;
#endif
}
NF_IFP uint32_t nf_ifp_rsqrt(uint32_t f) {
#if defined(__CUDA_ARCH__)
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(f)));
    return __float_as_uint(y);
#else
    float x, y; uint32_t r; memcpy(&x, &f, 4); y = (float)(1.0 / sqrt((double)x)); memcpy(&r, &y, 4);
    return r + (uint32_t)nf_ifp_off;
#endif
}

/* The exponent's two leading bits differ: 2^-511 <= |x| < 2^513, by the high word. */
NF_IFP int nf_ifp_moderate(uint32_t h) { return (int)((h ^ (h << 1)) >> 30) & 1; }

/* A divisor: its significand and the 31-bit reciprocal R < 2^31 / beta <= R + 5, beta its
 * significand in [1, 2). Several quotients by one divisor share it. */
typedef struct { uint32_t mh, ml, r, h; } nf_divisor;

NF_IFP nf_divisor nf_divisor_of(double b) {
    nf_divisor o;
    o.h = nf_ifp_hi(b);
    o.ml = nf_ifp_lo(b);
    o.mh = (o.h & 0xfffffu) | 0x100000u;
    /* 1 / beta to 2^-22 from beta's head, as y 2^30 */
    const uint32_t y = nf_ifp_rcp((nf_ifp_shl(o.mh, o.ml, 3) & 0x7fffffu) | 0x3f800000u);
    const uint32_t y30 = (y - 0x3f000000u + 0x800000u) << 6;
    /* Newton: 1 - beta y in units of 2^-52 (its 2^61 vanishes modulo 2^32), then y (2 - beta y) */
    const uint64_t t = (uint64_t)nf_ifp_shl(o.mh, o.ml, 11) * y30;
    const int32_t e = (int32_t)nf_ifp_shr((uint32_t)(t >> 32), (uint32_t)t, 9);
    o.r = 2u * y30 - 3u - (uint32_t)(nf_ifp_mulhi_s((int32_t)y30, e) >> 19);
    return o;
}

/* a / b for moderate a and b; *unsure is set where the bits do not settle the rounding or the
 * quotient is not normal. */
NF_IFP double nf_div_digits(double a, nf_divisor b, int *unsure) {
    const uint32_t ha = nf_ifp_hi(a), la = nf_ifp_lo(a);
    const uint32_t mah = (ha & 0xfffffu) | 0x100000u;
    const uint64_t mb = ((uint64_t)b.mh << 32) | b.ml, ma = ((uint64_t)mah << 32) | la;
    /* the ratio of the significands in [1, 2): double the dividend if it is the smaller */
    const uint32_t less = ma < mb;
    const uint64_t m = ma << less;
    /* first digit: ratio 2^29, at most 7 too small; remainder m 2^29 - q1 mb < 7 mb */
    const uint32_t q1 = nf_ifp_mulhi((uint32_t)(m >> 22), b.r);
    const uint64_t r1 = (m << 29) - (uint64_t)q1 * b.ml - ((uint64_t)(q1 * b.mh) << 32);
    /* second digit, 27 bits further */
    const uint32_t q2 = nf_ifp_mulhi((uint32_t)(r1 >> 24), b.r);
    const uint64_t r2 = (r1 << 27) - (uint64_t)q2 * b.ml - ((uint64_t)(q2 * b.mh) << 32);
    /* third digit, 27 more; its remainder is not needed */
    const uint32_t q3 = nf_ifp_mulhi((uint32_t)(r2 >> 24), b.r);
    const uint64_t q = (uint64_t)q1 * 0x8000000u + q2 + (q3 >> 27);       /* ratio 2^56 */
    const uint32_t frac = ((uint32_t)q << 28) | ((q3 << 5) >> 4);
    /* exponent field (ea - eb + 1023 - less) - 1, the significand's leading bit adds the one;
     * a field below 1 wraps */
    const uint32_t e = ((ha & 0x7ff00000u) - (b.h & 0x7ff00000u) + 0x3fe00000u) - (less << 20);
    *unsure = (frac - 0x7fffffc0u < 0x40u) | (e >= 0x7fd00000u);
    const uint64_t r = (q >> 4) + (frac >> 31) + ((uint64_t)(e | ((ha ^ b.h) & 0x80000000u)) << 32);
    return nf_ifp_make((uint32_t)(r >> 32), (uint32_t)r);
}

/* a / b where *sure, without a branch (a may be a zero). */
NF_IFP double nf_div_try(double a, nf_divisor b, int *sure) {
    int unsure;
    const double q = nf_div_digits(a, b, &unsure);
    const uint32_t ha = nf_ifp_hi(a);
    const int zero = ((ha << 1) | nf_ifp_lo(a)) == 0u;
    *sure = nf_ifp_moderate(b.h) & ((nf_ifp_moderate(ha) & (unsure ^ 1)) | zero);
    return zero ? nf_ifp_make((ha ^ b.h) & 0x80000000u, 0u) : q;
}

/* a / b, rounded as the machine division rounds. */
NF_IFP double nf_div_by(double a, double b, nf_divisor v) {
    int unsure;
    const double q = nf_div_digits(a, v, &unsure);
    const uint32_t ha = nf_ifp_hi(a);
    if (nf_ifp_moderate(ha) & nf_ifp_moderate(v.h) & (unsure ^ 1)) return q;
    if (((ha << 1) | nf_ifp_lo(a)) == 0u && nf_ifp_moderate(v.h))      /* +-0 / b */
        return nf_ifp_make((ha ^ v.h) & 0x80000000u, 0u);
    return a / b;
}
NF_IFP double nf_div(double a, double b) { return nf_div_by(a, b, nf_divisor_of(b)); }

/* sqrt(a), rounded as the machine square root rounds. */
NF_IFP double nf_sqrt(double a) {
    const uint32_t h = nf_ifp_hi(a), l = nf_ifp_lo(a);
    /* a = x 2^(2 k) with x in [1, 4): the unbiased exponent is odd when the field is even */
    const uint32_t odd = ~(h >> 20) & 1u;
    const uint32_t mh = (h & 0xfffffu) | 0x100000u;
    const uint64_t m = (((uint64_t)mh << 32) | l) << odd;                 /* x 2^52 */
    const uint32_t y = nf_ifp_rsqrt(((nf_ifp_shl(mh, l, 3) & 0x7fffffu) | 0x3f800000u) + (odd << 23));
    const uint32_t y30 = (y - 0x3f000000u + 0x800000u) << 6;           /* 2^30 / sqrt(x) */
    /* g = x y 2^30 and e = 1 - g y in units of 2^-51 (its 2^60 vanishes modulo 2^32) */
    const uint32_t g = (uint32_t)(((uint64_t)(uint32_t)(m >> 22) * y30) >> 30);
    const uint64_t t = (uint64_t)g * y30;
    const int32_t e = (int32_t)nf_ifp_shr((uint32_t)(t >> 32), (uint32_t)t, 9);
    /* Newton: the root's head 2^30 sqrt(x), at most 5 too small, and 2^31 / sqrt(x), likewise */
    const uint32_t s1 = g - 3u - (uint32_t)(nf_ifp_mulhi_s((int32_t)(g >> 1), e) >> 19);
    const uint32_t r = 2u * y30 - 4u - (uint32_t)(nf_ifp_mulhi_s((int32_t)y30, e) >> 19);
    /* remainder x 2^60 - s1^2 < 2^35; the next digit is remainder / (2 root), 28 bits further */
    const uint64_t r1 = (m << 8) - (uint64_t)s1 * s1;
    const uint32_t q2 = nf_ifp_mulhi((uint32_t)(r1 >> 3), r);
    const uint64_t s2 = (uint64_t)s1 * 0x8000000u + q2;                   /* sqrt(x) 2^57 */
    const uint32_t sl = (uint32_t)s2, sh = (uint32_t)(s2 >> 32);
    const uint64_t sq = (uint64_t)sl * sl + ((uint64_t)(sl * (2u * sh)) << 32);
    const uint64_t r2 = (m << 62) - sq;                                   /* x 2^114 - s2^2 */
    const uint32_t q3 = nf_ifp_mulhi((uint32_t)(r2 >> 30), r);            /* 27 bits further */
    const uint64_t q = s2 + (q3 >> 27);
    const uint32_t frac = ((uint32_t)q << 27) | (q3 & 0x7ffffffu);
    /* exponent field (ea + 1023) / 2 rounded down for x in [1, 4), less one */
    const uint32_t eh = (((h >> 20) + 1023u) >> 1) - 1u;
    const uint64_t out = (q >> 5) + (frac >> 31) + ((uint64_t)eh << 52);
    if (h - 0x00100000u < 0x7fe00000u && frac - 0x7fffffc0u >= 0x40u)
        return nf_ifp_make((uint32_t)(out >> 32), (uint32_t)out);
    if (((h << 1) | l) == 0u) return a;                                   /* +-0 */
    return sqrt(a);
}

/* Products and scalings in integer arithmetic for straight-line code: each returns the machine's
 * bits or sets *bad, which the caller tests once at the end to take the machine path instead.
 * A product costs about as much on the integer units as on the FP64 pipe; code that spreads its
 * products over both runs them side by side. */

/* x is +-0. */
NF_IFP int nf_ifp_zero(uint32_t h, uint32_t l) { return ((h << 1) | l) == 0u; }

/* a b: both moderate, or one a zero and the other moderate or a zero. */
NF_IFP double nf_mul_try(double a, double b, uint32_t *bad) {
    const uint32_t ha = nf_ifp_hi(a), la = nf_ifp_lo(a), hb = nf_ifp_hi(b), lb = nf_ifp_lo(b);
    const uint32_t ma = (ha & 0xfffffu) | 0x100000u, mb = (hb & 0xfffffu) | 0x100000u;
    const int za = nf_ifp_zero(ha, la), zb = nf_ifp_zero(hb, lb);
    /* the 106-bit product of the significands, in [2^104, 2^106); its top 64 bits in t (above
     * 2^106 2^-64 a leading zero at most), the rest only as zero or not */
    const uint64_t p = (uint64_t)la * lb;
    const uint64_t q = (uint64_t)la * mb + ((uint64_t)ma * lb + (p >> 32));
    const uint64_t r = (uint64_t)ma * mb + (q >> 32);
    const uint32_t th = nf_ifp_shr((uint32_t)(r >> 32), (uint32_t)r, 10);
    const uint32_t rest = ((uint32_t)q & 0x3ffu) | (uint32_t)p;
    const uint32_t tl = nf_ifp_shr((uint32_t)r, (uint32_t)q, 10) | (rest < 1u ? rest : 1u);
    const uint32_t n = th >> 31;                       /* 0: normalise by one place */
    const uint64_t t = (((uint64_t)th << 32) | tl) << (n ^ 1u);
    const uint32_t e = (ha & 0x7ff00000u) + (hb & 0x7ff00000u) - 0x3ff00000u + (n << 20);
    const uint32_t sign = (ha ^ hb) & 0x80000000u;
    *bad |= ((uint32_t)((nf_ifp_moderate(ha) | za) & (nf_ifp_moderate(hb) | zb)) ^ 1u)
            | ((e >= 0x7fe00000u) & (uint32_t)((za | zb) ^ 1));
    /* round to nearest even at bit 11 */
    const uint32_t up = (((uint32_t)t & 0x7ffu) + 0x3ffu + ((uint32_t)(t >> 11) & 1u)) >> 11;
    const uint64_t v = (t >> 11) + up + ((uint64_t)(e + sign - 0x100000u) << 32);
    const int zero = za | zb;
    return nf_ifp_make(zero ? sign : (uint32_t)(v >> 32), zero ? 0u : (uint32_t)v);
}

/* x 2^k, |k| <= 8: a zero or a number in 2^+-1000. */
NF_IFP double nf_scale_try(double x, int k, uint32_t *bad) {
    const uint32_t h = nf_ifp_hi(x), l = nf_ifp_lo(x);
    const int normal = (h & 0x7fffffffu) - 0x01700000u < 0x7d000000u;
    const int zero = nf_ifp_zero(h, l);
    *bad |= (uint32_t)(normal | zero) ^ 1u;
    return nf_ifp_make(zero ? h : h + ((uint32_t)k << 20), l);
}

/* x 2^k, |k| <= 8, by the machine's product outside nf_scale_try's range. */
NF_IFP double nf_scale2(double x, int k) {
    uint32_t bad = 0;
    double r = nf_scale_try(x, k, &bad);
    if (bad) {
        const double f = nf_ifp_make((uint32_t)(1023 + k) << 20, 0u);
#if defined(__CUDA_ARCH__)
        asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(x), "d"(f));
#else
        r = x * f;
#endif
    }
    return r;
}

/* a b. */
NF_IFP double nf_mul(double a, double b) {
    uint32_t bad = 0;
    double r = nf_mul_try(a, b, &bad);
    if (bad) {
#if defined(__CUDA_ARCH__)
        /* volatile: a branch around the instruction, which the compiler would otherwise issue
         * for every product and select from */
        asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
#else
        r = a * b;
#endif
    }
    return r;
}

/* a / b (nf_div_try) with the same convention. */
NF_IFP double nf_quot_try(double a, nf_divisor b, uint32_t *bad) {
    int sure;
    const double q = nf_div_try(a, b, &sure);
    *bad |= (uint32_t)sure ^ 1u;
    return q;
}

#endif /* NF_IFP_H */
