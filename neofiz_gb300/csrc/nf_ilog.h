/*
 * nf_ilog.h -- nf_log and nf_pow (nf_math.h) with the logarithm in integer arithmetic, the same
 * bits.
 *
 * nf_log_dd spends about thirty FP64 instructions, 64 to 76 cycles each on GB300; here the same
 * formula is summed in 96-bit fixed point (units of 2^-84) by the integer units:
 *
 *   log x = k ln2 + (-log invc) + r - rh^2/2 - rl rh + rh^3 (1/3 - rh/4 + rh^2/5 - rh^3/6 + rh^4/7)
 *
 * with r = z invc - 1 = rh + rl exact, rh the part nf_log_dd's rounded product gives. nf_log_dd
 * rounds inside: its cubic term (|rh^3 / 3| < 2^-25.5) five times and the sum of its small
 * terms, together less than 2^-76 for |k| <= 64; the fixed-point terms are truncated by less
 * than 2^-77. So the two sums lie within NF_LOG_SLACK = 2^-75 of each other, and where no
 * rounding boundary lies that close to the fixed-point sum, both round to the same double
 * (Ziv's test: A. Ziv, "Fast evaluation of elementary mathematical functions with correctly
 * rounded last bit", ACM TOMS 17, 1991). Where one does, and outside 2^-64 <= x < 2^64 or for
 * |log x| < 2^-8, nf_math.h's own sequence runs: the results are its results always.
 *
 * nf_pow's exponential follows nf_exp_dd instruction by instruction; the low part of the
 * logarithm, known to the slack, enters it once, in the rounded sum a + plo, and the same test
 * there shows that the slack cannot change the sum.
 */
#ifndef NF_ILOG_H
#define NF_ILOG_H

#include "nf_math.h"
#include "nf_ifp.h"

#define NF_LOG_SLACK_EXP (-75)

#if defined(__CUDACC__)
#define NF_ILOG_SLOW static __host__ __device__ __noinline__
static __device__ const uint32_t nf_log_words_d[8 * 128] = { NF_LOG_WORDS };
#else
#define NF_ILOG_SLOW static
#endif
static const uint32_t nf_log_words_h[8 * 128] = { NF_LOG_WORDS };

/* Counts the slow paths in host tests. */
#if !defined(__CUDA_ARCH__)
static long nf_ilog_slow_count = 0;
#define NF_ILOG_COUNT() (nf_ilog_slow_count++)
#else
#define NF_ILOG_COUNT() ((void)0)
#endif

NF_ILOG_SLOW double nf_log_slow(double x) { NF_ILOG_COUNT(); return nf_log(x); }
NF_ILOG_SLOW double nf_pow_slow(double x, double y) { NF_ILOG_COUNT(); return nf_pow(x, y); }

/* The high 64 bits of a b, at most two units too small. */
NF_IFP uint64_t nf_ilog_mulhi64(uint64_t a, uint64_t b) {
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a;
    const uint32_t bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
    return (uint64_t)ah * bh + nf_ifp_mulhi(ah, bl) + nf_ifp_mulhi(al, bh);
}
/* Leading zeros of a nonzero word. */
NF_IFP int nf_ilog_clz(uint32_t x) {
#if defined(__CUDA_ARCH__)
    return __clz((int)x);
#else
    return __builtin_clz(x);
#endif
}
/* (hi:lo) << s, upper word, 0 <= s < 32. */
NF_IFP uint32_t nf_ilog_up(uint32_t hi, uint32_t lo, int s) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_l(lo, hi, s);
#else
    return s ? (hi << s) | (lo >> (32 - s)) : hi;
#endif
}

/* The fixed-point logarithm, normalised: |log x| = (w2:w1:w0) 2^(-84 - n) with w2's top bit set,
 * neg its sign mask; returns 0 where the method does not apply. */
typedef struct { uint32_t w2, w1, w0, neg; int n; } nf_ilog;

NF_IFP int nf_ilog_of(double x, nf_ilog *o) {
    const uint32_t h = nf_ifp_hi(x), l = nf_ifp_lo(x);
    /* x = 2^k z, table entry j: as nf_log_dd (NF_LOG_OFF's low word is zero) */
    const uint32_t th = h - (uint32_t)(NF_LOG_OFF >> 32);
    const int32_t k = (int32_t)th >> 20;
    const uint32_t j = (th >> 13) & 127u;
    const uint32_t hz = (uint32_t)(NF_LOG_OFF >> 32) + (th & 0xfffffu);
#if defined(__CUDA_ARCH__)
    const uint4 wa = __ldg(reinterpret_cast<const uint4 *>(nf_log_words_d) + 2 * j);
    const uint32_t il = wa.x, ih = wa.y, c0 = wa.z, c1 = wa.w;
    const uint32_t c2 = __ldg(nf_log_words_d + 8 * j + 4);
#else
    const uint32_t *w = nf_log_words_h + 8 * j;
    const uint32_t il = w[0], ih = w[1], c0 = w[2], c1 = w[3], c2 = w[4];
#endif
    /* P = (z 2^53) (invc 2^53), r = P 2^-106 - 1 in words p0, p1, t (signed) */
    const uint32_t f = (hz >> 20) & 1u;                /* z's exponent field is 1022 or 1023 */
    const uint32_t mh = (hz & 0xfffffu) | 0x100000u;
    const uint32_t zh = nf_ilog_up(mh, l, (int)f), zl = l << f;
    const uint64_t a0 = (uint64_t)zl * il;
    const uint64_t a1 = (uint64_t)zl * ih + ((uint64_t)zh * il + (a0 >> 32));
    const int64_t t = (int64_t)((uint64_t)zh * ih + (a1 >> 32)) - ((int64_t)1 << 42);
    const uint32_t p0 = (uint32_t)a0, p1 = (uint32_t)a1;
    const uint32_t tl = (uint32_t)t, tu = (uint32_t)((uint64_t)t >> 32);
    /* rh: r rounded as the product z invc rounds, to 2^-52 from 1 up and 2^-53 below */
    const int64_t d = (int64_t)(((uint64_t)t << 11) | (p1 >> 21));    /* r 2^53, floor */
    const uint32_t rest = nf_ifp_shl(p1, p0, 11);                     /* the next 32 bits */
    const int up = t >= 0;
    const uint32_t frac = up ? ((uint32_t)d << 31) | (rest >> 1) : rest;
    /* a halfway case is left to the slow path (frac alone decides: a few more go there) */
    if (frac == 0x80000000u) return 0;
    const int64_t rh = up ? (d & ~(int64_t)1) + 2 * (int64_t)(frac >> 31) : d + (int64_t)(frac >> 31);
    const int32_t rl = up ? (int32_t)frac : (int32_t)frac >> 1;       /* rl 2^84 */
    /* rh^2 exactly: A = (rh 2^53)^2, below 2^92 */
    const uint64_t a = (uint64_t)(rh < 0 ? -rh : rh);
    const uint32_t b0 = (uint32_t)a, b1 = (uint32_t)(a >> 32);
    const uint64_t s0 = (uint64_t)b0 * b0;
    const uint64_t s1 = (uint64_t)b0 * (2u * b1) + (s0 >> 32);
    const uint32_t s2 = b1 * b1 + (uint32_t)(s1 >> 32);
    const uint32_t A0 = (uint32_t)s0, A1 = (uint32_t)s1, A2 = s2;
    /* S = rh^2 2^78, and the cubic's factor T = 1/3 - rh/4 + rh^2/5 - rh^3/6 + rh^4/7 in 2^-64 */
    const uint32_t Sh = nf_ifp_shr(A2, A1, 28), Sl = nf_ifp_shr(A1, A0, 28);
    const uint64_t S = ((uint64_t)Sh << 32) | Sl;
    const uint32_t q47 = nf_ifp_shl(Sh, Sl, 1);                       /* rh^2 2^47, below 2^31 */
    const int32_t r39 = (int32_t)(rh >> 14);                          /* rh 2^39 */
    const uint64_t fifth = (uint64_t)Sh * 0x33333333u + nf_ifp_mulhi(Sl, 0x33333333u)
                           + (nf_ifp_mulhi(Sh, 0x33333333u));         /* rh^2 / 5 2^78 */
    const int32_t cube = nf_ifp_mulhi_s(nf_ifp_mulhi_s((int32_t)q47, r39), 715827883);  /* / 6, 2^54 */
    const uint32_t four = nf_ifp_mulhi(nf_ifp_mulhi(q47, q47), 2454267026u);  /* rh^4 / 7 2^64 */
    const uint64_t T = 0x5555555555555555ULL - ((uint64_t)rh << 9) + (fifth >> 14)
                       - ((uint64_t)(int64_t)cube << 10) + four;
    const uint64_t r3 = nf_ilog_mulhi64(S, a << 18);                  /* |rh|^3 2^85 */
    const uint64_t C = nf_ilog_mulhi64(r3, T) >> 1;                   /* |cubic| 2^84 */
    const int32_t cross = nf_ifp_mulhi_s(rl, r39) >> 7;               /* rl rh 2^84 */
    /* the sum, modulo 2^96 */
    const uint32_t kb = (uint32_t)(k + NF_LOG_BIAS);
    const uint64_t e0 = (uint64_t)kb * NF_LN2_FIX0 + c0;
    const uint64_t e1 = (uint64_t)kb * NF_LN2_FIX1 + c1 + (e0 >> 32);
    uint32_t L2 = kb * NF_LN2_FIX2 + c2 + (uint32_t)(e1 >> 32);
    uint64_t lo = ((uint64_t)(uint32_t)e1 << 32) | (uint32_t)e0;
    /* + r 2^84 */
    const uint64_t rlow = ((uint64_t)nf_ifp_shr(tl, p1, 22) << 32) | nf_ifp_shr(p1, p0, 22);
    lo += rlow;
    L2 += nf_ifp_shr(tu, tl, 22) + (lo < rlow);
    /* - rh^2 / 2 2^84 */
    const uint64_t half = ((uint64_t)nf_ifp_shr(A2, A1, 23) << 32) | nf_ifp_shr(A1, A0, 23);
    L2 -= (A2 >> 23) + (lo < half);
    lo -= half;
    /* +- C - rl rh: below 2^60 together */
    const int64_t tail = (rh < 0 ? -(int64_t)C : (int64_t)C) - cross;
    const uint64_t sum = lo + (uint64_t)tail;
    L2 += (uint32_t)((int32_t)(tail >> 63)) + (sum < lo);
    lo = sum;
    /* magnitude (a unit of 2^-84 aside) and normalisation */
    const uint32_t neg = (uint32_t)((int32_t)L2 >> 31);
    const uint32_t m2 = L2 ^ neg, m1 = (uint32_t)(lo >> 32) ^ neg, m0 = (uint32_t)lo ^ neg;
    const int n = nf_ilog_clz(m2 | 1u);
    o->w2 = nf_ilog_up(m2, m1, n);
    o->w1 = nf_ilog_up(m1, m0, n);
    o->w0 = m0 << n;
    o->neg = neg & 0x80000000u;
    o->n = n;
    /* 2^-64 <= x < 2^64 (so |k| <= 64), |log x| >= 2^-8 */
    return (h - 0x3bf00000u < 0x08000000u) & (m2 >= 0x1000u);
}

/* The rounded logarithm from the normalised sum; the bits below the last place as a 32-bit
 * fraction of it in *below. */
NF_IFP double nf_ilog_round(nf_ilog v, uint32_t *below) {
    *below = nf_ifp_shl(v.w1, v.w0, 21);
    const uint64_t m = ((((uint64_t)v.w2 << 32) | v.w1) >> 11) + (*below >> 31)
                       + ((uint64_t)((uint32_t)(1033 - v.n) << 20 | v.neg) << 32);
    return nf_ifp_make((uint32_t)(m >> 32), (uint32_t)m);
}
/* The slack in units of below is 2^(84 - 75 + n - 11), n <= 19: whether half lies within it. */
NF_IFP int nf_ilog_near_half(uint32_t below, int n) {
    return below - 0x80000000u + (1u << n) < (2u << n);
}

/* nf_log(x) where *sure, without a branch. */
NF_IFP double nf_log_try(double x, int *sure) {
    nf_ilog v;
    uint32_t below;
    const int ok = nf_ilog_of(x, &v);
    const double r = nf_ilog_round(v, &below);
    *sure = ok & !nf_ilog_near_half(below, v.n);
    return r;
}
NF_IFP double nf_log_fast(double x) {
    int sure;
    const double r = nf_log_try(x, &sure);
    return sure ? r : nf_log_slow(x);
}

/* nf_pow(x, y) where *sure, without a branch. */
NF_IFP double nf_pow_try(double x, double y, int *sure) {
    nf_ilog v;
    uint32_t below;
    const uint32_t yh = nf_ifp_hi(y);
    /* 2^-9 <= y < 2 */
    const int ok = nf_ilog_of(x, &v) & (yh - 0x3f600000u < 0x00a00000u);
    const double lh = nf_ilog_round(v, &below);
    /* lo = log x - lh: 43 bits and a sign */
    const uint64_t rest = ((uint64_t)(v.w1 & 0x7ffu) << 32) | v.w0;
    const int roundedUp = (int)(below >> 31);
    uint64_t g = roundedUp ? ((uint64_t)0x800 << 32) - rest : rest;
    g |= 1u;
    const uint32_t gh = (uint32_t)(g >> 32);
    const int sh = gh ? nf_ilog_clz(gh) : 32 + nf_ilog_clz((uint32_t)g);     /* >= 20 */
    g <<= sh;                                                                /* top bit set */
    /* value g 2^(-84 - n - sh): field 1023 + 63 - 84 - n - sh, the leading bit adds one to it */
    const uint64_t gb = (g >> 11) + ((uint64_t)((uint32_t)(1001 - v.n - sh) << 20) << 32);
    const double ll = nf_ifp_make((uint32_t)(gb >> 32) | (v.neg ^ (roundedUp ? 0x80000000u : 0u)),
                                  (uint32_t)gb);
    const double p = y * lh;
    const double plo = fma(y, ll, fma(y, lh, -p));
    /* nf_exp_dd(p, plo) */
    const double kd = rint(p * NF_EXP_N_OVER_LN2);
    const int n = (int)kd;
    const double al = fma(-kd, NF_EXP_L_LO, fma(-kd, NF_EXP_L_HI, p));
    const double r = al + plo;
    /* the sum's error and how far it stays from half an ulp of r (all exact), against y times
     * the slack (the high words of two doubles order as they do) */
    const double e = plo - (r - al);
    const uint32_t rx = nf_ifp_hi(r) & 0x7ff00000u;
    const double gap = nf_ifp_make(rx - (53u << 20), 0u) - fabs(e);
    *sure = ok & ((int32_t)nf_ifp_hi(gap) > (int32_t)(yh - ((uint32_t)(-NF_LOG_SLACK_EXP) << 20)))
            & (rx > (60u << 20)) & !nf_ilog_near_half(below, v.n);
    const int j = n & 127, m = (n - j) / 128;
    const double thi = nf_exp_tab(2 * j), tlo = nf_exp_tab(2 * j + 1);
    double t = fma(r, 0x1.1111111111111p-7, 0x1.5555555555555p-5);
    t = fma(r, t, 0x1.5555555555555p-3);
    t = fma(r, t, 0.5);
    const double q = fma(r * r, t, r);
    const double er = thi + fma(thi, q, tlo);          /* in [0.99, 2): |p| < 90 scales by bits */
    return nf_ifp_make(nf_ifp_hi(er) + ((uint32_t)m << 20), nf_ifp_lo(er));
}
NF_IFP double nf_pow_fast(double x, double y) {
    int sure;
    const double r = nf_pow_try(x, y, &sure);
    return sure ? r : nf_pow_slow(x, y);
}

#endif /* NF_ILOG_H */
