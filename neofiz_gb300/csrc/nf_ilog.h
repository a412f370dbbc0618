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
 * terms, together less than 240 units for |k| <= 64; the fixed-point terms are off by less than
 * 115 (the -rh^3/6 term 77, k ln2 32). So the two sums lie within 384 units of each other (223
 * is the most that 160 million random arguments showed, half of them within 2^+-8, by the program
 * of tests/test_log_table.py), and where no
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

/* (NF_EXP_L_HI + NF_EXP_L_LO) 2^96, exact */
#define NF_LN2_128_0 0x5793c767u
#define NF_LN2_128_1 0xefa39ef3u
#define NF_LN2_128_2 0x0162e42fu

/* A row of the logarithm's table; the device reads its first four words as one 16-byte load. */
struct alignas(16) nf_log_row { uint32_t w[8]; };

#if defined(__CUDACC__)
#define NF_ILOG_SLOW static __host__ __device__ __noinline__
static __device__ const nf_log_row nf_log_rows_d[128] = { NF_LOG_WORDS };
#else
#define NF_ILOG_SLOW static
#endif
static const nf_log_row nf_log_rows_h[128] = { NF_LOG_WORDS };

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
    const uint4 wa = __ldg(reinterpret_cast<const uint4 *>(nf_log_rows_d[j].w));
    const uint32_t il = wa.x, ih = wa.y, c0 = wa.z, c1 = wa.w;
    const uint32_t c2 = __ldg(nf_log_rows_d[j].w + 4);
#else
    const uint32_t *w = nf_log_rows_h[j].w;
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
/* Whether half lies within the slack (384 2^n units, below 2^(n - 2) of below's; n <= 19). */
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

/* The last sum of a power whose r the slack may move by a unit: er = RN(thi + w). inRange: only
 * r's rounding is open, |r| in [2^(-1 - z), 2^-z). */
typedef struct { double thi, w, er; int inRange, z; } nf_pow_tail;

/* nf_pow(x, y) where *sure, without a branch. The product p = y lh, its error, the reduced
 * argument a = p - n ln2/128 and the sum r = a + plo are nf_exp_dd's, each rounded as its FP64
 * operation rounds: products and differences are exact in fixed point (n ln2/128 is a multiple
 * of 2^-96), so every rounding is known but the last, which has the slack in it and is sure
 * where the sum's tail stays that far from half a unit. */
NF_IFP double nf_pow_try(double x, double y, int *sure, nf_pow_tail *tail) {
    nf_ilog v;
    uint32_t below;
    const uint32_t yh = nf_ifp_hi(y), yl = nf_ifp_lo(y);
    /* 2^-9 <= y < 2 */
    int ok = nf_ilog_of(x, &v) & (yh - 0x3f600000u < 0x00a00000u);
    below = nf_ifp_shl(v.w1, v.w0, 21);
    ok &= !nf_ilog_near_half(below, v.n);
    /* |lh| = lm 2^(-41 - n) (lm up to 2^53), |log x| - |lh| = g 2^(-84 - n) */
    const uint32_t up = below >> 31;
    const uint64_t lm = ((((uint64_t)v.w2 << 32) | v.w1) >> 11) + up;
    const int64_t g = (int64_t)(((uint64_t)(v.w1 & 0x7ffu) << 32) | v.w0) - ((int64_t)up << 43);
    /* P = y's significand times lm, in units 2^(ey - n - 93); p its 53-bit rounding */
    const int ey = (int)(yh >> 20) - 1023;
    const uint32_t myh = (yh & 0xfffffu) | 0x100000u;
    const uint32_t ll = (uint32_t)lm, lh = (uint32_t)(lm >> 32);
    const uint64_t b0 = (uint64_t)yl * ll;
    const uint64_t b1 = (uint64_t)yl * lh + ((uint64_t)myh * ll + (b0 >> 32));
    const uint64_t b2 = (uint64_t)myh * lh + (b1 >> 32);       /* P = b2 : lo b1 : lo b0 */
    const uint32_t P0 = (uint32_t)b0, P1 = (uint32_t)b1, P2 = (uint32_t)b2, P3 = (uint32_t)(b2 >> 32);
    const int top = (int)(P3 >> 9);                            /* P >= 2^105 */
    /* shifted so that 53 bits are dropped */
    const uint32_t s0 = P0 << (top ^ 1), s1 = nf_ilog_up(P1, P0, top ^ 1);
    const uint32_t s2 = nf_ilog_up(P2, P1, top ^ 1), s3 = nf_ilog_up(P3, P2, top ^ 1);
    const uint32_t half = (s1 >> 20) & 1u;
    const uint64_t pm = ((((uint64_t)s3 << 32) | s2) << 11 | (s1 >> 21)) + half;
    const int64_t pr = (int64_t)(((uint64_t)(s1 & 0x1fffffu) << 32) | s0) - ((int64_t)half << 53);
    ok &= ((s1 & 0x1fffffu) != 0x100000u);                     /* a halfway case, or near one */
    /* |p| in [2^k, 2^(k+1)): p = pm 2^(k - 52) */
    const int k = ey - v.n + 11 + top;
    /* n = rint(p 128 / ln2) from its integer and 20 fraction bits, at most 4 units off */
    const uint32_t v20 = nf_ifp_mulhi((uint32_t)(pm >> 21), 0xb8aa3b29u) >> ((3 - k) & 31);
    const uint32_t n = (v20 + 0x80000u) >> 20;
    ok &= (((v20 + 4u - 0x80000u) & 0xfffffu) >= 8u) & (k <= 3);
    /* a = RN(p - n ln2/128) in units of 2^-96: |p| is below 2^4 and the difference below 2^-8 */
    const int sp = 44 + k;
    const uint32_t q0 = (uint32_t)pm << (sp & 31), q1 = nf_ilog_up((uint32_t)(pm >> 32), (uint32_t)pm, sp & 31);
    const uint32_t q2 = nf_ilog_up(0u, (uint32_t)(pm >> 32), sp & 31);
    const int wide = sp >= 32;
    const uint32_t t0 = wide ? 0u : q0, t1 = wide ? q0 : q1, t2 = wide ? q1 : q2;
    const uint64_t m0 = (uint64_t)n * NF_LN2_128_0;
    const uint64_t m1 = (uint64_t)n * NF_LN2_128_1 + (m0 >> 32);
    const uint32_t m2 = n * NF_LN2_128_2 + (uint32_t)(m1 >> 32);
    const uint64_t tl = ((uint64_t)t1 << 32) | t0, ml = ((uint64_t)(uint32_t)m1 << 32) | (uint32_t)m0;
    const uint64_t dl = tl - ml;
    const uint32_t dh = t2 - m2 - (tl < ml);
    const uint32_t neg = (uint32_t)((int32_t)dh >> 31);
    /* |difference|, exactly */
    const uint64_t al = (dl ^ (((uint64_t)neg << 32) | neg)) + (neg & 1u);
    const uint32_t ah = (dh ^ neg) + (uint32_t)((neg & 1u) & (al == 0u));
    ok &= (ah >= 0x10u) & (sp >= 0);
    const int z = nf_ilog_clz(ah | 1u);
    const uint32_t u2 = nf_ilog_up(ah, (uint32_t)(al >> 32), z);
    const uint32_t u1 = nf_ilog_up((uint32_t)(al >> 32), (uint32_t)al, z), u0 = (uint32_t)al << z;
    /* rounded to 53 bits: a = am 2^43 in units 2^(-96 - z); a halfway case is not settled */
    const uint32_t au = (u1 >> 10) & 1u;
    const uint64_t am = ((((uint64_t)u2 << 32) | u1) >> 11) + au;
    ok &= !(((u1 & 0x7ffu) == 0x400u) & (u0 == 0u));
    /* plo = perr + y ll in units 2^(ey - n - 93), then in a's */
    const uint64_t gm = nf_ilog_mulhi64((((uint64_t)myh << 32) | yl) << 11,
                                        (uint64_t)(g < 0 ? -g : g) << 19) >> 9;
    const int64_t pl = (pr >> (top ^ 1)) + (g < 0 ? -(int64_t)gm : (int64_t)gm);
    const int sh = ey - v.n + 3 + z;
    const int64_t ps = neg ? -pl : pl;
    ok &= (sh <= 40) & (sh >= -20);
    /* r = RN(a + plo): a ends above the lower 43 bits; 32 bits of the fraction below */
    const uint64_t low = sh >= 0 ? (uint64_t)ps << (sh & 63) : (uint64_t)(ps >> (-sh & 63));
    const uint32_t f32 = (uint32_t)(low >> 11);
    const uint64_t rm = am + (uint64_t)(ps >> ((43 - sh) & 63)) + (f32 >> 31);
    /* the slack of y ll in units of that fraction: 384 2^n y / 2^43 2^(sh - 11) */
    const int ts = ey + z - 10;
    const uint32_t w3 = (3u * myh) >> 2;
    const uint32_t ws = (ts >= 0 ? w3 << (ts & 31) : w3 >> (-ts & 31)) + 4u;
    ok &= (uint32_t)(rm >> 52) == 1u;
    *sure = ok & (ts <= 9) & (f32 - 0x80000000u + ws >= 2u * ws);
    const uint64_t rb = rm + ((uint64_t)((uint32_t)(1021 - z) << 20 | ((neg << 31) ^ v.neg)) << 32);
    const double r = nf_ifp_make((uint32_t)(rb >> 32), (uint32_t)rb);
    /* nf_exp_dd from r on */
    const int ni = v.neg ? -(int)n : (int)n;
    const int j = ni & 127, m = (ni - j) / 128;
    const double thi = nf_exp_tab(2 * j), tlo = nf_exp_tab(2 * j + 1);
    double t = fma(r, 0x1.1111111111111p-7, 0x1.5555555555555p-5);
    t = fma(r, t, 0x1.5555555555555p-3);
    t = fma(r, t, 0.5);
    const double q = fma(r * r, t, r);
    const double w = fma(thi, q, tlo);
    const double er = thi + w;                         /* in [0.99, 2): |p| < 16 scales by bits */
    tail->thi = thi; tail->w = w; tail->er = er; tail->inRange = ok; tail->z = z;
    return nf_ifp_make(nf_ifp_hi(er) + ((uint32_t)m << 20), nf_ifp_lo(er));
}
/* Whether the power's last sum is sure although r's rounding is not: r one unit, 2^(-53 - z),
 * off moves q by less than two units and one of its own rounding, and w, with thi below 2 and
 * its own rounding, by less than sixteen; the sum's error must stay that far from half a unit. */
NF_IFP int nf_pow_settled(const nf_pow_tail *t) {
    const double e = (t->thi - t->er) + t->w;          /* exact: |w| < thi */
    const uint32_t unit = nf_ifp_hi(t->er) & 0x7ff00000u;
    const double gap = nf_ifp_make(unit - (53u << 20), 0u) - fabs(e);
    return t->inRange & ((int32_t)nf_ifp_hi(gap) > (int32_t)((uint32_t)(1023 - 49 - t->z) << 20));
}
NF_IFP double nf_pow_fast(double x, double y) {
    int sure;
    nf_pow_tail tail;
    const double r = nf_pow_try(x, y, &sure, &tail);
    return sure || nf_pow_settled(&tail) ? r : nf_pow_slow(x, y);
}

#endif /* NF_ILOG_H */
