/*
 * mkg_math64.h -- double precision division, square root, exp, log, powers
 * and roots of cubics in integer arithmetic.
 * Prepended (as text) to generated double precision kernels; also compiles
 * as host C++ for the tests.
 *
 * GB300 issues one double precision instruction for a warp about every 67
 * cycles per scheduler, and a 32-bit integer instruction every cycle (a
 * 32 x 32 -> 64 multiply-add every two to four). The library's exp is some
 * twenty double precision instructions and its division eight, so in a cell
 * model they are most of a step's time. Here both run on the integer pipes:
 * about 75 and 65 instructions, and no double precision one; the others
 * likewise. Arguments outside the common range go to the library's function.
 *
 * Measured (one time step): with exp and division alone, the launch shape
 * unchanged, a 200-cell Beeler-Reuter cable 24.2 -> 13.8 us, a 256 x 256
 * sheet of a 48-state model 457 -> 218 us. With all of them, and the tile of
 * the cable and the launch shape of the sheet as they are by default now, 2.4
 * and 115 us: 153 double precision instructions per tile and step instead of
 * 727, and 660 instead of 2900; the sheet's step has 25,000 integer ones.
 *
 * The tables mkg_exp_tab and mkg_log_tab are written by the exporter.
 */
#ifndef MKG_MATH64_H
#define MKG_MATH64_H

typedef unsigned int mkg_u32;
typedef unsigned long long mkg_u64;

#ifdef __CUDACC__
#define MKG_M64 static __device__ __forceinline__
#define MKG_M64_SLOW static __device__ __noinline__
/* The functions proper: inlined, or (MKG_M64_OUTLINE) called, where the
 * code of a large model would otherwise not fit the instruction caches */
#ifdef MKG_M64_OUTLINE
#define MKG_M64_FN MKG_M64_SLOW
#else
#define MKG_M64_FN MKG_M64
#endif
MKG_M64 mkg_u32 mkg_mulhi(mkg_u32 a, mkg_u32 b) { return __umulhi(a, b); }
/* Bits 32.. of (hi:lo) << s and bits 0..31 of (hi:lo) >> s, s in 0..31 */
MKG_M64 mkg_u32 mkg_shl(mkg_u32 lo, mkg_u32 hi, mkg_u32 s)
{
    return __funnelshift_l(lo, hi, s);
}
MKG_M64 mkg_u32 mkg_shr(mkg_u32 lo, mkg_u32 hi, mkg_u32 s)
{
    return __funnelshift_r(lo, hi, s);
}
/* 1 / x for the float in [1, 2] whose bits are given: bits of a float in
 * [0.5, 1) within an ulp */
MKG_M64 mkg_u32 mkg_rcp_bits(mkg_u32 b)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(b)));
    return __float_as_uint(fmaxf(y, 0.5f));
}
MKG_M64 mkg_u32 mkg_hi(double x) { return (mkg_u32)__double2hiint(x); }
MKG_M64 mkg_u32 mkg_lo(double x) { return (mkg_u32)__double2loint(x); }
MKG_M64 double mkg_make(mkg_u32 hi, mkg_u32 lo)
{
    return __hiloint2double((int)hi, (int)lo);
}
MKG_M64 mkg_u64 mkg_exp_entry(mkg_u32 j) { return __ldg(mkg_exp_tab + j); }
MKG_M64 mkg_u64 mkg_log_entry(int k, mkg_u32 j)
{
    return __ldg(mkg_log_tab + 2 * j + k);
}
MKG_M64 mkg_u32 mkg_clz(mkg_u32 x) { return (mkg_u32)__clz((int)x); }
/* 1 / sqrt(x) of a float in [1, 4) by its bits: 1.31 fixed point */
MKG_M64 mkg_u32 mkg_rsqrt_fixed(mkg_u32 b)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(b)));
    return __float2uint_rz(y * 2147483648.0f);
}
/* Starting value of mkg_cos_third: z in units of 2^-61, result 2^-63 */
MKG_M64 mkg_u64 mkg_cos_third_start(long long z)
{
    const float f = (float)(int)(z >> 32) * 1.862645149e-9f;
    const float c = cosf(acosf(f) * 0.33333334f);
    return (mkg_u64)__float2uint_rz(c * 2147483648.0f) << 32;
}
/* 1 / (12 c^2 - 3) for c^2 (2.30), 4.28 fixed point */
MKG_M64 mkg_u32 mkg_slope_inverse(mkg_u32 c2)
{
    const float s = (float)(int)(c2 - 0x10000000u) * 1.117587090e-8f;
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(s));
    return __float2uint_rz(y * 268435456.0f);
}
#endif

MKG_M64_SLOW double mkg_exp_slow(double x) { return exp(x); }
MKG_M64_SLOW double mkg_div_slow(double a, double b) { return a / b; }
MKG_M64_SLOW double mkg_sqrt_slow(double x) { return sqrt(x); }
MKG_M64_SLOW double mkg_log_slow(double x) { return log(x); }
MKG_M64_SLOW double mkg_pow_slow(double x, double p) { return pow(x, p); }
MKG_M64_SLOW double mkg_cos_third_slow(double z) { return cos(acos(z) / 3); }

/* a * b / 2^64, low by at most three */
MKG_M64 mkg_u64 mkg_mulhi64(mkg_u64 a, mkg_u64 b)
{
    const mkg_u32 ah = (mkg_u32)(a >> 32), al = (mkg_u32)a;
    const mkg_u32 bh = (mkg_u32)(b >> 32), bl = (mkg_u32)b;
    return (mkg_u64)ah * bh + mkg_mulhi(ah, bl) + mkg_mulhi(al, bh);
}

/*
 * The rest of mkg_exp for |x| = x2:x1:x0 (64 bits after the point, below
 * 708) and its sign s (all ones: negative).
 */
MKG_M64 double mkg_exp_fixed(mkg_u32 x2, mkg_u32 x1, mkg_u32 x0, mkg_u32 s)
{
    /* k = floor(|x| log2(e)) from the leading bits, never too large for
     * x > 0 and never too small (plus one) for x < 0, so that r >= 0 */
    const mkg_u32 t = mkg_shl(x1, x2, 22) + (s & 8u);
    const mkg_u32 k = (mkg_mulhi(t, 0x5c551d94u) >> 20) - s;
    /* The fraction of k ln2, ln2 to 96 bits, and r (mod 1) */
    const mkg_u64 d1 = (mkg_u64)k * 0xd1cf79abu + mkg_mulhi(k, 0xc9e3b398u);
    const mkg_u32 d2 = k * 0xb17217f7u + (mkg_u32)(d1 >> 32);
    const mkg_u64 sm = ((mkg_u64)s << 32) | s;
    mkg_u64 r = (((mkg_u64)x1 << 32) | x0) -
                (((mkg_u64)d2 << 32) | (mkg_u32)d1);
    r = (r ^ sm) - sm;
    const mkg_u64 tab = mkg_exp_entry((mkg_u32)(r >> 56));
    /* g = G 2^-72; S = 1/2 + g (1/6 + g (1/24 + g (1/120 + g/720))) */
    const mkg_u64 G = r << 8;
    const mkg_u32 u = (mkg_u32)(G >> 32);
    const mkg_u32 s5 = mkg_mulhi(u, 1457u) + 2236962u;      /* 2^28, 1/120 */
    const mkg_u32 s4 = (mkg_mulhi(u, s5) + 2863311531u) >> 10;  /* 2^26 */
    const mkg_u32 s3 = mkg_mulhi(u, s4) + 2863311531u;      /* 2^34, 1/6 */
    const mkg_u64 S = (((mkg_u64)u * s3) >> 10) + 0x8000000000000000ull;
    /* p = e^g - 1 = g + g g S, 64 bits after the point */
    const mkg_u64 p = (G >> 8) + (mkg_mulhi64(G, mkg_mulhi64(G, S)) >> 16);
    /* 62 bits after the point, in [1, 2 + 2^-16) */
    mkg_u64 R = tab + mkg_mulhi64(tab, p);
    const mkg_u32 top = (mkg_u32)(R >> 63);
    R += (mkg_u64)(0x200u << top);
    R >>= 10u + top;
    const mkg_u32 ke = (k ^ s) - s + 1022u + top;
    return mkg_make((mkg_u32)(R >> 32) + (ke << 20), (mkg_u32)R);
}

/*
 * e^x, within 0.57 ulp on the device (CUDA's: 0.85, root mean square 0.301
 * against 0.289 here; for |x| < 0.01 0.51, 0.2885 and 0.2887). Table-driven as in P.T.P. Tang, "Table-driven
 * implementation of the exponential function in IEEE floating-point
 * arithmetic" (ACM TOMS 15, 1989), in 64-bit fixed point:
 *   |x| as a fixed-point number, 64 bits after the point (exact for
 *       |x| >= 2^-11);
 *   k with |x| - k ln2 (x < 0: k ln2 - |x|) = r in [0, ln2 + 2^-18);
 *   r = j/256 + g: e^r = e^(j/256) (1 + g (1 + g S(g))), S from the series;
 *   rounded to 53 bits, exponent added.
 */
MKG_M64_FN double mkg_exp(double x)
{
    const mkg_u32 hx = mkg_hi(x), lx = mkg_lo(x);
    const mkg_u32 ax = hx & 0x7fffffffu;
    /* 2^-54 <= |x| < 708 (0x40862000); others (0, tiny, large, inf, NaN) */
    if (ax - 0x3c900000u >= 0x40862000u - 0x3c900000u)
        return mkg_exp_slow(x);
    const mkg_u32 s = (mkg_u32)((int)hx >> 31);     /* all ones: x < 0 */
    /* |x| = m 2^(e-52) = (m << 21) >> (9 - e) with 64 bits after the point */
    const mkg_u32 sh = 1032u - (ax >> 20);          /* 0 .. 63 */
    const mkg_u32 mh = (ax & 0xfffffu) | 0x100000u;
    mkg_u32 m2 = mh >> 11;
    mkg_u32 m1 = mkg_shl(lx, mh, 21);
    mkg_u32 m0 = lx << 21;
    if (sh & 32u) {
        m0 = m1;
        m1 = m2;
        m2 = 0;
    }
    const mkg_u32 b = sh & 31u;
    const mkg_u32 x0 = mkg_shr(m0, m1, b);
    const mkg_u32 x1 = mkg_shr(m1, m2, b);
    const mkg_u32 x2 = m2 >> b;
    return mkg_exp_fixed(x2, x1, x0, s);
}

/*
 * a / b, correctly rounded, by two 30-bit quotient digits from a 31-bit
 * reciprocal of b's significand and the exact remainder (long division as
 * in D.E. Knuth, The Art of Computer Programming 2, 4.3.1, with Newton's
 * iteration for the reciprocal). y: 2^32 / significand, at most that and
 * low by less than 2^3.
 */
MKG_M64 double mkg_div_by(double a, double b, mkg_u32 y)
{
    const mkg_u32 ha = mkg_hi(a), la = mkg_lo(a);
    const mkg_u32 hb = mkg_hi(b), lb = mkg_lo(b);
    const mkg_u32 ea = (ha >> 20) & 0x7ffu, eb = (hb >> 20) & 0x7ffu;
    /* Exponent of the quotient if a's significand is the larger; a, b and
     * the quotient normal numbers, else the general division */
    const mkg_u32 eq = ea - eb + 1023u;
    if (ea - 1u >= 2046u || eb - 1u >= 2046u || eq - 2u >= 2044u)
        return mkg_div_slow(a, b);
    const mkg_u32 ma = (ha & 0xfffffu) | 0x100000u;
    const mkg_u32 mb = (hb & 0xfffffu) | 0x100000u;
    /* First digit: q1 2^-31 <= a/b, low by less than 9 units */
    const mkg_u32 q1 = mkg_mulhi(mkg_shl(la, ma, 11), y);
    /* Remainder (a 2^31 - q1 b), below 2^57 */
    const mkg_u64 pb = (mkg_u64)q1 * lb;
    const mkg_u64 a31 = ((mkg_u64)mkg_shl(la, ma, 31) << 32) | (la << 31);
    const mkg_u64 r1 = a31 - pb - ((mkg_u64)(q1 * mb) << 32);
    /* Second digit, and the quotient in units of 2^-58, low by at most 4 */
    const mkg_u32 q2 = mkg_mulhi((mkg_u32)(r1 >> 25), y);
    const mkg_u64 Q = ((mkg_u64)q1 << 27) + q2;
    const mkg_u32 small = (Q >> 58) ? 0u : 1u;      /* quotient below 1 */
    const mkg_u64 n = Q >> (6u - small);
    /* Exact remainder of the truncated quotient decides the rounding (a
     * quotient of two 53-bit numbers is never half-way) */
    const mkg_u32 nl = (mkg_u32)n, nh = (mkg_u32)(n >> 32);
    const mkg_u64 nb = (mkg_u64)nl * lb +
                       ((mkg_u64)(nl * mb + nh * lb) << 32);
    const mkg_u64 rem = ((mkg_u64)(la << (20u + small)) << 32) - nb;
    const mkg_u64 b53 = ((mkg_u64)mb << 32) | lb;
    const mkg_u64 out = n + ((mkg_u64)((eq - 1u - small) << 20) << 32) +
                        (2 * rem > b53 ? 1u : 0u);
    return mkg_make((mkg_u32)(out >> 32) + ((ha ^ hb) & 0x80000000u),
                    (mkg_u32)out);
}

MKG_M64_FN double mkg_div(double a, double b)
{
    /* Leading 32 bits of b's significand (1.31); the reciprocal of its
     * leading 24 bits, rounded up, to an ulp; then one Newton step, taken
     * two units low so that y b never exceeds 2^32 */
    const mkg_u32 bh = mkg_shl(mkg_lo(b), mkg_hi(b) | 0x100000u, 11);
    const mkg_u32 y0 = (mkg_rcp_bits(
        ((bh >> 8) & 0x7fffffu) + 0x3f800001u) << 8) | 0x80000000u;
    const int e = (int)(0x7ffffffeu - mkg_mulhi(bh, y0));
    const mkg_u32 y = y0 + (mkg_u32)(((long long)e * (long long)y0) >> 31);
    return mkg_div_by(a, b, y);
}

/*
 * Square root, correctly rounded: a reciprocal root good to 27 bits (the
 * device's approximation and one Newton step), the root s1 it gives, the
 * next digits from the remainder, and the exact remainder of the rounded
 * root, which says whether a neighbour is closer ((n + 1/2)^2 = n^2 + n +
 * 1/4).
 */
MKG_M64_FN double mkg_sqrt(double x)
{
    const mkg_u32 hx = mkg_hi(x), lx = mkg_lo(x);
    if (hx - 0x00100000u >= 0x7fe00000u) return mkg_sqrt_slow(x);
    const mkg_u32 eb = hx >> 20;
    const mkg_u32 odd = (eb & 1u) ^ 1u;        /* exponent eb - 1023 odd */
    const mkg_u32 mh = (hx & 0xfffffu) | 0x100000u;
    /* v in [1, 4): 62 bits after the point */
    const mkg_u64 m = ((mkg_u64)mh << 32) | lx;
    const mkg_u64 A = m << (10u + odd);
    const mkg_u32 ah = (mkg_u32)(A >> 32);
    const mkg_u32 y0 = mkg_rsqrt_fixed(
        ((mh << 3 | lx >> 29) & 0x7fffffu) | (0x3f800000u + (odd << 23)));
    /* y0 (1.31); v y0^2 - 1 in units of 2^-28, taken four units high, so
     * that s1 is not above the root */
    const int e = (int)mkg_mulhi(mkg_mulhi(y0, y0), ah) - (1 << 28) + 4;
    const mkg_u32 y = y0 - (mkg_u32)(((long long)e * (long long)y0) >> 29);
    const mkg_u32 s1 = (mkg_u32)(((mkg_u64)ah * y) >> 30);
    const long long r = (long long)(A - (mkg_u64)s1 * s1);
    const mkg_u64 S = ((mkg_u64)s1 << 29) +
                      (mkg_u64)(((r >> 8) * (long long)y) >> 26);
    mkg_u64 n = (S + 128u) >> 8;
    const long long rem = (long long)((m << (52u + odd)) - n * n);
    n += rem > (long long)n ? 1u : 0u;
    n -= rem <= -(long long)n ? 1u : 0u;
    const mkg_u64 out = n + ((mkg_u64)(((eb - odd + 1023u) >> 1) - 1u) << 52);
    return mkg_make((mkg_u32)(out >> 32), (mkg_u32)out);
}

/*
 * log x = e ln2 - log c + log(1 + r), 1 + r = c m exact: c an 11-bit
 * reciprocal of x's significand m, rounded up, by its leading 8 bits (a
 * table, as in P.T.P. Tang, "Table-driven implementation of the logarithm
 * function in IEEE floating-point arithmetic", ACM TOMS 16, 1990). The
 * magnitude in fixed point, 64 bits after the point, within 2^-61; sign:
 * all ones for x < 1.
 */
struct mkg_log_t {
    mkg_u32 i;          /* integer part */
    mkg_u64 f;          /* 64 bits after the point */
    mkg_u32 s;
};

MKG_M64 mkg_log_t mkg_log_fixed(mkg_u32 hx, mkg_u32 lx)
{
    const mkg_u32 mh = (hx & 0xfffffu) | 0x100000u;
    const mkg_u64 tab = mkg_log_entry(0, (hx >> 12) & 0xffu);
    const mkg_u32 c = (mkg_u32)mkg_log_entry(1, (hx >> 12) & 0xffu);
    /* r in units of 2^-63, below 2^-7.4; R: r 2^7, 64 bits */
    const mkg_u64 r63 = (mkg_u64)c * lx + ((mkg_u64)(c * mh) << 32) -
                        0x8000000000000000ull;
    const mkg_u64 R = r63 << 8;
    const mkg_u32 u = (mkg_u32)(R >> 32);
    /* log(1 + r) = r - r^2 (1/2 - r (1/3 - r (1/4 - r (1/5 - ...)))) */
    mkg_u32 a = 715827882u - (mkg_mulhi(u, 613566757u) >> 7);   /* 2^32: 1/6 */
    a = 858993459u - (mkg_mulhi(u, a) >> 7);                    /* 1/5 */
    a = 2147483648u - (mkg_mulhi(u, a) >> 6);                   /* 2^33: 1/4 */
    const mkg_u64 a3 = 0x5555555555555555ull - (((mkg_u64)u * a) >> 8);
    const mkg_u64 a2 = 0x8000000000000000ull - (mkg_mulhi64(R, a3) >> 7);
    const mkg_u64 ra2 = mkg_mulhi64(R, a2) >> 7;
    const mkg_u64 L = tab + (r63 << 1) - (mkg_mulhi64(R, ra2) >> 7);
    /* |e| ln2, then plus or minus L */
    const int e = (int)(hx >> 20) - 1023;
    mkg_log_t g;
    g.s = (mkg_u32)(e >> 31);
    const mkg_u32 k = ((mkg_u32)e ^ g.s) - g.s;
    const mkg_u64 d1 = (mkg_u64)k * 0xd1cf79abu + mkg_mulhi(k, 0xc9e3b398u);
    const mkg_u64 d2 = (mkg_u64)k * 0xb17217f7u + (d1 >> 32);
    const mkg_u64 D = (d2 << 32) | (mkg_u32)d1;
    const mkg_u32 Di = (mkg_u32)(d2 >> 32);
    if (g.s) {
        g.f = D - L;
        g.i = Di - (D < L ? 1u : 0u);
    } else {
        g.f = D + L;
        g.i = Di + (g.f < L ? 1u : 0u);
    }
    return g;
}

/* Logarithm, within 0.52 ulp (CUDA's: 0.54 measured, specified to 1); where
 * its magnitude is below 2^-5 the library's function, which is the more exact
 * there (0.501 ulp; the fixed point is off by 0.53 from 2^-6 and by 0.55 from
 * 2^-7 on) */
MKG_M64_FN double mkg_log(double x)
{
    const mkg_u32 hx = mkg_hi(x);
    if (hx - 0x00100000u >= 0x7fe00000u) return mkg_log_slow(x);
    const mkg_log_t g = mkg_log_fixed(hx, mkg_lo(x));
    const mkg_u32 fh = (mkg_u32)(g.f >> 32), fl = (mkg_u32)g.f;
    if (g.i == 0 ? fh < 0x08000000u : g.i > 0x7fffffffu)
        return mkg_log_slow(x);
    /* The leading one to the top of 64 bits, 53 of them rounded */
    const mkg_u32 z = g.i ? mkg_clz(g.i) : mkg_clz(fh);
    const mkg_u32 w2 = g.i ? g.i : fh, w1 = g.i ? fh : fl,
                  w0 = g.i ? fl : 0u;
    const mkg_u64 W = ((mkg_u64)mkg_shl(w1, w2, z) << 32) |
                      mkg_shl(w0, w1, z);
    const mkg_u32 ex = (g.i ? 1023u + 31u : 1023u - 1u) - z;
    const mkg_u64 n = (W >> 11) + ((W >> 10) & 1u);
    const mkg_u64 out = n + ((mkg_u64)(ex - 1u) << 52);
    return mkg_make((mkg_u32)(out >> 32) | (g.s & 0x80000000u),
                    (mkg_u32)out);
}

/*
 * x^p for a literal p, 2^-8 <= |p| < 16: e^(p log x) with the product in
 * fixed point; P = |p| 2^60 (exact), neg all ones for p < 0. Within 0.6 ulp
 * (CUDA's pow: 1.3).
 */
MKG_M64_FN double mkg_pow_literal(double x, double p, mkg_u64 P, mkg_u32 neg)
{
    const mkg_u32 hx = mkg_hi(x);
    if (hx - 0x00100000u >= 0x7fe00000u) return mkg_pow_slow(x, p);
    const mkg_log_t g = mkg_log_fixed(hx, mkg_lo(x));
    /* g P in units of 2^-124, to 60 bits after the point and four zeros */
    const mkg_u64 lo = mkg_mulhi64(g.f, P);
    const mkg_u32 ph = (mkg_u32)(P >> 32), pl = (mkg_u32)P;
    const mkg_u64 i0 = (mkg_u64)g.i * pl;
    const mkg_u64 i1 = (mkg_u64)g.i * ph + (i0 >> 32);
    const mkg_u64 sum = ((i1 << 32) | (mkg_u32)i0) + lo;
    const mkg_u32 top = (mkg_u32)(i1 >> 32) + (sum < lo ? 1u : 0u);
    const mkg_u32 t2 = (top << 4) | (mkg_u32)(sum >> 60);
    /* Arguments of the exponential outside [2^-40, 700), and x = 1 */
    if (g.i > 1100u || t2 >= 700u || (t2 == 0 && sum < (1ull << 20)))
        return mkg_pow_slow(x, p);
    const mkg_u64 t = sum << 4;
    return mkg_exp_fixed(t2, (mkg_u32)(t >> 32), (mkg_u32)t, g.s ^ neg);
}

/*
 * cos(acos(z) / 3), which cubic roots are written with: the root c in
 * [1/2, 1] of 4 c^3 - 3 c = z, by two Newton steps in fixed point from the
 * single precision value, within 0.6 ulp (CUDA's functions: 2.0). Where the
 * slope vanishes (z near -1) and outside (-1, 1), the library's functions.
 */
MKG_M64_FN double mkg_cos_third(double z)
{
    const mkg_u32 hz = mkg_hi(z);
    const mkg_u32 az = hz & 0x7fffffffu;
    const mkg_u32 sg = (mkg_u32)((int)hz >> 31);
    /* |z| < 1, z >= -(1 - 2^-11) and not tiny */
    if (az >= 0x3ff00000u || az < 0x3c000000u ||
        (sg && az >= 0x3feffc00u))
        return mkg_cos_third_slow(z);
    /* z in units of 2^-61 */
    const mkg_u32 mh = (hz & 0xfffffu) | 0x100000u;
    const mkg_u64 m = ((mkg_u64)mh << 32) | mkg_lo(z);
    const mkg_u32 sh = 1022u - (az >> 20);       /* |z| = m 2^-(53 + sh) */
    const mkg_u64 zm = (m << 8) >> sh;
    const mkg_u64 z61 = (zm ^ (((mkg_u64)sg << 32) | sg)) -
                        (((mkg_u64)sg << 32) | sg);
    mkg_u64 C = mkg_cos_third_start((long long)z61);   /* 2^-63 */
    for (int it = 0; it < 2; ++it) {
        const mkg_u64 c2 = mkg_mulhi64(C, C);          /* 2^-62 */
        const mkg_u64 g = 4u * c2 - 0xc000000000000000ull;   /* 4 c^2 - 3 */
        const bool down = (long long)g < 0;
        const mkg_u64 cg = mkg_mulhi64(C, down ? 0u - g : g);   /* 2^-61 */
        const long long F = (long long)((down ? 0u - cg : cg) - z61);
        const mkg_u32 inv = mkg_slope_inverse((mkg_u32)(c2 >> 32));
        const long long d = it == 0
            ? ((F >> 16) * (long long)inv) >> 12
            : (F * (long long)inv) >> 28;
        C -= (mkg_u64)d << 2;
    }
    const mkg_u64 n = ((C + 512u) >> 10) + ((mkg_u64)1021u << 52);
    return mkg_make((mkg_u32)(n >> 32), (mkg_u32)n);
}

#endif /* MKG_MATH64_H */
