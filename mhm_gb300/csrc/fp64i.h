/*
 * fp64i.h -- IEEE-754 double comparisons and division on the integer pipe.
 *
 * GB300's FP64 pipe issues ~0.5 T thread-ops/s, and a double compare (DSETP)
 * or the refinement steps of a double division occupy it like an FMA; the
 * integer pipes are tens of times faster.  Sign masks on a double's bits go
 * through hm_abs_bits, or the compiler turns them back into FP64 |x|.  These functions return exactly
 * what the IEEE operations return (round-to-nearest-even), so kernels that
 * use them stay bit-identical to host code using plain C operators.
 *
 * Comparisons: hm_gt/ge/lt/le follow IEEE for all non-NaN operands (+0 == -0,
 * infinities ordered); the *_ieee variants are also false for NaN operands.
 * Division: hm_div(a, b) == a / b for all inputs; normal/zero operands with a
 * normal result take the integer path (float reciprocal seed, two Newton
 * steps in 64-bit fixed point, one product, and the exact remainder where that
 * leaves the rounding open); everything else (subnormal, infinite, NaN, zero
 * divisor, out-of-range results) uses the native division.
 * hm_div_r(a, b, hm_recip_of(b)) is the same division with the divisor's
 * reciprocal computed beforehand.
 */
#ifndef MHM_FP64I_H
#define MHM_FP64I_H

#include "hmath.h"

/* order key: monotone in the value for non-NaN doubles, +0 and -0 -> 0
 * (the sign-cleared bits through hm_abs_bits, which stays on the integer
 * pipe) */
HM_FN int64_t hm_okey(double x)
{
    const uint64_t u = hm_d2b(x);
    const int64_t m = (int64_t)hm_abs_bits(u);
    return (int64_t)u < 0 ? -m : m;
}
HM_FN int hm_isnan_i(double x) { return hm_abs_bits(hm_d2b(x)) > 0x7ff0000000000000ULL; }
HM_FN int hm_gt(double a, double b) { return hm_okey(a) > hm_okey(b); }
HM_FN int hm_ge(double a, double b) { return hm_okey(a) >= hm_okey(b); }
HM_FN int hm_lt(double a, double b) { return hm_okey(a) < hm_okey(b); }
HM_FN int hm_le(double a, double b) { return hm_okey(a) <= hm_okey(b); }
HM_FN int hm_gt_ieee(double a, double b) { return !hm_isnan_i(a) && !hm_isnan_i(b) && hm_gt(a, b); }
HM_FN int hm_lt_ieee(double a, double b) { return !hm_isnan_i(a) && !hm_isnan_i(b) && hm_lt(a, b); }
HM_FN int hm_ge_ieee(double a, double b) { return !hm_isnan_i(a) && !hm_isnan_i(b) && hm_ge(a, b); }
/* x > 0, x < 0 against the constant zero */
HM_FN int hm_gt0(double x) { return hm_okey(x) > 0; }
HM_FN int hm_lt0(double x) { return hm_okey(x) < 0; }
/* c ? a : b as a select of the bit patterns: a select of doubles is issued
 * as an FP64-pipe move on this GPU (measured), an integer select is not */
HM_FN double hm_sel(int c, double a, double b) { return hm_b2d(c ? hm_d2b(a) : hm_d2b(b)); }
/* -x as a flip of the sign bit on the integer pipe (inline PTX on the device,
 * so that it is not turned into an FP64 negation); a + (-b) is exactly a - b */
HM_FN double hm_neg(double x)
{
#if defined(__CUDA_ARCH__)
    uint64_t r;
    asm("xor.b64 %0, %1, 0x8000000000000000;" : "=l"(r) : "l"(hm_d2b(x)));
    return hm_b2d(r);
#else
    return hm_b2d(hm_d2b(x) ^ 0x8000000000000000ULL);
#endif
}
/* min/max with the selection rules of the reference's (a < b ? a : b) */
HM_FN double hm_min_sel(double a, double b) { return hm_sel(hm_lt(a, b), a, b); }

/* reciprocal seed 1/x in float, correctly rounded on host and device */
HM_FN float hm_frcp(float x)
{
#if defined(__CUDA_ARCH__)
    return __frcp_rn(x);
#else
    return 1.0f / x;
#endif
}

HM_FN uint32_t hm_f2b(float f)
{
#if defined(__CUDA_ARCH__)
    return (uint32_t)__float_as_uint(f);
#else
    uint32_t b;
    memcpy(&b, &f, sizeof b);
    return b;
#endif
}

/* 64-bit fixed-point reciprocal of a divisor mantissa Mb in (2^52, 2^53):
 * floor(2^116 / Mb) from a float seed (~24 bits), two Newton steps
 * y' = y (2 - Mb y / 2^116), which approach from below and end less than 3
 * short, and the remainder.  Depends on the divisor only, so a divisor that
 * stays fixed over many divisions (a cell's soil parameters over a chunk of
 * steps) needs it once: hm_recip_of. */
HM_FN uint64_t hm_recip_mant(uint64_t Mb)
{
    const float fy = hm_frcp((float)(uint32_t)(Mb >> 29)); /* in (2^-24, 2^-23] */
    const uint32_t fb = hm_f2b(fy);
    const int sh = (int)((fb >> 23) & 0xffu) - 127 - 23 + 116 - 29; /* 40 or 41 */
    const uint64_t fm = (uint64_t)((fb & 0x7fffffu) | 0x800000u);
    uint64_t inv = (sh >= 41 && fm == 0x800000u) ? 0xffffffffffffffffULL : fm << sh;
    for (int it = 0; it < 2; ++it) {
        /* err = (2^116 - Mb*inv) >> 52, |err| < 2^42: bits 52..115 of the
         * 128-bit difference, from its two limbs */
        const uint64_t t_lo = Mb * inv, t_hi = hm_umulhi(Mb, inv);
        const uint64_t e_lo = (uint64_t)0 - t_lo;
        const uint64_t e_hi = ((uint64_t)1 << 52) - t_hi - (t_lo != 0);
        const int64_t err_s = (int64_t)((e_hi << 12) | (e_lo >> 52));
        inv = inv + (uint64_t)(hm_smulhi((int64_t)(inv >> 1), err_s) * 2);
    }
    uint64_t rem = (uint64_t)0 - Mb * inv; /* 2^116 - Mb*inv, below 3 Mb */
    for (int it = 0; it < 2; ++it)
        if (rem >= Mb) {
            rem -= Mb;
            inv += 1;
        }
    return inv;
}

/* The reciprocal hm_div_r wants for divisor b: 0 for one that is zero,
 * subnormal, infinite or NaN, the largest number for a power of two. */
HM_FN_BIG uint64_t hm_recip_of(double b)
{
    const uint64_t ub = hm_d2b(b);
    const uint32_t ebf = (uint32_t)(ub >> 52) & 0x7ffu;
    const uint64_t Mb = (ub & 0x000fffffffffffffULL) | 0x0010000000000000ULL;
    if (ebf - 1u >= 0x7feu) return 0;
    return Mb == 0x0010000000000000ULL ? 0xffffffffffffffffULL : hm_recip_mant(Mb);
}

/* The divisions hm_div_r leaves: native, or by the exact remainder. */
HM_FN_BIG double hm_div_rest(double a, double b, uint64_t inv)
{
    const uint64_t ua = hm_d2b(a), ub = hm_d2b(b);
    const uint32_t eaf = (uint32_t)(ua >> 52) & 0x7ffu, ebf = (uint32_t)(ub >> 52) & 0x7ffu;
    const uint64_t sign = (ua ^ ub) & 0x8000000000000000ULL;
    if (ebf - 1u >= 0x7feu || (eaf - 1u >= 0x7feu && hm_abs_bits(ua) != 0))
        return a / b; /* b zero/subnormal/inf/NaN, or a subnormal/inf/NaN */
    if (hm_abs_bits(ua) == 0)
        return hm_b2d(sign); /* +-0 / normal */
    uint64_t Ma = (ua & 0x000fffffffffffffULL) | 0x0010000000000000ULL;
    const uint64_t Mb = (ub & 0x000fffffffffffffULL) | 0x0010000000000000ULL;
    int e = (int)eaf - (int)ebf; /* unbiased exponent of the quotient */
    if (Ma < Mb) {
        Ma <<= 1;
        e -= 1;
    }
    if (e > 1023 || e < -1022)
        return a / b; /* overflow or subnormal result: native path */
    /* Q <= Ma * 2^54 / Mb in [2^54, 2^55), at most 2 too small; the remainder
     * Ma*2^54 - Q*Mb is below 2^57, so modulo 2^64 suffices */
    uint64_t Q = (hm_umulhi(Ma, inv) << 2) | ((Ma * inv) >> 62);
    uint64_t r = (Ma << 54) - Q * Mb;
    for (int c = 0; c < 3; ++c)
        if (r >= Mb) {
            Q += 1;
            r -= Mb;
        }
    /* round Q (55 bits: 53 + guard + round) to nearest even */
    uint64_t m53 = Q >> 2;
    const uint32_t g = (uint32_t)(Q & 3u);
    if (g > 2 || (g == 2 && (r != 0 || (m53 & 1))))
        m53++;
    /* m53 in [2^52, 2^53]; a carry to 2^53 moves into the exponent field */
    return hm_b2d(sign | (((uint64_t)(e + 1022) << 52) + m53));
}

/* a / b, correctly rounded, given inv = hm_recip_of(b).
 * The quotient to 63 bits is one high product, less than 4 too small; a
 * quotient of doubles is never halfway between two doubles, so only where the
 * half lies within those 4 (one division in 512) its remainder decides. */
HM_FN_BIG double hm_div_r(double a, double b, uint64_t inv)
{
    const uint64_t ua = hm_d2b(a);
    const uint32_t ha = hm_hi(ua), hb = hm_hi(hm_d2b(b)), sign = (ha ^ hb) & 0x80000000u;
    int e = (int)((ha >> 20) & 0x7ffu) - (int)((hb >> 20) & 0x7ffu);
    uint64_t q = hm_umulhi(ua << 11 | 0x8000000000000000ULL, inv);
    if (!(q >> 63)) {
        q <<= 1;
        e -= 1;
    }
    if (hm_unlikely(inv == 0 || ((ha >> 20) & 0x7ffu) - 1u >= 0x7feu || (uint32_t)(e + 1022) >= 2045u ||
                    (hm_lo(q) & 0x7fcu) == 0x3fcu)) {
        if (inv != 0 && hm_abs_bits(ua) == 0)
            return hm_b2d((uint64_t)sign << 32); /* +-0 / normal */
        return hm_div_rest(a, b, inv);
    }
    return hm_round63(q, e, sign);
}

/* a / b, correctly rounded */
HM_FN_BIG double hm_div(double a, double b) { return hm_div_r(a, b, hm_recip_of(b)); }

/* ---- a horizon's uptake in one go ----
 * With S the soil moisture, pw the wilting point, f the root fraction, a the
 * remaining demand and den = FC - pw (inv = hm_recip_of(den), eden its biased
 * exponent), the actual evapotranspiration of the Feddes stress
 *     r = a * f                        (wet: S >= FC)
 *     r = a * ((f * (S - pw)) / den)   (pw < S < FC)
 * and the storage left, S - r, each of the five operations rounded to nearest
 * even as in FP64, on the integer pipe: one unpacking and one packing instead
 * of a trip to the FP64 pipe for each (64 cycles of it a warp).
 * Returns 0, with nothing written, where the operands leave what it assumes:
 * hm_uptake_par / hm_uptake_var in range, S and pw within 2^11 of each other,
 * r below S / 2, and no carry or tie that needs more than 64 bits. */
HM_FN uint64_t hm_top(uint64_t x) { return x << 11 | 0x8000000000000000ULL; } /* mantissa, leading bit at 63 */
/* a 64-bit mantissa to 53 bits, ties to even (0 with the carry lost) */
HM_FN uint64_t hm_rne11(uint64_t x) { return (x + 0x3ffu + ((hm_lo(x) >> 11) & 1u)) & 0xfffffffffffff800ULL; }
/* positive, within 2^-200 .. 2^200 */
HM_FN int hm_uptake_var(double x) { return hm_hi(hm_d2b(x)) - 0x33700000u < 0x19000000u; }
/* the product of two mantissas, leading bit at 63, its low bits as a sticky
 * bit; *e the exponent it adds */
HM_FN uint64_t hm_mul_top(uint64_t a, uint64_t b, int *e)
{
    uint64_t h = hm_umulhi(a, b), l = a * b;
    *e = 1;
    if (!(h >> 63)) {
        h = h << 1 | l >> 63;
        l <<= 1;
        *e = 0;
    }
    return h | (l != 0);
}
HM_FN int hm_uptake(double S_, double pw_, double f_, double a_, int wet, uint64_t inv, int eden, double *r_, double *left_)
{
    const uint64_t Sb = hm_d2b(S_), pb = hm_d2b(pw_), fb = hm_d2b(f_), ab = hm_d2b(a_);
    const uint64_t S = hm_top(Sb);
    const int es = (int)(hm_hi(Sb) >> 20);
    uint64_t T = hm_top(fb); /* the stress factor */
    int et = (int)(hm_hi(fb) >> 20), e;
    if (!wet) {
        const int d = es - (int)(hm_hi(pb) >> 20);
        uint64_t D = S - (hm_top(pb) >> (d & 63)); /* exact */
        const int lz = hm_clz64(D | 1);
        D = hm_rne11(D << lz);
        const uint64_t P = hm_rne11(hm_mul_top(D, T, &e));
        uint64_t q = hm_umulhi(P, inv);
        et += es - lz + e - eden;
        if (!(q >> 63)) {
            q <<= 1;
            et -= 1;
        }
        T = (q + 0x400u) & 0xfffffffffffff800ULL;
        if (d > 11 || (int32_t)(hm_hi(D) & hm_hi(P) & hm_hi(T)) >= 0 || (hm_lo(q) & 0x7fcu) == 0x3fcu)
            return 0;
    }
    const uint64_t R = hm_rne11(hm_mul_top(hm_top(ab), T, &e));
    const int er = (int)(hm_hi(ab) >> 20) + et + e - 1023;
    const int d = es - er;
    if ((uint32_t)(d - 2) > 60u || (int32_t)hm_hi(R) >= 0)
        return 0;
    const uint64_t y = R >> d, part = (y << d) != R;
    uint64_t D = S - y - part;
    const uint32_t up = (uint32_t)(hm_hi(D) >> 31) ^ 1u; /* below half the binade */
    D = D << up | part;
    const uint64_t m = (D >> 11) + ((hm_lo(D) & 0x7ffu) + ((hm_lo(D) >> 11) & 1u) > 0x400u);
    *left_ = hm_b2d(m + ((uint64_t)(uint32_t)(es - (int)up - 1) << 52));
    *r_ = hm_b2d((R >> 11) + ((uint64_t)(uint32_t)(er - 1) << 52));
    return 1;
}

#endif /* MHM_FP64I_H */
