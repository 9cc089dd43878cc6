/*
 * mhd_x64.h -- IEEE double division, square root, comparisons and a minmod
 * slope on the 32-bit integer pipe, bit for bit what the FP64 unit gives.
 *
 * The plain form's kernels are bound by the FP64 pipe: it has two lanes per SM,
 * so a warp instruction takes 16 cycles of it while the integer pipes and the
 * schedulers idle.  A division or a square root is eight or nine such
 * instructions; here it is about 75 integer ones, and leaves the pipe to the
 * additions and multiplications (the pipe stays 84 % active, with about 350 FP64
 * instructions per r face where the compiler's division and root take 600).
 *
 * Division and square root are digit recurrences (Ercegovac and Lang, Division
 * and Square Root: Digit-Recurrence Algorithms and Implementations) of three
 * digits of 15 to 22 bits: a digit is the remainder's leading 32 bits times a
 * 22-bit reciprocal (root) rounded down, the remainder is exact in 64-bit
 * integers, and the last digit is corrected until the remainder is below the
 * divisor, which makes the truncated quotient (root) exact.  It has one bit
 * more than a double, and neither a quotient nor a root of doubles ever lies
 * midway between two of them, so adding half an ulp and truncating rounds to
 * nearest.  Zeros, subnormals, infinities, NaNs and results near either end of
 * the exponent range go to the FP64 unit.
 *
 * Plain C++: the host compiles it too, for the tests.
 */
#ifndef MHD_X64_H
#define MHD_X64_H

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define MHD_X64_FN __host__ __device__ __forceinline__
/* division and root are called, not inlined: 24 copies a face do not fit the
 * instruction cache (stalls for want of an instruction 3.3 -> 0.2 per issue) */
#define MHD_X64_CALL static __host__ __device__ __noinline__
#else
#define MHD_X64_CALL static
#define MHD_X64_FN static inline
#endif

namespace mhd {

#ifdef __CUDA_ARCH__
MHD_X64_FN uint32_t x_hi(double a) { return (uint32_t)__double2hiint(a); }
MHD_X64_FN uint32_t x_lo(double a) { return (uint32_t)__double2loint(a); }
MHD_X64_FN double x_of(uint32_t hi, uint32_t lo) { return __hiloint2double((int)hi, (int)lo); }
MHD_X64_FN uint32_t x_mulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
MHD_X64_FN float x_float(uint32_t b) { return __uint_as_float(b); }
MHD_X64_FN uint32_t x_bits(float f) { return __float_as_uint(f); }
/* approximations to 2^-22 */
MHD_X64_FN float x_rcp(float f) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f)); return r; }
MHD_X64_FN float x_rsqrt(float f) { float r; asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f)); return r; }
#else
MHD_X64_FN uint32_t x_hi(double a) { uint64_t u; memcpy(&u, &a, 8); return (uint32_t)(u >> 32); }
MHD_X64_FN uint32_t x_lo(double a) { uint64_t u; memcpy(&u, &a, 8); return (uint32_t)u; }
MHD_X64_FN double x_of(uint32_t hi, uint32_t lo) { uint64_t u = (uint64_t)hi << 32 | lo; double a; memcpy(&a, &u, 8); return a; }
MHD_X64_FN uint32_t x_mulhi(uint32_t a, uint32_t b) { return (uint32_t)((uint64_t)a * b >> 32); }
MHD_X64_FN float x_float(uint32_t b) { float f; memcpy(&f, &b, 4); return f; }
MHD_X64_FN uint32_t x_bits(float f) { uint32_t b; memcpy(&b, &f, 4); return b; }
MHD_X64_FN float x_rcp(float f) { return 1.0f / f; }
MHD_X64_FN float x_rsqrt(float f) { return 1.0f / sqrtf(f); }
#endif

/* a is an infinity or NaN */
MHD_X64_FN bool x_special(double a) { return (x_hi(a) & 0x7ff00000u) == 0x7ff00000u; }
MHD_X64_FN bool x_zero(double a) { return ((x_hi(a) << 1) | x_lo(a)) == 0u; }
/* the magnitude's bits, ordered as the magnitude */
MHD_X64_FN uint64_t x_mag(double a) { return (uint64_t)(x_hi(a) & 0x7fffffffu) << 32 | x_lo(a); }

/* y in [0.5, 1] less 3 2^-23 as a fraction of 2^32: below the number that y,
 * off by 2^-22 at most, approximates */
MHD_X64_FN uint32_t x_frac(float y)
{
    return x_bits(y + 0.99999964f) << 9;
}

/* a / b */
MHD_X64_CALL double x_div(double a, double b)
{
    const uint32_t ah = x_hi(a), bh = x_hi(b), sign = (ah ^ bh) & 0x80000000u;
    const uint32_t ea = ah >> 20 & 0x7ffu, eb = bh >> 20 & 0x7ffu, er = ea - eb + 1023u;
    if (ea - 1u < 2046u && eb - 1u < 2046u && er - 2u < 2043u) {
        const uint64_t ma = (uint64_t)(ah & 0xfffffu | 0x100000u) << 32 | x_lo(a);
        const uint64_t mb = (uint64_t)(bh & 0xfffffu | 0x100000u) << 32 | x_lo(b);
        /* 1 / mb (as a number in [1, 2)) from its leading 24 bits */
        const uint32_t y = x_frac(x_rcp(x_float((uint32_t)(mb >> 29) & 0x7fffffu | 0x3f800000u)));
        const uint32_t q1 = x_mulhi((uint32_t)(ma >> 21), y) >> 10;            /* ma 2^21 / mb */
        const uint64_t r1 = (ma << 21) - q1 * mb;
        const uint32_t q2 = x_mulhi((uint32_t)(r1 >> 24), y) >> 10;            /* r1 2^18 / mb */
        const uint64_t r2 = (r1 << 18) - q2 * mb;
        uint32_t q3 = x_mulhi((uint32_t)(r2 >> 24), y) >> 13;                  /* r2 2^15 / mb */
        uint64_t r3 = (r2 << 15) - q3 * mb;
        if (r3 >= mb) { r3 -= mb; q3++; }
        if (r3 >= mb) { r3 -= mb; q3++; }
        if (r3 < mb) {
            const uint64_t q = ((uint64_t)q1 << 33) + ((uint64_t)q2 << 15) + q3;   /* floor(ma 2^54 / mb) */
            const bool ge = ma >= mb;
            const uint64_t m = ge ? (q + 2u) >> 2 : (q + 1u) >> 1;
            return x_of(sign + ((er - (ge ? 1u : 2u)) << 20) + (uint32_t)(m >> 32), (uint32_t)m);
        }
    }
    if (((ah << 1) | x_lo(a)) == 0u && eb - 1u < 2046u) return x_of(sign, 0u);   /* 0 / b */
    return a / b;
}

/* sqrt(a) */
MHD_X64_CALL double x_sqrt(double a)
{
    const uint32_t ah = x_hi(a), ea = ah >> 20;   /* with the sign: above 0x7ff for a negative */
    if (ea - 1u < 2046u) {
        const uint32_t odd = ~ea & 1u;            /* the unbiased exponent is odd */
        const uint64_t n = ((uint64_t)(ah & 0xfffffu | 0x100000u) << 32 | x_lo(a)) << odd;   /* [1, 4) 2^52 */
        const float mf = x_float(((uint32_t)(n >> (29 + odd)) & 0x7fffffu) + (odd ? 0x40000000u : 0x3f800000u));
        const float yf = x_rsqrt(mf);
        const uint32_t y = x_frac(yf);
        /* leading 22 bits of the root, from below */
        const uint32_t s1 = (x_bits(fmaxf(mf * yf * 0.99999952f, 1.0f)) & 0x7fffffu | 0x800000u) >> 2;
        const uint64_t r1 = n - ((uint64_t)s1 * s1 << 10);
        const uint32_t d2 = x_mulhi((uint32_t)(r1 >> 5), y) >> 9;
        const uint64_t r2 = (r1 << 26) - d2 * (((uint64_t)s1 << 19) + d2);
        const uint64_t s2 = ((uint64_t)s1 << 18) + d2;
        const uint32_t d3 = x_mulhi((uint32_t)(r2 >> 13), y) >> 13;
        uint64_t r3 = (r2 << 28) - d3 * ((s2 << 15) + d3);
        uint64_t s = (s2 << 14) + d3;                                        /* floor(sqrt(n 2^54)), or up to 2 less */
        if (r3 > 2u * s) { r3 -= 2u * s + 1u; s++; }
        if (r3 > 2u * s) { r3 -= 2u * s + 1u; s++; }
        if (r3 <= 2u * s) {
            const uint64_t m = (s + 1u) >> 1;
            return x_of((((ea + 1023u - odd * 1u) >> 1) - 1u << 20) + (uint32_t)(m >> 32), (uint32_t)m);
        }
    }
    return sqrt(a);
}

/* a > b, a >= 0 and a <= 0 */
MHD_X64_FN bool x_gt(double a, double b)
{
    if (x_special(a) || x_special(b)) return a > b;
    const int64_t ma = (int64_t)x_mag(a), mb = (int64_t)x_mag(b);
    return ((int32_t)x_hi(a) < 0 ? -ma : ma) > ((int32_t)x_hi(b) < 0 ? -mb : mb);
}
MHD_X64_FN bool x_ge0(double a) { return ((int32_t)x_hi(a) >= 0 || x_zero(a)) && x_mag(a) <= 0x7ff0000000000000ull; }
MHD_X64_FN bool x_le0(double a) { return ((int32_t)x_hi(a) < 0 || x_zero(a)) && x_mag(a) <= 0x7ff0000000000000ull; }

/* a b > 0, where the factors' exponents show that the product, however it
 * rounds, is neither zero nor NaN; otherwise by the product */
MHD_X64_FN bool x_same_sign(double a, double b)
{
    const uint32_t ea = x_hi(a) >> 20 & 0x7ffu, eb = x_hi(b) >> 20 & 0x7ffu;
    if (ea - 1u < 2046u && eb - 1u < 2046u && ea + eb >= 972u) return (int32_t)(x_hi(a) ^ x_hi(b)) >= 0;
    if ((x_zero(a) && eb < 2047u) || (x_zero(b) && ea < 2047u)) return false;
    return !(a * b <= 0.0);
}
/* of numbers of one sign the one nearest to zero (limiterx.h:200-204, 361-365:
 * the least of positive ones, the greatest of negative ones); infinities and
 * NaNs as the reference's comparisons take them */
MHD_X64_FN double x_nearer(double a, double b)
{
    if (x_special(a) || x_special(b)) return a > 0.0 ? (a > b ? b : a) : (a > b ? a : b);
    return x_mag(a) > x_mag(b) ? b : a;
}
MHD_X64_FN double x_nearest(double a, double b, double c)
{
    if (x_special(a) || x_special(b) || x_special(c)) {
        if (a > 0.0) { b = b > c ? c : b; return a > b ? b : a; }
        b = b > c ? b : c;
        return a > b ? a : b;
    }
    b = x_mag(b) > x_mag(c) ? c : b;
    return x_mag(a) > x_mag(b) ? b : a;
}

/* |a| / a */
MHD_X64_FN double x_sign(double a)
{
    if (x_special(a) || x_zero(a)) return fabs(a) / a;
    return x_of(x_hi(a) & 0x80000000u | 0x3ff00000u, 0u);
}

/* a times s, s the sign of x_sign */
MHD_X64_FN double x_mulsign(double a, double s)
{
    if ((x_hi(s) & 0x7fffffffu) == 0x3ff00000u && x_lo(s) == 0u) return x_of(x_hi(a) ^ (x_hi(s) & 0x80000000u), x_lo(a));
    return a * s;
}
/* (a + a s) / 2, s the sign of x_sign */
MHD_X64_FN double x_doubled_half(double a, double s)
{
    if ((x_hi(a) >> 20 & 0x7ffu) < 2046u && (x_hi(s) & 0x7fffffffu) == 0x3ff00000u && x_lo(s) == 0u)
        return (int32_t)x_hi(s) < 0 ? 0.0 : a;
    return (a + a * s) * 0.5;
}
/* a 2^-1 and a 2^n (n = 1, 2) */
MHD_X64_FN double x_half(double a)
{
    if ((x_hi(a) >> 20 & 0x7ffu) - 2u < 2045u) return x_of(x_hi(a) - 0x100000u, x_lo(a));
    return x_zero(a) ? a : a * 0.5;
}
MHD_X64_FN double x_up(double a, int n)
{
    if ((x_hi(a) >> 20 & 0x7ffu) - 1u < 2043u) return x_of(x_hi(a) + ((uint32_t)n << 20), x_lo(a));
    return x_zero(a) ? a : a * (double)(1 << n);
}

} /* namespace mhd */

#endif
