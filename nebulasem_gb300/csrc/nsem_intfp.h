/*
 * Correctly rounded (nearest, ties to even) double-precision multiplication,
 * division and square root in 32-bit integer arithmetic.
 *
 * Why: GB300 issues about 1.6 FP64 instructions per clock and SM and runs
 * divisions and square roots as 8-10 of them each, while its integer pipes
 * issue about a hundred.  The FP64 kernels are bound by the FP64 pipe, so an
 * operation done here is nearly free of it; IEEE 754 fixes the result, so it
 * is the same bits.  Measured (clocks per operation and SM, 2048 threads
 * resident): division 4.5, by a prepared divisor here 0.72; square root 4.7,
 * here 0.89; product 0.65, here 0.40 and beside the FP64 pipe's additions.
 *
 * Methods (mathematics only):
 *   division: normalised 53-bit significands A, B; a 32-bit reciprocal of B
 *     from a single-precision one and a Newton step, kept below the true
 *     value; two quotient digits (28 + 29 bits) by multiplication and exact
 *     remainder, each an underestimate; the rounding is decided by comparing
 *     the exact remainder with the distance to the next rounding boundary
 *     (a quotient is never a tie);
 *   square root: the same with a reciprocal square root, one digit and a
 *     linear correction, decided by the sign of M - T^2 at the next boundary.
 * Operands outside the normal range, or results near its ends, take the
 * hardware operation.
 */
#ifndef NSEM_INTFP_H
#define NSEM_INTFP_H

#include <stdint.h>

#ifdef __CUDACC__
#define NSEM_IHD __host__ __device__ __forceinline__
#else
#include <math.h>
#include <string.h>
#define NSEM_IHD static inline
#endif

NSEM_IHD uint64_t nsem_bits(double x) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return u;
#endif
}
NSEM_IHD double nsem_from_bits(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t u = (uint64_t)hi << 32 | lo;
    double x;
    memcpy(&x, &u, 8);
    return x;
#endif
}
NSEM_IHD uint32_t nsem_mulhi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)((uint64_t)a * b >> 32);
#endif
}
/* single-precision seeds: 1 / f and 1 / sqrt(f) to a few units in the last
 * place, f normal */
NSEM_IHD float nsem_seed_rcp(float f) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
    return y;
#else
    return 1.0f / f;
#endif
}
NSEM_IHD float nsem_seed_rsqrt(float f) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
    return y;
#else
    return 1.0f / sqrtf(f);
#endif
}
NSEM_IHD float nsem_float_bits(uint32_t u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    memcpy(&f, &u, 4);
    return f;
#endif
}
NSEM_IHD uint32_t nsem_bits_float(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
#endif
}
/* 2^32 y for a seed y in (0.5, 1], lowered by 2^-21 so that it stays below
 * the value it approximates (and below 1) */
NSEM_IHD uint32_t nsem_seed_fix(float y) {
    const uint32_t u = nsem_bits_float(y * (1.0f - 0x1p-21f));
    return ((u & 0x7fffffu) | 0x800000u) << (8 - (126 - (u >> 23)));
}

/* a divisor b = +-B 2^(e - 1075) prepared for nsem_div_by */
typedef struct {
    double b;
    uint64_t B;
    uint32_t r;   /* 2^63 / (B >> 21), from below, within 2^-29 */
} nsem_divisor;

NSEM_IHD nsem_divisor nsem_make_divisor(double b) {
    nsem_divisor d;
    const uint64_t u = nsem_bits(b);
    d.b = b;
    d.B = (u & 0xfffffffffffffull) | 0x10000000000000ull;
    const uint32_t b32 = (uint32_t)(d.B >> 21);
    const uint32_t r0 = nsem_seed_fix(nsem_seed_rcp(nsem_float_bits(0x3f800000u | (uint32_t)(d.B >> 29 & 0x7fffffu))));
    /* one Newton step on the rounded-up B: stays below */
    const uint64_t e = 0x8000000000000000ull - ((uint64_t)b32 * r0 + r0);
    d.r = r0 + nsem_mulhi32(r0, (uint32_t)(e >> 31));
    return d;
}

/* a / d.b */
NSEM_IHD double nsem_div_by(double a, nsem_divisor d) {
    const uint64_t ua = nsem_bits(a), ub = nsem_bits(d.b);
    const uint32_t ah = (uint32_t)(ua >> 32), bh = (uint32_t)(ub >> 32);
    const uint32_t ea = ah >> 20 & 0x7ffu, eb = bh >> 20 & 0x7ffu;
    const uint32_t sign = (ah ^ bh) & 0x80000000u;
    if (!(ea - 1u < 2046u && eb - 1u < 2046u && ea - eb + 900u <= 1800u)) {
        if ((ua << 1) == 0 && eb - 1u < 2046u) return nsem_from_bits(sign, 0);
        return a / d.b;
    }
    const uint64_t A = (ua & 0xfffffffffffffull) | 0x10000000000000ull;
    /* a/b in (0.5, 2): first digit at 2^-28, second at 2^-57 */
    const uint32_t q1 = nsem_mulhi32((uint32_t)(A >> 21), d.r) >> 3;
    const uint64_t r1 = (A << 28) - (uint64_t)q1 * d.B;                /* < 2.5 B */
    const uint32_t q2 = nsem_mulhi32((uint32_t)(r1 >> 23), d.r);
    const uint64_t r2 = (r1 << 29) - (uint64_t)q2 * d.B;               /* < 5 B */
    const uint64_t Q = ((uint64_t)q1 << 29) + q2;                      /* 57 or 58 bits, low by < 5 */
    const uint32_t s = 4u + (uint32_t)(Q >> 57);
    const uint64_t Qh = Q + (1u << (s - 1));
    const uint32_t gap = (1u << s) - ((uint32_t)Qh & ((1u << s) - 1u));
    const uint64_t m = (Qh >> s) + (r2 >= (uint64_t)gap * d.B);
    /* the significand's leading bit adds one to the exponent field */
    const uint64_t out = m + ((uint64_t)(ea - eb + 1017u + s) << 52);
    return nsem_from_bits((uint32_t)(out >> 32) | sign, (uint32_t)out);
}

NSEM_IHD double nsem_div(double a, double b) { return nsem_div_by(a, nsem_make_divisor(b)); }

NSEM_IHD double nsem_sqrt(double a) {
    const uint64_t ua = nsem_bits(a);
    const uint32_t ah = (uint32_t)(ua >> 32);
    if (!(ah - 0x100000u < 0x7fe00000u)) {
        if ((ua << 1) == 0) return a;
        return sqrt(a);
    }
    const uint32_t ea = ah >> 20, odd = (ea & 1u) ^ 1u;                /* e = ea - 1023 odd */
    const uint64_t M0 = (ua & 0xfffffffffffffull) | 0x10000000000000ull;
    const uint64_t M = M0 << odd;                                      /* [2^52, 2^54) */
    const uint32_t r0 = nsem_seed_fix(nsem_seed_rsqrt(nsem_float_bits(
        (0x3f800000u + (odd << 23)) | (uint32_t)(M0 >> 29 & 0x7fffffu))));
    /* Newton step: r = 2^32 / sqrt(m), m = M / 2^52 in [1, 4), from below */
    const uint32_t m32 = (uint32_t)(M >> 22);
    const uint64_t e = 0x4000000000000000ull - ((uint64_t)m32 + 1u) * ((uint64_t)nsem_mulhi32(r0, r0) + 1u);
    const uint32_t r = r0 + (nsem_mulhi32(r0, (uint32_t)(e >> 30)) >> 1);
    /* sqrt(m) at 2^-30, then its correction at 2^-57, both from below */
    const uint32_t g = nsem_mulhi32(m32, r);
    const uint64_t R = (M << 8) - (uint64_t)g * g;                     /* < 2^36 */
    const uint32_t D = nsem_mulhi32((uint32_t)(R >> 4), r);
    const uint64_t S = ((uint64_t)g << 27) + D;                        /* 58 bits, low by < 16 */
    const uint64_t Sh = S + 16u;
    const uint64_t T = ((Sh >> 5) * 2u) + 1u;                          /* next boundary, 16 units */
    const int64_t diff = (int64_t)((M << 54) - T * T);
    const uint64_t m = (Sh >> 5) + (diff >= 0);
    const uint64_t out = m + ((uint64_t)((ea - odd + 1023u) / 2u - 1u) << 52);
    return nsem_from_bits((uint32_t)(out >> 32), (uint32_t)out);
}

/* a factor prepared for nsem_mul_normal: its significand at bit 62 */
typedef struct {
    uint32_t h;        /* high word: sign and exponent */
    uint32_t x1, x0;   /* significand << 10 */
} nsem_factor;

NSEM_IHD nsem_factor nsem_make_factor(double a) {
    nsem_factor f;
    const uint64_t u = nsem_bits(a);
    const uint64_t x = ((u & 0xfffffffffffffull) | 0x10000000000000ull) << 10;
    f.h = (uint32_t)(u >> 32);
    f.x1 = (uint32_t)(x >> 32);
    f.x0 = (uint32_t)x;
    return f;
}

/* the product for operands that are zero or normal with a normal result (the
 * caller has bounded their exponents); zero_hi: the high word of a zero product.
 * About 32 instructions, four of them 32 x 32 + 64-bit multiply-adds. */
NSEM_IHD double nsem_mul_bits(nsem_factor f, double b, uint32_t zero_hi) {
    const uint64_t ub = nsem_bits(b);
    const uint32_t bh = (uint32_t)(ub >> 32), b0 = (uint32_t)ub;
    const uint32_t b1 = (bh & 0xfffffu) | 0x100000u;
    const uint64_t p = (uint64_t)f.x0 * b0;
    const uint64_t t = (uint64_t)f.x1 * b0 + (p >> 32);
    const uint64_t u = (uint64_t)f.x0 * b1 + t;
    const uint64_t H = (uint64_t)f.x1 * b1 + (u >> 32);                /* [2^50, 2^52) */
    const uint32_t norm = (uint32_t)(H >> 51), s = 2u - norm;
    const uint32_t hh = (uint32_t)(H >> 32), hl = (uint32_t)H, ul = (uint32_t)u;
#ifdef __CUDA_ARCH__
    const uint32_t mh = __funnelshift_l(hl, hh, s), ml = __funnelshift_l(ul, hl, s);
    const uint32_t st = min((uint32_t)p, 1u);
#else
    const uint32_t mh = hh << s | hl >> (32u - s), ml = hl << s | ul >> (32u - s);
    const uint32_t st = (uint32_t)p != 0u;
#endif
    /* round to nearest even: the 32 bits below the significand plus half less
     * one, plus one when it is odd or more bits follow, carry into it; the
     * significand's leading bit adds one to the exponent field */
    const uint32_t rem = ul << s, half = 0x7fffffffu + ((ml | st) & 1u);
    const uint32_t base = (f.h & 0xfff00000u) + (bh & 0xfff00000u) - (1024u << 20) + (norm << 20);
    uint32_t lo, hi;
#ifdef __CUDA_ARCH__
    asm("{\n\t.reg .u32 d;\n\tadd.cc.u32 d, %2, %3;\n\taddc.cc.u32 %0, %4, 0;\n\taddc.u32 %1, %5, %6;\n\t}"
        : "=r"(lo), "=r"(hi) : "r"(rem), "r"(half), "r"(ml), "r"(mh), "r"(base));
#else
    const uint64_t m = ((uint64_t)mh << 32 | ml) + (((uint64_t)rem + half) >> 32) + ((uint64_t)base << 32);
    lo = (uint32_t)m;
    hi = (uint32_t)(m >> 32);
#endif
    const int zero = ((f.h & 0x7ff00000u) == 0u) | ((bh & 0x7ff00000u) == 0u);
    return nsem_from_bits(zero ? zero_hi : hi, zero ? 0u : lo);
}

/* a zero product is +0: for sums that start at +0, which show no zero's sign */
NSEM_IHD double nsem_mul_normal(nsem_factor f, double b) { return nsem_mul_bits(f, b, 0u); }

/* a zero product has the sign of its factors */
NSEM_IHD double nsem_mul_signed(nsem_factor f, double b) {
    return nsem_mul_bits(f, b, (f.h ^ (uint32_t)(nsem_bits(b) >> 32)) & 0x80000000u);
}

#endif
