/*
 * fpint.h -- correctly rounded FP64 division, square root and polynomial steps
 * on the integer pipe.
 *
 * GB300 issues one FP64 warp instruction per ~76 cycles and SM sub-partition
 * (64 for a lone warp, however many of its lanes are active), and its division and
 * square root are sequences of about nine of them.  The integer pipe is idle
 * meanwhile, so the operations below do their work on the mantissas as integers.
 * Each returns the value IEEE-754 rounding gives, bit for bit, so code that uses
 * them in place of /, sqrt() and fma() keeps its results; what is outside their
 * range (zeros, subnormals, infinities, NaN, results near the exponent limits) goes
 * to the hardware operation.
 *
 * Division and square root: digit recurrences.  A 32-bit reciprocal (or reciprocal
 * square root) that never exceeds the true one gives ~20 bits of the result at a
 * time, from below; the remainder is exact in wrap-around 64-bit arithmetic, and
 * its last comparison decides the last bit.  Neither operation has ties: a
 * quotient or root that is not representable never lies half-way between two
 * representable numbers.
 *
 * Polynomial step p x + c with |p x| small beside |c| (Taylor series by Horner's
 * rule): the sum stays in c's binade, so it is a 64-bit fixed-point sum with 10 bits
 * below the last one of the result.  Where those bits are too near the rounding
 * boundary to decide (about 1 in 300), the step is an FP64 fma.
 *
 * Measured on one GB300: the FP64 integrator 34.0 -> 20.7 ms on 1.9e5 Ar trajectories and
 * 22.7 -> 13.2 ms on 1.7e5 of H2, the SPANE sampler 9.1 -> 5.5 ms on 1e7 candidates, the
 * collection 3.4 -> 1.6 ms on 4.0e6 electrons, the SPA sampler 28.6 -> 18.8 ms on 3e6
 * candidates; the latency of a lone warp changes little (the integer chains are as long).
 *
 * Compiles as C++ for the host too; the CPU tests compare every operation with the
 * host's own FP64 arithmetic.
 */
#ifndef ETRAJ_FPINT_H
#define ETRAJ_FPINT_H

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define FI_FN static __host__ __device__ __forceinline__
#define FI_NI static __host__ __device__ __noinline__
#else
#define FI_FN static inline
#define FI_NI static inline
#endif

FI_FN uint64_t fi_bits(double x) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    memcpy(&u, &x, sizeof u);
    return u;
#endif
}
FI_FN double fi_real(uint64_t u) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)u);
#else
    double x;
    memcpy(&x, &u, sizeof x);
    return x;
#endif
}
FI_FN uint32_t fi_hi(double x) {
#if defined(__CUDA_ARCH__)
    return (uint32_t)__double2hiint(x);
#else
    return (uint32_t)(fi_bits(x) >> 32);
#endif
}
FI_FN uint32_t fi_lo(double x) {
#if defined(__CUDA_ARCH__)
    return (uint32_t)__double2loint(x);
#else
    return (uint32_t)fi_bits(x);
#endif
}
FI_FN float fi_f(uint32_t u) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float f;
    memcpy(&f, &u, sizeof f);
    return f;
#endif
}
FI_FN uint32_t fi_fbits(float f) {
#if defined(__CUDA_ARCH__)
    return __float_as_uint(f);
#else
    uint32_t u;
    memcpy(&u, &f, sizeof u);
    return u;
#endif
}
FI_FN uint32_t fi_mulhi(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
/* approximate 1/f and 1/sqrt(f), off by at most 2^-23 and 2^-22.9 of them (the PTX
 * manual's bounds); FI_TEST_ERR moves the host's by that many 2^-23 */
FI_FN float fi_rcp_approx(float f) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
    return r;
#elif defined(FI_TEST_ERR)
    return (float)((1.0 / (double)f) * (1.0 + (FI_TEST_ERR) * 1.1920928955078125e-7));
#else
    return 1.0f / f;
#endif
}
FI_FN float fi_rsqrt_approx(float f) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
    return r;
#elif defined(FI_TEST_ERR)
    return (float)((1.0 / sqrt((double)f)) * (1.0 + (FI_TEST_ERR) * 1.1920928955078125e-7));
#else
    return 1.0f / sqrtf(f);
#endif
}
/* d m modulo 2^64 */
FI_FN uint64_t fi_mul64(uint32_t d, uint64_t m) {
    return (uint64_t)d * (uint32_t)m + ((uint64_t)(d * (uint32_t)(m >> 32)) << 32);
}
/* an approximation v of a reciprocal in [1/2, 1] as 2^32 v, lowered by 8 x 2^-24.  The
 * input's truncation raises v by at most 2 x 2^-24 (1/f) or 1 x 2^-24 (1/sqrt f), the
 * approximation moves it by at most 2 x 2^-24 or 2.2 x 2^-24, so the result is never above
 * the true value and below it by at most 10.2 x 2^-24, 2^-19.6 of it; the digits below allow
 * 2^-19.4.  (The tests keep every bit at twice the approximations' errors.) */
FI_FN uint32_t fi_below(float v) { return (fi_fbits(v) - 0x3f000000u - 8u) * 256u + 0x80000000u; }

/* ---- a / b ---------------------------------------------------------------------
 * ma, mb: the mantissas as 53-bit integers, ma doubled when below mb, so that
 * q = ma / mb is in [1, 2); R <= 2^84 / mb.  Digits and remainders, each digit low by
 * e_i >= 0 units (the deficit of R times the digit, and two truncations):
 *   d1 = q 2^29 - e1,           e1 < 2^10.7, r1 = ma 2^29 - d1 mb = e1 mb < 2^63.7
 *   d2 = (r1 / mb) 2^19 - e2,   e2 < 2^10.3, r2 = r1 2^19 - d2 mb = e2 mb < 2^63.4
 *   d3 = (r2 / mb) 2^5 - e3,    e3 < 1.1,    r3 = r2 2^5 - d3 mb < 2 mb
 * and floor(q 2^53) = d1 2^24 + d2 2^5 + d3, plus 1 when r3 >= mb: the result's 53 bits
 * and one more, which rounds it. */
FI_NI double fi_div(double a, double b) {
    const uint32_t ah = fi_hi(a), al = fi_lo(a), bh = fi_hi(b), bl = fi_lo(b);
    const int ea = (int)((ah >> 20) & 0x7ffu), eb = (int)((bh >> 20) & 0x7ffu);
    int e = ea - eb + 1023;
    if (!((uint32_t)(ea - 1) < 2046u && (uint32_t)(eb - 1) < 2046u && (uint32_t)(e - 2) < 2043u)) return a / b;
    uint64_t ma = ((uint64_t)((ah & 0xfffffu) | 0x100000u) << 32) | al;
    const uint64_t mb = ((uint64_t)((bh & 0xfffffu) | 0x100000u) << 32) | bl;
    const uint32_t R = fi_below(fi_rcp_approx(fi_f(((bh & 0xfffffu) << 3) | (bl >> 29) | 0x3f800000u)));
    if (ma < mb) {
        ma <<= 1;
        e -= 1;
    }
    const uint32_t d1 = fi_mulhi((uint32_t)(ma >> 22), R) >> 1;
    const uint64_t r1 = (ma << 29) - fi_mul64(d1, mb);
    const uint32_t d2 = fi_mulhi((uint32_t)(r1 >> 32), R) >> 1;
    const uint64_t r2 = (r1 << 19) - fi_mul64(d2, mb);
    const uint32_t d3 = fi_mulhi((uint32_t)(r2 >> 32), R) >> 15;
    const uint64_t r3 = (r2 << 5) - fi_mul64(d3, mb);
    const uint64_t q = ((uint64_t)d1 << 24) + (((uint64_t)d2 << 5) + d3) + (r3 >= mb ? 2u : 1u);
    return fi_real((q >> 1) + ((uint64_t)((((uint32_t)(e - 1)) << 20) | ((ah ^ bh) & 0x80000000u)) << 32));
}

/* ---- sqrt(a) --------------------------------------------------------------------
 * M: the mantissa as a 53-bit integer, doubled for an odd exponent, so that
 * s = sqrt(M 2^-52) is in [1, 2); Y <= 2^32 / s.  From below, with S_i the root so far:
 *   s1 = s 2^29 - e1,                      e1 < 2^10.7, r1 = M 2^6 - s1^2 < 2^41.7
 *   d2 = r1 2^20 / (2 s 2^29) - ...,       e2 < 2^12.3, r2 = r1 2^40 - d2 (2 s1 2^20 + d2) < 2^63.3
 *   d3 = r2 2^4 / (2 s 2^49) - ...,        e3 < 1.3,    r3 = r2 2^8 - d3 (2 S2 2^4 + d3)
 * and floor(s 2^53) is S3 = S2 2^4 + d3, plus 1 when r3 > 2 S3. */
FI_NI double fi_sqrt(double a) {
    const uint32_t ah = fi_hi(a), al = fi_lo(a);
    if (ah - 0x00100000u >= 0x7fe00000u) return sqrt(a); /* zero, subnormal, negative, infinite, NaN */
    const int e = (int)(ah >> 20) - 1023;
    const int odd = e & 1;
    const uint64_t M = (((uint64_t)((ah & 0xfffffu) | 0x100000u) << 32) | al) << odd;
    const uint32_t Y = fi_below(fi_rsqrt_approx(
        fi_f((((ah & 0xfffffu) << 3) | (al >> 29) | 0x3f800000u) + ((uint32_t)odd << 23))));
    const uint32_t s1 = fi_mulhi((uint32_t)(M >> 22), Y) >> 1;
    const uint64_t r1 = (M << 6) - (uint64_t)s1 * s1;
    const uint32_t d2 = fi_mulhi((uint32_t)(r1 >> 10), Y);
    const uint64_t r2 = (r1 << 40) - fi_mul64(d2, ((uint64_t)s1 << 21) + d2);
    const uint64_t S2 = ((uint64_t)s1 << 20) + d2;
    const uint32_t d3 = fi_mulhi((uint32_t)(r2 >> 32), Y) >> 14;
    const uint64_t r3 = (r2 << 8) - fi_mul64(d3, (S2 << 5) + d3);
    const uint64_t S3 = (S2 << 4) + d3;
    const uint64_t S = S3 + (r3 > 2u * S3 ? 2u : 1u);
    return fi_real((S >> 1) + ((uint64_t)(uint32_t)(((e - odd) >> 1) + 1022) << 52));
}

/* ---- rounding, comparison and scaling ------------------------------------------------ */
/* rint(y) for |y| < 2^19, and the same as an integer */
FI_FN double fi_rint_small(double y, int* k) {
    const uint32_t h = fi_hi(y), l = fi_lo(y), a = h & 0x7fffffffu, sign = h & 0x80000000u;
    const int e = (int)(a >> 20) - 1023;
    uint32_t r, i;
    if (e < 0) {
        i = (a > 0x3fe00000u || (a == 0x3fe00000u && l != 0u)) ? 1u : 0u; /* above 1/2 */
        r = i ? 0x3ff00000u : 0u;
    } else {
        const int sh = 20 - e; /* 2 .. 20 fraction bits in the high word */
        const uint32_t unit = 1u << sh;
        /* (for e = 0 the unit bit is the implicit one: odd) */
        const uint32_t odd = ((a | (e == 0 ? 0x100000u : 0u)) >> sh) & 1u;
        r = (a + (unit >> 1) - 1u + ((l != 0u) ? 1u : odd)) & ~(unit - 1u);
        i = ((r & 0xfffffu) | 0x100000u) >> (20 - ((int)(r >> 20) - 1023));
    }
    *k = sign ? -(int)i : (int)i;
    return fi_real((uint64_t)(r | sign) << 32);
}
/* (double)k, |k| < 2^20 */
FI_FN double fi_from_int(int k) {
    const uint32_t a = (uint32_t)(k < 0 ? -k : k);
    if (a == 0u) return 0.0;
#if defined(__CUDA_ARCH__)
    const int lz = __clz((int)a);
#else
    const int lz = __builtin_clz(a);
#endif
    const uint32_t h = (uint32_t)(1023 + 31 - lz) * 1048576u + (((a << lz) << 1) >> 12);
    return fi_real((uint64_t)(h | ((uint32_t)k & 0x80000000u)) << 32);
}
/* x 2^k; x and the result normal (k may be negative) */
FI_FN double fi_scale(double x, int k) { return fi_real(fi_bits(x) + ((uint64_t)(uint32_t)k << 52)); }
/* x / 2 */
FI_FN double fi_half(double x) {
    return ((fi_hi(x) & 0x7fffffffu) - 0x00200000u < 0x7fd00000u) ? fi_scale(x, -1) : 0.5 * x;
}
/* w = 1 - h and e = (1 - w) - h, for 2^-11 <= h < 1/2: in units of 2^-64, w the multiple of
 * 2^11 nearest 2^64 - h (ties to even), e the exact rest */
FI_FN double fi_one_minus(double h, double* e) {
    const uint32_t hh = fi_hi(h);
    const uint64_t m = ((uint64_t)((hh & 0xfffffu) | 0x100000u) << 32) | fi_lo(h);
    const uint64_t v = 0u - (m << ((hh >> 20) - 1011u));
    const uint64_t w = (v + 0x3ffu + ((v >> 11) & 1u)) & ~(uint64_t)0x7ff;
    const int r = (int)(int64_t)(v - w);
    *e = r ? fi_scale(fi_from_int(r), -64) : 0.0;
    return fi_real((w >> 11) + ((uint64_t)1021u << 52));
}
FI_FN int fi_isnan(double x) { return (fi_bits(x) & 0x7fffffffffffffffull) > 0x7ff0000000000000ull; }
FI_FN int fi_iszero(double x) { return (fi_bits(x) << 1) == 0ull; }
/* a < b, neither NaN */
FI_FN int fi_lt(double a, double b) {
    int64_t i = (int64_t)fi_bits(a), j = (int64_t)fi_bits(b);
    if ((uint64_t)((i | j) << 1) == 0ull) return 0; /* both zero */
    i ^= (int64_t)((uint64_t)(i >> 63) >> 1);
    j ^= (int64_t)((uint64_t)(j >> 63) >> 1);
    return i < j;
}

/* ---- Horner steps ------------------------------------------------------------------
 * p = P 2^(E - 62) with P in [2^62, 2^63), its low 10 bits 0; x = X 2^(ex - 62) likewise. */
typedef struct {
    uint32_t Xh, Xl;
    int ex;
    uint32_t neg; /* 0, or all ones for x < 0 */
    double x;
} fi_arg;
FI_FN fi_arg fi_arg_of(double x) {
    const uint32_t h = fi_hi(x), l = fi_lo(x);
    fi_arg A;
    A.Xh = ((((h & 0xfffffu) | 0x100000u) << 10) | (l >> 22));
    A.Xl = l << 10;
    A.ex = (int)((h >> 20) & 0x7ffu) - 1023; /* x = 0 and subnormals: so small that p x vanishes */
    A.neg = (uint32_t)((int32_t)h >> 31);
    A.x = x;
    return A;
}
FI_FN uint64_t fi_mant(double c) { return ((fi_bits(c) & 0xfffffffffffffull) | 0x10000000000000ull) << 10; }
FI_FN int fi_expo(double c) { return (int)((fi_bits(c) >> 52) & 0x7ffu) - 1023; }
FI_FN double fi_pack(uint64_t P, int E) { return fi_real((P >> 10) + ((uint64_t)(uint32_t)(E + 1022) << 52)); }

/* p x 2^62 in units of the last place of a number with exponent Ec, low by less than 2 */
FI_FN uint64_t fi_term(uint64_t P, int E, const fi_arg* A, int Ec) {
    const uint32_t Ph = (uint32_t)(P >> 32), Pl = (uint32_t)P;
    const uint64_t mid = (uint64_t)Ph * A->Xl + (uint64_t)Pl * A->Xh; /* both below 2^63 */
    const uint64_t hi = (uint64_t)Ph * A->Xh + (uint32_t)(mid >> 32);
    int s = (Ec - E - 2) - A->ex;
    s = s > 63 ? 63 : s;
    return hi >> s;
}
/* The step p <- c + d p x with |c| and |p|: magnitudes (c, |p| > 0), d = +1 or -1 the
 * sign of p x relative to c.  The sum must lie in c's binade, and s above at 1 or more. */
FI_FN uint64_t fi_step_add(uint64_t P, int E, const fi_arg* A, double c) {
    const uint64_t R = fi_mant(c) + 512u + fi_term(P, E, A, fi_expo(c));
    if ((((uint32_t)R + 2u) & 0x3ffu) < 3u) return fi_mant(fma(fi_pack(P, E), A->x, c));
    return R & ~(uint64_t)0x3ff;
}
FI_FN uint64_t fi_step_sub(uint64_t P, int E, const fi_arg* A, double c) {
    const uint64_t R = fi_mant(c) + 512u - fi_term(P, E, A, fi_expo(c));
    if (((uint32_t)R & 0x3ffu) < 2u) return fi_mant(fma(-fi_pack(P, E), A->x, c));
    return R & ~(uint64_t)0x3ff;
}
/* either sign of x, c > 0: c + p x (the complement in place of the negative is low by 1 more) */
FI_FN uint64_t fi_step_any(uint64_t P, int E, const fi_arg* A, double c) {
    const uint64_t m = ((uint64_t)A->neg << 32) | A->neg;
    const uint64_t R = fi_mant(c) + 512u + (fi_term(P, E, A, fi_expo(c)) ^ m);
    if ((((uint32_t)R + 2u) & 0x3ffu) < 3u) return fi_mant(fma(fi_pack(P, E), A->x, c));
    return R & ~(uint64_t)0x3ff;
}

/* ---- the polynomials of detmath.h, step for step --------------------------------------- */
/* e^r - 1 - r over r^2, |r| <= ~ln2/2 (dm_expm1_tail) */
FI_NI double fi_expm1_tail(double r) {
    const fi_arg A = fi_arg_of(r);
    uint64_t P = fi_mant(1.0 / 6227020800.0);
    P = fi_step_any(P, fi_expo(1.0 / 6227020800.0), &A, 1.0 / 479001600.0);
    P = fi_step_any(P, fi_expo(1.0 / 479001600.0), &A, 1.0 / 39916800.0);
    P = fi_step_any(P, fi_expo(1.0 / 39916800.0), &A, 1.0 / 3628800.0);
    P = fi_step_any(P, fi_expo(1.0 / 3628800.0), &A, 1.0 / 362880.0);
    P = fi_step_any(P, fi_expo(1.0 / 362880.0), &A, 1.0 / 40320.0);
    P = fi_step_any(P, fi_expo(1.0 / 40320.0), &A, 1.0 / 5040.0);
    P = fi_step_any(P, fi_expo(1.0 / 5040.0), &A, 1.0 / 720.0);
    P = fi_step_any(P, fi_expo(1.0 / 720.0), &A, 1.0 / 120.0);
    P = fi_step_any(P, fi_expo(1.0 / 120.0), &A, 1.0 / 24.0);
    P = fi_step_any(P, fi_expo(1.0 / 24.0), &A, 1.0 / 6.0);
    return fma(fi_pack(P, fi_expo(1.0 / 6.0)), r, 0.5); /* (crosses a binade for r < 0) */
}
/* the sine's and the cosine's series in r2 <= (pi/4)^2 (dm_sincos) */
typedef struct { double s, c; } fi_pair;
FI_NI fi_pair fi_sincos_poly(double r2) {
    const fi_arg A = fi_arg_of(r2);
    uint64_t S = fi_mant(1.0 / 121645100408832000.0), C = fi_mant(1.0 / 6402373705728000.0);
    S = fi_step_sub(S, fi_expo(1.0 / 121645100408832000.0), &A, 1.0 / 355687428096000.0);
    C = fi_step_sub(C, fi_expo(1.0 / 6402373705728000.0), &A, 1.0 / 20922789888000.0);
    S = fi_step_sub(S, fi_expo(1.0 / 355687428096000.0), &A, 1.0 / 1307674368000.0);
    C = fi_step_sub(C, fi_expo(1.0 / 20922789888000.0), &A, 1.0 / 87178291200.0);
    S = fi_step_sub(S, fi_expo(1.0 / 1307674368000.0), &A, 1.0 / 6227020800.0);
    C = fi_step_sub(C, fi_expo(1.0 / 87178291200.0), &A, 1.0 / 479001600.0);
    S = fi_step_sub(S, fi_expo(1.0 / 6227020800.0), &A, 1.0 / 39916800.0);
    C = fi_step_sub(C, fi_expo(1.0 / 479001600.0), &A, 1.0 / 3628800.0);
    S = fi_step_sub(S, fi_expo(1.0 / 39916800.0), &A, 1.0 / 362880.0);
    C = fi_step_sub(C, fi_expo(1.0 / 3628800.0), &A, 1.0 / 40320.0);
    S = fi_step_sub(S, fi_expo(1.0 / 362880.0), &A, 1.0 / 5040.0);
    C = fi_step_sub(C, fi_expo(1.0 / 40320.0), &A, 1.0 / 720.0);
    S = fi_step_sub(S, fi_expo(1.0 / 5040.0), &A, 1.0 / 120.0);
    C = fi_step_sub(C, fi_expo(1.0 / 720.0), &A, 1.0 / 24.0);
    S = fi_step_sub(S, fi_expo(1.0 / 120.0), &A, 1.0 / 6.0);
    fi_pair v;
    v.s = -fi_pack(S, fi_expo(1.0 / 6.0));
    v.c = fi_pack(C, fi_expo(1.0 / 24.0));
    return v;
}
/* 1/3 + s2/5 + ... + s2^10/23, s2 <= 0.0295 (dm_log) */
FI_NI double fi_log_poly(double s2) {
    const fi_arg A = fi_arg_of(s2);
    uint64_t P = fi_mant(1.0 / 23.0);
    P = fi_step_add(P, fi_expo(1.0 / 23.0), &A, 1.0 / 21.0);
    P = fi_step_add(P, fi_expo(1.0 / 21.0), &A, 1.0 / 19.0);
    P = fi_step_add(P, fi_expo(1.0 / 19.0), &A, 1.0 / 17.0);
    P = fi_step_add(P, fi_expo(1.0 / 17.0), &A, 1.0 / 15.0);
    P = fi_step_add(P, fi_expo(1.0 / 15.0), &A, 1.0 / 13.0);
    P = fi_step_add(P, fi_expo(1.0 / 13.0), &A, 1.0 / 11.0);
    P = fi_step_add(P, fi_expo(1.0 / 11.0), &A, 1.0 / 9.0);
    P = fi_step_add(P, fi_expo(1.0 / 9.0), &A, 1.0 / 7.0);
    P = fi_step_add(P, fi_expo(1.0 / 7.0), &A, 1.0 / 5.0);
    P = fi_step_add(P, fi_expo(1.0 / 5.0), &A, 1.0 / 3.0);
    return fi_pack(P, fi_expo(1.0 / 3.0));
}
/* -1/3 + y2/5 - ... - y2^8/19, y2 <= 0.0097 (dm_atan) */
FI_NI double fi_atan_poly(double y2) {
    const fi_arg A = fi_arg_of(y2);
    uint64_t P = fi_mant(1.0 / 19.0);
    P = fi_step_sub(P, fi_expo(1.0 / 19.0), &A, 1.0 / 17.0);
    P = fi_step_sub(P, fi_expo(1.0 / 17.0), &A, 1.0 / 15.0);
    P = fi_step_sub(P, fi_expo(1.0 / 15.0), &A, 1.0 / 13.0);
    P = fi_step_sub(P, fi_expo(1.0 / 13.0), &A, 1.0 / 11.0);
    P = fi_step_sub(P, fi_expo(1.0 / 11.0), &A, 1.0 / 9.0);
    P = fi_step_sub(P, fi_expo(1.0 / 9.0), &A, 1.0 / 7.0);
    P = fi_step_sub(P, fi_expo(1.0 / 7.0), &A, 1.0 / 5.0);
    P = fi_step_sub(P, fi_expo(1.0 / 5.0), &A, 1.0 / 3.0);
    return -fi_pack(P, fi_expo(1.0 / 3.0));
}
#endif
