// lsh_ieee.h -- IEEE-754 double division, reciprocal and square root
// (round to nearest even) on the integer pipe.
//
// The GPU's FP64 unit takes one warp instruction per 16 cycles and SM and
// returns it about 55 cycles later; a division or square root built from
// FP64 operations holds it for 5 to 8 of them, one after the other.  The
// forms here hold it for none: schoolbook long division (and the
// digit-by-digit square root) with two digits of about 30 and 24 bits in
// 32-bit integer arithmetic.
//   1. A 32-bit approximation Y of the divisor's reciprocal (of the inverse
//      square root) from the FP32 approximation instruction and one Newton
//      step, biased low so that it never exceeds the exact value.
//   2. The first digit from Y, then the exact remainder.  It is below 2^56,
//      so its low 64 bits are the whole of it, although the products behind
//      it have 85 to 107 bits.
//   3. The second digit from the remainder and Y, low by less than 2 units;
//      the exact second remainder says whether it is one too small.
//   4. The digits are then the exact floor of the result with at least one
//      bit below the last place.  A quotient of two doubles, or a square
//      root of one, is never half way between two doubles, so that bit alone
//      decides the rounding.
// The result does not depend on the approximation instruction's exact bits,
// only on its documented error bound (rcp.approx.ftz.f32: 1 ulp;
// rsqrt.approx.ftz.f32: 2^-22.9 relative); `Seed` supplies it, so that the
// host can run the same steps with any error inside the bound.  Operands or
// results outside the normal range (zero divisors, subnormals, infinities,
// NaN, negative radicands) take the hardware operation; a zero dividend or
// radicand (still water) does not.
//
// Measured on the GB300, against the compiler's FP64 sequences: ns per warp
// operation and SM with all warps busy (less the 9.4 ns of the FP64 add that
// follows in the loop), and cycles of a dependent chain with one warp (less
// that add's 55):
//   reciprocal   1.0 ns against 42.8,  226 cycles against 350
//   division     2.5 ns against 70.0,  290 cycles against 560
//   square root  2.8 ns against 70.0,  245 cycles against 595
// A single-layer edge holds 4 divisions and 3 square roots: of its 200 FP64
// instructions they were 45.  2048^2 fjord step 1.44 -> 1.23 ms, 1024^2 wet
// shelf (second order) 2.13 -> 1.67 ms.
#pragma once

#include "lsh_fpmath.h"

namespace lshm {

LSH_HD uint32_t mulhi32(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

// (hi:lo) << s, its high word; 0 < s < 32
LSH_HD uint32_t funnel_l(uint32_t lo, uint32_t hi, int s) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_l(lo, hi, s);
#else
    return (hi << s) | (lo >> (32 - s));
#endif
}

// low 64 bits of a (bh:bl)
LSH_HD uint64_t mul_lo64(uint32_t a, uint32_t bl, uint32_t bh) {
    return (uint64_t)a * bl + ((uint64_t)(a * bh) << 32);
}

#if defined(__CUDACC__)
struct HwSeed {
    __device__ static float rcp(float x) {
        float y;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
        return y;
    }
    __device__ static float rsqrt(float x) {
        float y;
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
        return y;
    }
};
#endif

// Y <= 2^84 / B < Y + 3.1 for a 53-bit significand B = (bh:bl) in [2^52, 2^53).
// b = B / 2^52 cut to 24 bits and the approximation's 1 ulp put the seed at
// most 4 units of 2^-24 above 1/b; it is taken 5 units low, so b y0 = 1 - d
// with 0 <= d < 2^-20.4, and the Newton step leaves 1 - d^2.  Cutting b to
// 32 bits can lift that by 2^-31, which the final -2 covers.
template <class Seed>
LSH_HD uint32_t recip32(uint32_t bl, uint32_t bh) {
    const float y = Seed::rcp(ffrom_bits(funnel_l(bl, bh, 3) + 0x3f000000u));
    const uint32_t y0 = fbits_of(y) * 256u + (0x80000000u - 5u * 256u);  // y in [1/2, 1] -> y 2^32, less 5 units
    const uint64_t t = (uint64_t)funnel_l(bl, bh, 11) * y0;              // b y0 2^63
    const uint32_t d = (uint32_t)((0 - t) >> 11);                        // (1 - b y0) 2^52
    return y0 + (mulhi32(y0, d) >> 20) - 2u;
}

// 1 / b for eb, the exponent field of b, in [1, 2044]
template <class Seed>
LSH_HD double rcp_normal(uint32_t lo, uint32_t hi) {
    const uint32_t eb = (hi >> 20) & 0x7ffu;
    const uint32_t bh = (hi & 0xfffffu) | 0x100000u;
    const uint64_t B = ((uint64_t)bh << 32) | lo;
    const uint32_t y = recip32<Seed>(lo, bh);
    const uint64_t r1 = 0 - mul_lo64(y, lo, bh);                     // 2^84 - y B, in [0, 3.1 B)
    const uint32_t q2 = mulhi32((uint32_t)(r1 >> 24), y) >> 6;       // r1 2^22 / B, low by < 1.1
    const uint64_t r2 = (r1 << 22) - mul_lo64(q2, lo, bh);           // in [0, 1.1 B)
    uint64_t q = ((uint64_t)y << 22) + q2 + 1u;                      // floor(2^106 / B), and 1 to round
    if (r2 >= B) q += 1u;
    const uint64_t m = q >> 1;                                       // [2^52, 2^53]
    return from_halves((uint32_t)m, (uint32_t)(m >> 32) + ((2044u - eb) << 20) + (hi & 0x80000000u));
}

// a / b for both exponent fields in [1, 2046] and their difference in [-1021, 1022]
template <class Seed>
LSH_HD double div_normal(uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi) {
    const uint32_t ah = (ahi & 0xfffffu) | 0x100000u, bh = (bhi & 0xfffffu) | 0x100000u;
    const uint64_t A = ((uint64_t)ah << 32) | alo, B = ((uint64_t)bh << 32) | blo;
    const uint32_t y = recip32<Seed>(blo, bh);
    const uint32_t q1 = mulhi32(funnel_l(alo, ah, 11), y);           // A / B 2^31, low by < 5.1
    const uint64_t r1 = (A << 31) - mul_lo64(q1, blo, bh);           // in [0, 5.1 B)
    const uint32_t q2 = mulhi32((uint32_t)(r1 >> 24), y) >> 5;       // r1 2^23 / B, low by < 1.2
    const uint64_t r2 = (r1 << 23) - mul_lo64(q2, blo, bh);          // in [0, 1.2 B)
    uint64_t q = ((uint64_t)q1 << 23) + q2;                          // floor(A / B 2^54), in [2^53, 2^55)
    if (r2 >= B) q += 1u;
    const uint32_t s = 1u + (uint32_t)(q >> 54);                     // bits below the last place
    const uint64_t m = (q + s) >> s;                                 // half a unit is 2^(s - 1) = s
    const uint32_t e = ((ahi >> 20) & 0x7ffu) - ((bhi >> 20) & 0x7ffu) + 1020u + s;
    return from_halves((uint32_t)m, (uint32_t)(m >> 32) + (e << 20) + ((ahi ^ bhi) & 0x80000000u));
}

// sqrt(x) for x > 0 and its exponent field in [1, 2046].  x = m 4^k with
// m in [1, 4), M = m 2^52.  y is 1/sqrt(m) 2^32, low by less than 5 units:
// the seed 5 units of 2^-24 low (its error is below 3.2), one Newton step,
// and 3 units for the 32-bit square of the seed.
template <class Seed>
LSH_HD double sqrt_normal(uint32_t lo, uint32_t hi) {
    const uint32_t ex = hi >> 20;
    const uint32_t odd = (ex & 1u) ^ 1u;                             // x = 2^odd b 4^k
    const uint32_t bh = (hi & 0xfffffu) | 0x100000u;
    const uint64_t M = (((uint64_t)bh << 32) | lo) << odd;
    const float f = Seed::rsqrt(ffrom_bits(funnel_l(lo, bh, 3) + 0x3f000000u + (odd << 23)));
    const uint32_t y0 = fbits_of(f) * 256u + (0x80000000u - 5u * 256u);
    const uint32_t mn = (uint32_t)(M >> 22);                         // m 2^30
    const uint64_t t = (uint64_t)mn * mulhi32(y0, y0);               // m y0^2 2^62
    const uint32_t d = (uint32_t)((0 - t) >> 12);                    // (1 - m y0^2) 2^50
    const uint32_t y = y0 + (mulhi32(y0, d) >> 19) - 3u;
    const uint32_t s1 = mulhi32(mn, y);                              // sqrt(m) 2^30, low by < 7
    const uint64_t r1 = (M << 8) - (uint64_t)s1 * s1;                // below 2^35
    const uint32_t s2 = mulhi32((uint32_t)(r1 >> 4), y) >> 4;        // low by < 1.6
    uint64_t s = ((uint64_t)s1 << 23) + s2;
    const uint32_t slo = (uint32_t)s, shi = (uint32_t)(s >> 32);
    const uint64_t sq = (uint64_t)slo * slo + ((uint64_t)(2u * slo * shi) << 32);
    const uint64_t r2 = (M << 54) - sq;                              // M 2^54 - s^2, below 2^56
    if (r2 > 2u * s) s += 1u;                                        // floor(sqrt(m) 2^53)
    s = (s + 1u) >> 1;
    return from_halves((uint32_t)s, (uint32_t)(s >> 32) + ((((ex + 1023u) >> 1) - 1u) << 20));
}

LSH_HD double rcp(double b) {
#if defined(__CUDA_ARCH__)
    uint32_t lo, hi;
    halves(b, lo, hi);
    if (((hi >> 20) & 0x7ffu) - 1u < 2044u) return rcp_normal<HwSeed>(lo, hi);
#endif
    return 1.0 / b;
}

LSH_HD double div(double a, double b) {
#if defined(__CUDA_ARCH__)
    uint32_t alo, ahi, blo, bhi;
    halves(a, alo, ahi);
    halves(b, blo, bhi);
    const uint32_t ea = (ahi >> 20) & 0x7ffu, eb = (bhi >> 20) & 0x7ffu;
    if (eb - 1u < 2046u) {
        if (ea - 1u < 2046u && ea - eb + 1021u <= 2043u) return div_normal<HwSeed>(alo, ahi, blo, bhi);
        if (((ahi << 1) | alo) == 0u) return from_halves(0u, (ahi ^ bhi) & 0x80000000u);
    }
#endif
    return a / b;
}

LSH_HD double root(double x) {
#if defined(__CUDA_ARCH__)
    uint32_t lo, hi;
    halves(x, lo, hi);
    if (hi - 0x00100000u < 0x7fe00000u) return sqrt_normal<HwSeed>(lo, hi);
    if (((hi << 1) | lo) == 0u) return x;
    return ::sqrt(x);
#else
    return std::sqrt(x);
#endif
}

// The same as called functions, for code that holds many of them (the
// adjoint's bodies: about 40 an edge), where inlining each one multiplies
// the kernel's code and spills.
#if defined(__CUDACC__)
#define LSH_CALL static __host__ __device__ __noinline__
#else
#define LSH_CALL inline
#endif
LSH_CALL double rcp_call(double b) { return rcp(b); }
LSH_CALL double div_call(double a, double b) { return div(a, b); }
LSH_CALL double root_call(double x) { return root(x); }
#undef LSH_CALL

}  // namespace lshm
