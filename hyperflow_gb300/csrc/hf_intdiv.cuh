// Correctly rounded FP64 division and square root on the integer pipes.
//
// A warp's FP64 addition or product holds the SM's FP64 pipe for 19 cycles, a fused multiply-add for 16
// (measured), in which the SM can issue 76 or 64 others.  An IEEE division built from FP64 Newton steps
// costs about ten FP64 instructions; this one costs none, and about 60 others.  It is schoolbook
// long division with two large digits (see Muller et al., "Handbook of Floating-Point
// Arithmetic", the chapter on division; Moller & Granlund, "Improved division by invariant
// integers", IEEE TC 2011, for quotient digits from a truncated reciprocal):
//
//   a = ma 2^ea, b = mb 2^eb, ma, mb in [2^52, 2^53) (ma doubled when ma < mb, so that the
//   quotient mantissa lies in [1, 2));
//   X ~ 2^84 / mb, 32 bits: an FP32 reciprocal of mb's top 24 bits and one Newton step, always a
//   little low;
//   q1 = ma X / 2^54, 31 bits, and the remainder R1 = ma 2^30 - q1 mb; q2 = R1 X / 2^61, 23 bits
//   more, and the remainder R2 = R1 2^23 - q2 mb: both remainders are below 2^56, so exact modulo
//   2^64, and the digits are never too big;
//   Q = q1 2^23 + q2 is floor(ma 2^53 / mb) or one less, which R2 >= mb decides; the quotient
//   rounds to nearest at Q's lowest bit.
//
// One 32 x 32 -> 64 multiplication per digit and remainder word (9 in all) where a reciprocal
// refined to 64 bits took 64 x 64 -> 128 products.
//
// Every operand outside this fast path -- zero, subnormal, infinite or NaN divisor; a
// subnormal, infinite or NaN dividend; a quotient whose exponent may leave the normal range --
// goes to the hardware division, so the result equals `a / b` bit for bit for all inputs.
// A zero dividend over a normal divisor gives the correctly signed zero directly.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

// The arithmetic helpers compile for the device and for the host (the host build lets the
// CPU test suite run the exact kernel arithmetic against the oracle without a GPU).
#define HF_HD __host__ __device__ __forceinline__

namespace hf {

// The bit pattern of a double and back.  On the device through an opaque register move: from a plain
// reinterpretation the compiler recognises the masks and compares below as absolute values, negations
// and NaN tests and puts them back on the FP64 pipe, the stencils' bottleneck (MUSCL-Hancock at 2048^2
// from the plain reinterpretation: 221 FP64 additions per cell update for the 157 of the scheme,
// 53.1 M FP64 warp instructions and 3.47 ms a launch; through the move 38.7 M and 2.87 ms).
HF_HD uint64_t f64_bits(double x) {
#ifdef __CUDA_ARCH__
    uint64_t u;
    asm("mov.b64 %0, %1;" : "=l"(u) : "d"(x));
    return u;
#else
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return u;
#endif
}
HF_HD double f64_from(uint64_t u) {
#ifdef __CUDA_ARCH__
    double x;
    asm("mov.b64 %0, %1;" : "=d"(x) : "l"(u));
    return x;
#else
    double x;
    std::memcpy(&x, &u, 8);
    return x;
#endif
}
HF_HD uint32_t f32_bits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t u;
    std::memcpy(&u, &x, 4);
    return u;
#endif
}
HF_HD float f32_from(uint32_t u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float x;
    std::memcpy(&x, &u, 4);
    return x;
#endif
}
// FP32 seeds of the Newton iterations: approximate reciprocal and reciprocal square root
// (one special-function instruction each on the device).  The iterations converge from any
// seed within a few ulp, so the host build perturbs the exact value by up to +-4 ulp to
// exercise that margin.
HF_HD float rcp_f32(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    volatile float one = 1.0f;
    const uint32_t b = f32_bits(one / x);
    return f32_from(b + ((b * 2654435761u) >> 29) - 4u);
#endif
}
HF_HD float rsqrt_f32(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    volatile float one = 1.0f;
    const uint32_t b = f32_bits(one / std::sqrt(x));
    return f32_from(b + ((b * 2654435761u) >> 29) - 4u);
#endif
}
// IEEE comparisons on the integer pipes (NaN compares false, -0 equals +0).  A double's
// sign-magnitude bits map to an order-preserving signed key: key = sign ? -|x| : |x|.
constexpr uint64_t kAbs = 0x7FFFFFFFFFFFFFFFull, kInf = 0x7FF0000000000000ull;
HF_HD bool is_nan(double x) { return (f64_bits(x) & kAbs) > kInf; }
HF_HD int64_t order_key(double x) {
    const uint64_t u = f64_bits(x);
    const int64_t m = (int64_t)(u & kAbs);
    return (u >> 63) ? -m : m;
}
HF_HD bool lt(double a, double b) { return !is_nan(a) && !is_nan(b) && order_key(a) < order_key(b); }
HF_HD bool le0(double x) {            // x <= 0.0
    const uint64_t u = f64_bits(x), m = u & kAbs;
    return m == 0 || ((u >> 63) && m <= kInf);
}
HF_HD bool ge0(double x) {            // 0.0 <= x
    const uint64_t u = f64_bits(x), m = u & kAbs;
    return m == 0 || (!(u >> 63) && m <= kInf);
}
HF_HD bool gt0(double x) {            // 0.0 < x: sign clear, not zero, not NaN
    const uint64_t u = f64_bits(x);
    return u != 0 && u <= kInf;
}
// |x| <= t for a positive finite t (false for NaN)
HF_HD bool abs_le(double x, double t) { return (f64_bits(x) & kAbs) <= f64_bits(t); }

// 0.5 * x, equal to the FP64 multiplication for every x, on the integer pipe and without a
// branch: a normal x above the lowest binade has its exponent lowered by one (exact); for
// zeros, subnormals and the lowest normal binade the 53-bit significand-with-exponent-bit
// field is shifted right by one with round to nearest even (a carry into the exponent field
// gives the smallest normal, as the multiplication does); infinities and NaN are returned as
// they are.
HF_HD double half(double x) {
    const uint64_t u = f64_bits(x);
    const uint64_t sgn = u & 0x8000000000000000ull, a = u & 0x7FFFFFFFFFFFFFFFull;
    const uint32_t e = (uint32_t)(a >> 52);
    const uint64_t low = sgn | ((a >> 1) + (a & (a >> 1) & 1ull));   // e <= 1
    const uint64_t r = (e - 2u < 0x7FDu) ? u - (1ull << 52) : (e <= 1u ? low : u);
    return f64_from(r);
}

HF_HD double hw_div(double a, double b) { return a / b; }
HF_HD double hw_sqrt(double x) { return std::sqrt(x); }

// hi and lo words of a 64-bit value, their concatenation, and 32-bit helpers
HF_HD uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }
HF_HD uint32_t lo32(uint64_t x) { return (uint32_t)x; }
HF_HD uint64_t u64_of(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; }
HF_HD uint64_t wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
HF_HD uint32_t umulhi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
// the upper word of (hi:lo) << s, s in 1..31
HF_HD uint32_t fshl32(uint32_t hi, uint32_t lo, uint32_t s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, s);
#else
    return (hi << s) | (lo >> (32 - s));
#endif
}
// a b modulo 2^64 for a 32-bit a and a 64-bit b
HF_HD uint64_t mul_low(uint32_t a, uint64_t b) {
    const uint64_t l = wide(a, lo32(b));
    return u64_of(hi32(l) + a * hi32(b), lo32(l));
}
// y 2^23 for an FP32 value y in (0.5, 1], lowered by a relative 2^-20 so that a seed within a few
// ulp of the true value never exceeds it; no conversion instruction
HF_HD uint32_t seed23(float y) {
    const float low = 1.0f - 9.5367431640625e-7f;
#ifdef __CUDA_ARCH__
    const float v = __fmaf_rn(y, low, 1.0f);
#else
    const float v = std::fmaf(y, low, 1.0f);
#endif
    return f32_bits(v) - 0x3F800000u;
}

constexpr uint32_t kExpHi = 0x7FF00000u, kMantHi = 0x000FFFFFu, kOneHi = 0x00100000u;

// 2^84 / mb rounded down to within 5 units: the 32-bit reciprocal of the 53-bit mantissa mb of a
// normal B, in (2^31, 2^32).  An FP32 seed (19 bits, low), one Newton step from below, and 3 units
// off for the mantissa bits it does not see, so that the quotient's digits never come out too big.
HF_HD uint32_t recip32(uint64_t B) {
    const uint32_t bh = (uint32_t)(B >> 21) | 0x80000000u;               // mb's top 32 bits
    const uint32_t x0 = seed23(rcp_f32(f32_from(0x3F800000u | ((bh >> 8) & 0x7FFFFFu))));
    const uint64_t t = wide(bh, x0);                                     // 2^54 (1 - e)
    return (x0 << 9) - 3u + umulhi32(x0, ~(uint32_t)(t >> 13));          // x0 (1 + e)
}

// the quotient of the fast path (div_fast) from X = recip32(B)
HF_HD double quot32(uint64_t A, uint64_t B, uint32_t X) {
    const uint32_t ha = hi32(A), hb = hi32(B);
    uint64_t ma = u64_of((ha & kMantHi) | kOneHi, lo32(A));
    const uint64_t mb = u64_of((hb & kMantHi) | kOneHi, lo32(B));
    // ma / mb in [1, 2); the exponent field, less the 1 that the mantissa's leading bit adds
    uint32_t e = (ha & kExpHi) - (hb & kExpHi) + (1022u << 20);
    if (ma < mb) {
        ma += ma;
        e -= kOneHi;
    }
    // the first 31 bits, short by at most 6, and their exact remainder below 7 mb
    const uint32_t q1 = umulhi32((uint32_t)(ma >> 22), X);
    const uint64_t r1 = (ma << 30) - mul_low(q1, mb);
    // 23 more bits, short by at most 1; Q = floor(ma 2^53 / mb) or one less, R its remainder
    const uint32_t q2 = umulhi32((uint32_t)(r1 >> 24), X) >> 5;
    const uint64_t r2 = (r1 << 23) - mul_low(q2, mb);
    uint64_t q = wide(q1, 1u << 23) + q2;
    // round to nearest at the lowest of the 54 bits (a quotient of two 53-bit numbers is never a
    // halfway case); the carry out of the mantissa lands in the exponent field
    q = (q + (r2 >= mb ? 2u : 1u)) >> 1;
    return f64_from(u64_of(hi32(q) + e + ((ha ^ hb) & 0x80000000u), lo32(q)));
}

// a / b takes the integer path: both normal, and so is every quotient of their exponents
HF_HD bool div_fast(uint64_t A, uint64_t B) {
    const uint32_t ea = hi32(A) & kExpHi, eb = hi32(B) & kExpHi;
    return (ea - kOneHi < 0x7FE00000u) && (eb - kOneHi < 0x7FE00000u) && (ea - eb + (1021u << 20) < (2044u << 20));
}

// the other operands: a zero over a normal divisor is a signed zero (velocities at rest), the
// rest goes to the hardware
static __host__ __device__ __noinline__ double div_slow(double a, double b) {
    const uint64_t A = f64_bits(a), B = f64_bits(b);
    if ((A << 1) == 0 && (hi32(B) & kExpHi) - kOneHi < 0x7FE00000u)
        return f64_from((A ^ B) & 0x8000000000000000ull);
    return hw_div(a, b);
}

// Kept out of line: one shared copy keeps the general functions inside the instruction cache (measured faster
// than inlining every call, when the stencils made about 55 of them per cell).
static __host__ __device__ __noinline__ double div_rn(double a, double b) {
    const uint64_t A = f64_bits(a), B = f64_bits(b);
    if (!div_fast(A, B)) return div_slow(a, b);
    return quot32(A, B, recip32(B));
}

// Correctly rounded FP64 square root on the integer pipes, digit by digit as the division:
// x = z 4^k with z a 64-bit integer in [2^62, 2^64); Y ~ 2^31 / sqrt(z / 2^64) from an FP32
// reciprocal square root and one Newton step, low by at most 7 units; 32 bits of the root
// sqrt(z), short by at most 16, and their exact remainder; 22 more bits, short by at most 1;
// the exact remainder of the 54-bit root decides that 1, and its lowest bit the rounding (a
// square root is never a halfway case).  Zero, negative, subnormal, infinite and NaN arguments go
// to the hardware sqrt.  Out of line, as div_rn.
HF_HD double root32(uint64_t A) {   // A normal and positive
    const uint32_t h = hi32(A);
    const bool odd = (h & kOneHi) == 0;   // an odd exponent: the mantissa doubled
    uint64_t z = u64_of((h & kMantHi) | kOneHi, lo32(A)) << 10;
    if (odd) z += z;
    const uint32_t zh = hi32(z);
    const uint32_t m23 = (uint32_t)(A >> 29) & 0x7FFFFFu;
    const uint32_t y0 = seed23(rsqrt_f32(f32_from((odd ? 0x40000000u : 0x3F800000u) | m23)));
    const uint64_t t = wide(zh, (uint32_t)(wide(y0, y0) >> 14));         // 2^62 (1 - e)
    const uint32_t Y = (y0 << 9) - 5u + umulhi32(y0, ~(uint32_t)(t >> 22));
    const uint32_t s1 = (uint32_t)(wide(zh, Y) >> 31);
    const uint64_t r1 = z - wide(s1, s1);
    uint64_t s = wide(s1, 1u << 22) + (umulhi32((uint32_t)(r1 >> 5), Y) >> 5);
    const uint64_t sq = wide(lo32(s), lo32(s));
    const uint64_t r2 = u64_of((lo32(z) << 12) - hi32(sq) - 2u * lo32(s) * hi32(s), 0u) - lo32(sq);
    s = (s + (r2 > s + s ? 2u : 1u)) >> 1;
    return f64_from(u64_of(hi32(s) + (((h >> 20) + 1021u) >> 1 << 20), lo32(s)));
}
static __host__ __device__ __noinline__ double sqrt_rn(double x) {
    const uint64_t A = f64_bits(x);
    if (hi32(A) - kOneHi >= 0x7FE00000u) return hw_sqrt(x);
    return root32(A);
}

}  // namespace hf
