// soft64.cuh -- IEEE double division, square root and comparisons on the integer and FP32 pipes.
//
// GB300 issues one FP64 warp instruction per SM sub-partition every ~64 cycles (2 lanes per SM
// and clock) and a compiled double division or square root is ten of them or more, so the FP64
// kernels of this path were bound by that pipe while the integer and FP32 pipes idled.  The
// functions below give the correctly rounded (round to nearest, ties to even) IEEE result, the
// same bits as the hardware's instruction sequence, without any FP64 instruction for normal
// operands with a normal result; zeros, subnormals, infinities, NaN and results next to the
// exponent limits go to the hardware operation.
//
//   div:  schoolbook long division of the 53-bit significands in three digits of 21, 20 and 12
//         bits.  Each digit is the remainder's leading bits times an FP32 reciprocal of the
//         divisor that is biased low, so a digit is never too large; the remainders are exact
//         64-bit integers (two 32-bit multiplies a digit).  A quotient of two 53-bit significands
//         is never half-way between two doubles, so 54 quotient bits decide the rounding.
//   sqrt: the same digit recurrence, R - d (2 s + d), from an FP32 reciprocal square root.  A digit is never
//         too large if y <= (1 - 2^-24) / r for the root r (the product that forms it may round up by 2^-24).
//         With an approximation off by at most 2^-22 and one rounding of y, a bias of 3 x 2^-23 leaves that:
//         (1 + 2^-22) (1 - 1.5 x 2^-22) (1 + 2^-24) < 1 - 2^-24.  The other way a digit falls short by
//         less than 8, 15 and 2 units (the bounds below), so that the remainders keep to their 23 leading bits.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define SX_FN __host__ __device__ __forceinline__
#define SX_RARE static __host__ __device__ __noinline__
#else
#define SX_FN inline
#define SX_RARE static
#endif

namespace sx {

SX_FN uint64_t bits_of(double x) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return u;
#endif
}
SX_FN double of_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double x;
    memcpy(&x, &u, 8);
    return x;
#endif
}
SX_FN uint32_t fbits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t u;
    memcpy(&u, &x, 4);
    return u;
#endif
}
SX_FN float fof(uint32_t u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float x;
    memcpy(&x, &u, 4);
    return x;
#endif
}
// 1/x and 1/sqrt(x) to within 2^-22 relative (the hardware approximations, documented at 1 ulp and
// 2^-22.9; the rounded functions on the host, where a test may put others within 2^-22): the callers' bias covers
// either
#ifndef SX_HOST_RCP
#define SX_HOST_RCP(x) (1.0f / (x))
#define SX_HOST_RSQRT(x) (1.0f / sqrtf(x))
#endif
SX_FN float rcp_approx(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return SX_HOST_RCP(x);
#endif
}
SX_FN float rsqrt_approx(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return SX_HOST_RSQRT(x);
#endif
}
// an integer below 2^23 as a float, and the integer part of a float in [0, 2^23): through the
// significand of 2^23 + x, without the conversion unit
SX_FN float small_float(uint32_t x) { return fof(0x4b000000u | x) - 8388608.0f; }
SX_FN uint32_t small_int(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(__fadd_rd(x, 8388608.0f)) & 0x7fffffu;
#else
    return (uint32_t)x;
#endif
}
SX_FN uint64_t mul64x32(uint64_t b, uint32_t d) {       // b * d mod 2^64
    return (uint64_t)(uint32_t)b * d + ((uint64_t)((uint32_t)(b >> 32) * d) << 32);
}

constexpr uint64_t FRAC = 0xfffffffffffffull, IMPL = 0x10000000000000ull;

// operands or results outside the integer forms.  A zero numerator over a normal divisor is the
// common one (a component at rest): signed zero, without the hardware division.
SX_RARE double div_rare(double a, double b) {
    const uint64_t ua = bits_of(a), ub = bits_of(b);
    const uint32_t eb = (uint32_t)(ub >> 52) & 0x7ffu;
    if ((ua << 1) == 0 && eb - 1u < 2046u) return of_bits((ua ^ ub) & 0x8000000000000000ull);
    return a / b;
}

SX_FN double div(double a, double b) {
    const uint64_t ua = bits_of(a), ub = bits_of(b);
    const uint32_t ea = (uint32_t)(ua >> 52) & 0x7ffu, eb = (uint32_t)(ub >> 52) & 0x7ffu;
    uint64_t A = (ua & FRAC) | IMPL;
    const uint64_t B = (ub & FRAC) | IMPL;
    const uint32_t lt = A < B ? 1u : 0u;
    const uint32_t e = ea - eb + 1022u - lt;             // biased exponent of the result, less 1
    if (!(ea - 1u < 2046u && eb - 1u < 2046u && e - 1u < 2043u)) return div_rare(a, b);
    A <<= lt;                                            // A / B in [1, 2)
    // y <= 2^52 / B, by less than 13 * 2^-24 relative: the divisor's leading 24 bits rounded up
    const uint32_t bhi = (uint32_t)(ub >> 32), blo = (uint32_t)ub;
    const float fb = fof((((bhi << 3) | (blo >> 29)) & 0x7fffffu) + 0x3f800001u);
    const float y = rcp_approx(fb) * 0.99999952316284179688f;     // 1 - 2^-21
    // digit 1 (below 2^22): A / B in units of 2^-21, at most 6 too small
    const uint32_t d1 = small_int(small_float((uint32_t)(A >> 31)) * y);
    uint64_t R = (A << 21) - mul64x32(B, d1);            // < 6 B
    // digit 2 (below 2^23): units of 2^-41, at most 8 too small
    const uint32_t d2 = small_int(small_float((uint32_t)(R >> 33)) * (y * 2.0f));
    R = (R << 20) - mul64x32(B, d2);                     // < 8 B
    // digit 3 (below 2^15 + 8): units of 2^-53, at most 1 too small
    const uint32_t d3 = small_int(small_float((uint32_t)(R >> 33)) * (y * 0.0078125f));
    R = (R << 12) - mul64x32(B, d3);                     // < 2 B
    const uint64_t N = ((uint64_t)d1 << 32) + ((uint64_t)d2 << 12) + (d3 + (R >= B ? 1u : 0u));   // floor, 54 bits
    // rounding to 53 bits; the implicit bit carries into the exponent field
    const uint64_t sign = (ua ^ ub) & 0x8000000000000000ull;
    return of_bits(sign | (((uint64_t)e << 52) + ((N + 1) >> 1)));
}

// comparisons (an FP64 instruction each): the bit patterns as integers in the order of the values (both
// zeros 0), false with a NaN; face fluxes of 1,966,080 cells 15.62 -> 15.40 ms, an iteration 25.03 -> 24.71
SX_FN bool is_nan(double a) { return (bits_of(a) << 1) > 0xffe0000000000000ull; }
SX_FN int64_t order_of(double a) {
    const int64_t u = (int64_t)bits_of(a);
    return u < 0 ? (int64_t)(0x8000000000000000ull - (uint64_t)u) : u;
}
SX_FN bool less(double a, double b) { return order_of(a) < order_of(b) && !is_nan(a) && !is_nan(b); }
SX_FN bool less_equal(double a, double b) { return order_of(a) <= order_of(b) && !is_nan(a) && !is_nan(b); }
SX_FN bool equal(double a, double b) { return order_of(a) == order_of(b) && !is_nan(a) && !is_nan(b); }

SX_RARE double sqrt_rare(double a) { return ::sqrt(a); }

SX_FN double sqrt(double a) {
    const uint64_t ua = bits_of(a);
    const uint32_t ea = (uint32_t)(ua >> 52);            // sign included
    if (!(ea - 1u < 2046u)) return sqrt_rare(a);
    // a = X 2^-52 2^(2 h), X in [2^52, 2^54)
    const uint32_t odd = (ea & 1u) ^ 1u;                 // the unbiased exponent is odd
    const uint64_t X = ((ua & FRAC) | IMPL) << odd;
    const uint32_t e = ((ea + 1023u - odd) >> 1) - 1u;   // biased exponent of the root, less 1
    // y <= (1 - 2^-24) / sqrt(X 2^-52)
    const float x24 = small_float((uint32_t)(X >> 31));                        // in units of 2^-21
    const float y = rsqrt_approx((x24 + 1.0f) * 4.76837158203125e-7f) * 0.99999964237213134765625f;  // 1 - 3 2^-23
    // digit 1 (below 2^23): the root in units of 2^-22, too small by less than 3 r + 2 / r + 0.75 < 8
    const uint32_t d1 = small_int(x24 * (y * 2.0f));
    uint64_t R = X - (((uint64_t)d1 * d1) << 8);         // 2^8 times the remainder, < 2^35
    // digit 2 (below 2^23): units of 2^-42, less than 15 too small
    const uint32_t d2 = small_int(small_float((uint32_t)(R >> 13)) * (y * 4.0f));
    R = (R << 32) - mul64x32(((uint64_t)d1 << 21) + d2, d2);                   // < 60 x 2^42
    const uint64_t s = ((uint64_t)d1 << 20) + d2;
    // digit 3: units of 2^-53, at most 1 too small
    const uint32_t d3 = small_int(small_float((uint32_t)(R >> 25)) * (y * 0.0078125f));
    R = (R << 22) - mul64x32((s << 12) + d3, d3);
    uint64_t N = (s << 11) + d3;
    N += R > 2 * N ? 1u : 0u;
    return of_bits(((uint64_t)e << 52) + ((N + 1) >> 1));
}

}  // namespace sx

namespace tg {

// A double whose divisions and square roots take the forms above.  Same size and layout as
// double (the slot arrays are read through either), and every operation rounds as the
// double's does, so a kernel keeps its results bit for bit.
struct f64 {
    double v;
    f64() = default;
    SX_FN constexpr f64(double x) : v(x) {}
    SX_FN explicit operator double() const { return v; }
    SX_FN explicit operator float() const { return (float)v; }
    SX_FN f64 operator-() const { return f64(-v); }
};
SX_FN f64 operator+(f64 a, f64 b) { return f64(a.v + b.v); }
SX_FN f64 operator-(f64 a, f64 b) { return f64(a.v - b.v); }
SX_FN f64 operator*(f64 a, f64 b) { return f64(a.v * b.v); }
SX_FN f64 operator/(f64 a, f64 b) {
    return f64(sx::div(a.v, b.v));
}
SX_FN bool operator<(f64 a, f64 b) { return sx::less(a.v, b.v); }
SX_FN bool operator>(f64 a, f64 b) { return sx::less(b.v, a.v); }
SX_FN bool operator<=(f64 a, f64 b) { return sx::less_equal(a.v, b.v); }
SX_FN bool operator>=(f64 a, f64 b) { return sx::less_equal(b.v, a.v); }
SX_FN bool operator==(f64 a, f64 b) { return sx::equal(a.v, b.v); }
SX_FN bool operator!=(f64 a, f64 b) { return !sx::equal(a.v, b.v); }
using ::sqrt;
using ::fabs;
SX_FN f64 sqrt(f64 a) { return f64(sx::sqrt(a.v)); }
SX_FN f64 fabs(f64 a) { return f64(::fabs(a.v)); }

}  // namespace tg
