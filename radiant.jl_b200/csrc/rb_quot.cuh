// rb_quot.cuh -- quotients q / s of the sweeps, whose divisor s (a cell's collision term) is known
// before the dividend q (which waits for the cell's faces).
//
// With r near 1/s, v = q·r is within a few units in the last place of q/s, the residual q − s·v is
// exact in an FMA, and v + (q − s·v)·r is q/s but for a rounding and (a few units)·(the relative
// error of r): the method of P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor" (1990). The result is within half a unit in the last place and 2^-50 of one
// (FP32: 2^-22) of q/s, so it is the correctly rounded quotient unless q/s lies that close to the
// middle of two numbers. It holds where nothing on the way overflows and the residual does not
// underflow, which quot_in asks of q and quot_div_in of s; anything else (infinities, NaN, the ends
// of the exponent range, divisors that are not positive) takes the division. A zero q passes and
// keeps its sign. tests/test_quotients.py compares quot() with the division over the whole range.
//
// No branch stands between the quotients of a cell's directions (3D) or of a row's cells (2D), so
// their chains overlap: the callers look at all of them first, or afterwards, and branch once.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

namespace rb {

// a double's two words, and back; a float's bits, and back
__host__ __device__ __forceinline__ void quot_words(double x, uint32_t &hi, uint32_t &lo) {
#ifdef __CUDA_ARCH__
    hi = (uint32_t)__double2hiint(x);
    lo = (uint32_t)__double2loint(x);
#else
    uint64_t b;
    memcpy(&b, &x, 8);
    hi = (uint32_t)(b >> 32);
    lo = (uint32_t)b;
#endif
}
__host__ __device__ __forceinline__ double quot_double(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t b = (uint64_t)hi << 32 | lo;
    double x;
    memcpy(&x, &b, 8);
    return x;
#endif
}
__host__ __device__ __forceinline__ uint32_t quot_bits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t b;
    memcpy(&b, &x, 4);
    return b;
#endif
}
__host__ __device__ __forceinline__ float quot_float(uint32_t b) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float x;
    memcpy(&x, &b, 4);
    return x;
#endif
}

// 2^-900 <= |q| < 2^900 or zero; with 2^-100 <= s < 2^100 the quotient stays within 2^±1000 and
// the residual (a multiple of 2^-105·|q|) above the smallest subnormal
__host__ __device__ __forceinline__ bool quot_in(double q) {
    uint32_t hi, lo;
    quot_words(q, hi, lo);
    hi &= 0x7fffffffu;
    return (hi - ((1023u - 900u) << 20) < 1800u << 20) | ((hi | lo) == 0);
}
__host__ __device__ __forceinline__ bool quot_div_in(double s) {
    uint32_t hi, lo;
    quot_words(s, hi, lo);
    return hi - ((1023u - 100u) << 20) < 200u << 20;
}
// FP32: 2^-90 <= |q| < 2^90 or zero, 2^-30 <= s < 2^30
__host__ __device__ __forceinline__ bool quot_in(float q) {
    const uint32_t b = quot_bits(q) & 0x7fffffffu;
    return (b - ((127u - 90u) << 23) < 180u << 23) | (b == 0);
}
__host__ __device__ __forceinline__ bool quot_div_in(float s) {
    return quot_bits(s) - ((127u - 30u) << 23) < 60u << 23;
}

// 1 / s within a unit in the last place (quot_div_in(s)). FP64: r0, the approximate FP32 reciprocal
// of s cut to 24 bits; its relative error e = 1 − s·r0 (below 2^-21), then r0·(1 + e + e²), the
// series of 1/(1 − e) up to e³ < 2^-63. The words are moved between the formats by shifts: the
// conversions run at a quarter of their rate (two a quotient cost the 3D FP64 sweep 4 %).
__host__ __device__ __forceinline__ double quot_rcp(double s) {
    uint32_t hi, lo;
    quot_words(s, hi, lo);
    const uint32_t bias = (1023u - 127u) << 20;
    const float f = quot_float((hi - bias) << 3 | lo >> 29);
    float rf;
#ifdef __CUDA_ARCH__
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(f));
#else
    rf = 1.0f / f;
#endif
    const uint32_t b = quot_bits(rf);
    const double r0 = quot_double((b >> 3) + bias, b << 29);
    const double e = fma(-s, r0, 1.0);
    return fma(r0, fma(e, e, e), r0);
}
__host__ __device__ __forceinline__ float quot_rcp(float s) {
#ifdef __CUDA_ARCH__
    return __frcp_rn(s);
#else
    return 1.0f / s;
#endif
}

// q / s given r = quot_rcp(s) (quot_in(q), quot_div_in(s)); the residual's sign is turned so that a
// zero keeps the sign of q / s
__host__ __device__ __forceinline__ double quot_by(double q, double s, double r) {
    const double v = q * r;
    return fma(-fma(s, v, -q), r, v);
}
__host__ __device__ __forceinline__ float quot_by(float q, float s, float r) {
    const float v = q * r;
    return fmaf(-fmaf(s, v, -q), r, v);
}

// any q and s
template <typename R>
__host__ __device__ __forceinline__ R quot(R q, R s) {
    return quot_in(q) && quot_div_in(s) ? quot_by(q, s, quot_rcp(s)) : q / s;
}

}  // namespace rb
