// Conversions between FP32 and the 64-bit fixed-point density sums, in 32-bit
// integer arithmetic only.  Both round to nearest, ties to even, exactly like
// __float2ll_rn / __ll2float_rn on their ranges, but conversions to and from
// 64-bit types issue on the FP64 pipe, which runs at a small fraction of the
// FP32 rate on GB300; the density scatter converts every (cell, bin)
// contribution and the row pass every bin.
//
// The header compiles for the device and for the host, so that a host program
// can check the routines against the C library's conversions.
#pragma once

#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define ERP_FXP_FN __host__ __device__ __forceinline__
#else
#define ERP_FXP_FN static inline
#endif

namespace erp {

ERP_FXP_FN uint32_t fxp_float_bits(float v) {
#if defined(__CUDA_ARCH__)
    return __float_as_uint(v);
#else
    uint32_t b;
    memcpy(&b, &v, sizeof b);
    return b;
#endif
}

ERP_FXP_FN float fxp_bits_float(uint32_t b) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(b);
#else
    float v;
    memcpy(&v, &b, sizeof v);
    return v;
#endif
}

ERP_FXP_FN int fxp_clz32(uint32_t x) {   // x != 0
#if defined(__CUDA_ARCH__)
    return __clz((int)x);
#else
    return __builtin_clz(x);
#endif
}

// rint(v) for v in [0, 2^63) (round half to even).  Outside that range
// (negative, >= 2^63, infinite or NaN: the caller's error) the result is 0.
// A float of exponent field e holds the integer mantissa m (24 bits with the
// hidden one) times 2^(e - 150).
ERP_FXP_FN uint64_t fxp_rint_u64(float v) {
    const uint32_t b = fxp_float_bits(v);
    if (b >> 31) return 0;
    const int e = (int)(b >> 23);
    if (e < 126 || e >= 190) return 0;   // v < 0.5 (zero and subnormals included), or v >= 2^63
    const uint32_t m = (b & 0x7fffffu) | 0x800000u;
    if (e >= 150) return (uint64_t)m << (e - 150);   // already an integer
    const int sh = 150 - e;   // 1 .. 24
    uint32_t q = m >> sh;
    const uint32_t rem = m & ((1u << sh) - 1u), half = 1u << (sh - 1);
    q += (rem > half || (rem == half && (q & 1u))) ? 1u : 0u;
    return q;
}

// a b + 2^23 rounded towards minus infinity, for a b in [0, 2^23).  On the host the sum
// is formed in FP64, where nothing of it is lost that could reach the next integer (a is
// a float, b a power of two), and rounded to the float below.
ERP_FXP_FN float fxp_fma_down_2p23(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fmaf_rd(a, b, 8388608.0f);
#else
    const double sum = (double)a * (double)b + 8388608.0;
    const float t = (float)sum;
    return (double)t > sum ? fxp_bits_float(fxp_float_bits(t) - 1u) : t;
#endif
}
ERP_FXP_FN float fxp_fma(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
    return __fmaf_rn(a, b, c);
#else
    return __builtin_fmaf(a, b, c);
#endif
}

// floor(x 2^-b) for x in [0, 2^(b + 23)) as an integer, by adding 2^23 rounded down (the
// sum's low bits are that integer); x - floor 2^b exactly.  The host runs the same
// operations, so its test of the pieces is one of the device's arithmetic.
ERP_FXP_FN float fxp_high_part(float x, float inv_pow, float pow, uint32_t &high) {
    const float t = fxp_fma_down_2p23(x, inv_pow);
    high = fxp_float_bits(t) - 0x4b000000u;
    return fxp_fma(-(t - 8388608.0f), pow, x);
}

// rint(x) (round half to even, as fxp_rint_u64) as s0 + s1 2^B with s0 < 2^B, for x in
// [0, 2^2B), B = 21..23: nine FP32 and integer instructions and no conversion (those
// issue at a quarter of the rate).  The low part's own rounding to an integer, by
// adding 2^23, may reach 2^B and then carries.
template <int B>
ERP_FXP_FN void fxp_split2(float x, uint32_t &s0, uint32_t &s1) {
    static_assert(B >= 21 && B <= 23, "pieces");
    uint32_t high;
    const float r = fxp_high_part(x, 1.0f / (float)(1u << B), (float)(1u << B), high);
    const uint32_t low = fxp_float_bits(r + 8388608.0f) - 0x4b000000u;   // 0 .. 2^B
    s1 = high + (low >> B);
    s0 = low & ((1u << B) - 1u);
}
// ... as s0 + s1 2^21 + s2 2^42 for x in [0, 2^63).
ERP_FXP_FN void fxp_split3(float x, uint32_t &s0, uint32_t &s1, uint32_t &s2) {
    const float r = fxp_high_part(x, 1.0f / 4398046511104.0f, 4398046511104.0f, s2);
    fxp_split2<21>(r, s0, s1);
}

// (float)q, round half to even, for any q < 2^64.  The top set bit goes to bit 31
// of a 32-bit word whose bit 0 also stands for everything below it; that word's
// own conversion (a native 32-bit one) then rounds as the 64-bit value would, and
// the power of two is exact.  About 12 instructions, without a branch; the row pass
// converts every bin (its earlier form, which rounded the mantissa itself, took
// about 30).
ERP_FXP_FN float fxp_u64_to_float(uint64_t q) {
    const uint32_t hi = (uint32_t)(q >> 32), lo = (uint32_t)q;
    const int lz = hi ? fxp_clz32(hi) : 0;
#if defined(__CUDA_ARCH__)
    const uint32_t top = __funnelshift_l(lo, hi, lz);
#else
    const uint32_t top = (uint32_t)((q << lz) >> 32);
#endif
    const uint32_t word = hi ? top | ((lo << lz) ? 1u : 0u) : lo;
    const float scale = hi ? fxp_bits_float((uint32_t)(159 - lz) << 23) : 1.0f;   // 2^(32 - lz)
#if defined(__CUDA_ARCH__)
    return __fmul_rn(__uint2float_rn(word), scale);
#else
    return (float)word * scale;
#endif
}

}  // namespace erp

#undef ERP_FXP_FN
