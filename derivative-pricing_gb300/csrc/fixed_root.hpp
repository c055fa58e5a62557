// fixed_root.hpp -- reciprocal, square root and logarithm in 64-bit integers
// from an FP32 seed (host and device), for kernels whose FP64 pipe is the
// bottleneck: an FP64 operation holds a scheduler for 64 cycles on this GPU, a
// 32x32->64-bit integer product for 4.3, so a square root of 6 FP64 operations
// (384 cycles) takes about a quarter of that as 6 products and 20 additions and
// shifts.  Errors: 2^-59.4 relative at worst, against 2^-53 for
// a rounded double.
#pragma once

#include "fixed_math.hpp"

#ifndef __CUDA_ARCH__
#include <cmath>
#include <cstring>
#endif

namespace mcdg {

MCD_HD int32_t mul_hi_signed(int32_t a, int32_t b) {
#ifdef __CUDA_ARCH__
    return __mulhi(a, b);
#else
    return static_cast<int32_t>((static_cast<int64_t>(a) * b) >> 32);
#endif
}
MCD_HD uint64_t wide(uint32_t a, uint32_t b) { return static_cast<uint64_t>(a) * b; }
MCD_HD int count_lz64(uint64_t x) {
#ifdef __CUDA_ARCH__
    return __clzll(static_cast<long long>(x));
#else
    return __builtin_clzll(x);
#endif
}
MCD_HD uint64_t bits_of(double x) {
#ifdef __CUDA_ARCH__
    return static_cast<uint64_t>(__double_as_longlong(x));
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}
MCD_HD double double_of(uint64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double(static_cast<long long>(b));
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}
// Significand of a normal double, units of 2^-63 (in [2^63, 2^64)).
MCD_HD uint64_t significand(uint64_t bits) { return (bits << 11) | (1ull << 63); }
MCD_HD int exponent_of(uint64_t bits) { return static_cast<int>(bits >> 52) - 1023; }  // sign bit clear

// m 2^(e - 63) as a double for any m != 0.
MCD_HD double scaled_double(uint64_t m, int e) {
    const int lz = count_lz64(m);
    return double_of(double_bits(m << lz, e - lz));
}

// 1 / sqrt(a 2^-32), a in [2^30, 2^32), as 2 integer and 30 fraction bits, within
// 2^-21: the scaled float is added to 4, which leaves its bits in place.
MCD_HD uint32_t rsqrt_seed(uint32_t a) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint2float_rn(a)));
    return __float_as_uint(__fmaf_rn(r, 65536.0f, 4.0f)) * 512u - (0x40800000u * 512u);
#else
    const float v = std::fma(1.0f / std::sqrt(static_cast<float>(a)), 65536.0f, 4.0f);
    uint32_t b;
    std::memcpy(&b, &v, 4);
    return b * 512u - (0x40800000u * 512u);
#endif
}
// 1 / (a 2^-31), a in [2^31, 2^32), the same format, within 2^-22.
MCD_HD uint32_t rcp_seed(uint32_t a) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint2float_rn(a)));
    return __float_as_uint(__fmaf_rn(r, 2147483648.0f, 2.0f)) * 256u - (0x40000000u * 256u);
#else
    const float v = std::fma(1.0f / static_cast<float>(a), 2147483648.0f, 2.0f);
    uint32_t b;
    std::memcpy(&b, &v, 4);
    return b * 256u - (0x40000000u * 256u);
#endif
}

// sqrt(a) of a 64-bit fraction a in [1/4, 1) from y = 1/sqrt(a) (seed).
// h: a y less a bias of 2^-20 (so that the residual is positive), 32 bits;
// c: the first Newton term (units of 2^-49); d: the residual after both (2^-96,
// exact modulo 2^64, magnitude below 2^59); its term ends the root.
MCD_HD uint64_t sqrt_from_seed(uint64_t a, uint32_t y) {
    const uint32_t h = (mul_hi32(static_cast<uint32_t>(a >> 32), y) << 2) - 4096u;
    const uint64_t r1 = a - wide(h, h);
    const uint32_t c = mul_hi32(static_cast<uint32_t>(r1 >> 14), y);
    const int64_t d = static_cast<int64_t>((r1 << 32) - (wide(h, c) << 16) - (wide(c, c) >> 2));
    const int32_t k = mul_hi_signed(static_cast<int32_t>(d >> 28), static_cast<int32_t>(y >> 1)) >> 2;
    return (static_cast<uint64_t>(h) << 32) + (static_cast<uint64_t>(c) << 15) +
           static_cast<uint64_t>(static_cast<int64_t>(k));
}
MCD_HD uint64_t sqrt_frac(uint64_t a) { return sqrt_from_seed(a, rsqrt_seed(static_cast<uint32_t>(a >> 32))); }

// 1/m of a significand (units of 2^-63, in (2^62, 2^63)), y its seed: with
// e = 1 - m y, y (1 + e + e^2).
MCD_HD uint64_t rcp_from_seed(uint64_t m, uint32_t y) {
    const uint64_t q = (wide(static_cast<uint32_t>(m >> 32), y) << 3) + (wide(static_cast<uint32_t>(m), y) >> 29);
    const int64_t e = -static_cast<int64_t>(q);  // units of 2^-64
    const int32_t eh = static_cast<int32_t>(e >> 14);
    const int64_t t = e + (mul_hi_signed(eh, eh) >> 4);
    const int64_t yt = static_cast<int64_t>(static_cast<int32_t>(y)) * static_cast<int32_t>(t >> 32);
    const uint64_t r = (static_cast<uint64_t>(y) << 33) + (static_cast<uint64_t>(yt) << 1) +
                       (wide(y, static_cast<uint32_t>(t)) >> 31);
    return r < (1ull << 63) ? r : (1ull << 63) - 1;
}

// x > 0, normal.
MCD_HD double sqrt_int(double x) {
    const uint64_t b = bits_of(x);
    const uint64_t a = significand(b) >> (static_cast<uint32_t>(b >> 52) & 1u);
    return double_of(double_bits(sqrt_frac(a), exponent_of(b) >> 1));
}
// x > 0, normal with a normal reciprocal.
MCD_HD double rcp_int(double x) {
    const uint64_t b = bits_of(x), m = significand(b);
    const uint64_t r = rcp_from_seed(m, rcp_seed(static_cast<uint32_t>(m >> 32)));
    return double_of(double_bits(r << 1, -exponent_of(b) - 1));
}

// -ln(m 2^(-63 - e)), m in [2^63, 2^64), e in [1, 40], in units of 2^-59: with
// the table's c just above 1 / (the interval's left end), m c = 1 + t, 0 <= t <
// 2^-10 + 2^-30, and ln m = -ln c + t - t^2/2 + t^3 (1/3 - t (1/4 - t/5)).
MCD_HD uint32_t log_index(uint64_t m) { return static_cast<uint32_t>(m >> (63 - kLogBits)) & (kLogEntries - 1); }
MCD_HD uint64_t neg_log(uint64_t m, int e, uint32_t c, uint64_t neg_log_c) {
    constexpr uint64_t ln2 = 399572145162582989ull;  // units of 2^-59
    const uint64_t t = ((wide(static_cast<uint32_t>(m >> 32), c) - (1ull << 62)) << 2) +
                       (wide(static_cast<uint32_t>(m), c) >> 30);  // units of 2^-64
    const uint64_t t2 = mul_hi64(t << 9, t << 9);                   // units of 2^-82
    const uint32_t th = static_cast<uint32_t>(t >> 23);             // units of 2^-41
    const uint32_t q = (1u << 31) - mul_hi32(th, 3355443u);         // 1/4 - t/5, units of 2^-33
    const uint32_t r = 2863311531u - (mul_hi32(th, q) >> 9);        // 1/3 - ..., units of 2^-33
    const uint32_t t3 = mul_hi32(static_cast<uint32_t>(t2 >> 32), th);  // units of 2^-59
    const uint64_t log_1t = (t >> 5) - (t2 >> 24) + (mul_hi32(t3, r) >> 1);
    const uint64_t l = static_cast<uint64_t>(e) * ln2 - neg_log_c - log_1t;  // below 2^63.9
    return static_cast<uint32_t>(l >> 32) == 0xFFFFFFFFu ? 0 : l;            // a few units below zero
}

}  // namespace mcdg
