// lsm_math.cuh -- FP64 arithmetic shared by the Longstaff-Schwartz kernels: the
// stored path values, the basis and the continuation value.  Kernels that
// regenerate path values or replay decisions use these, so they agree with the
// backward pass bit for bit.
#pragma once

#include "fixed_path.cuh"
#include "lsm.hpp"

namespace mcdg {

// Fixed-point tables read through the L1 cache: kernels that draw too little
// for a copy in shared memory, or whose shared memory is taken.
struct GlobalTables {
    const FixedTables* __restrict__ t;
    __device__ __forceinline__ FixedNormal normal(uint32_t bits) const {
        const int32_t upper = static_cast<int32_t>(bits) >> 31;
        const QuantArg a = quant_arg(2u * (bits ^ static_cast<uint32_t>(upper)) + 1u);
        const ulonglong2 l = __ldg(reinterpret_cast<const ulonglong2*>(&t->lo[a.entry]));
        const ulonglong2 h = __ldg(reinterpret_cast<const ulonglong2*>(&t->hi[a.entry]));
        const QuantLo lo{l.x, l.y};
        const QuantHi hi{h.x, static_cast<uint32_t>(h.y), static_cast<uint32_t>(h.y >> 32)};
        return FixedNormal{quant_eval(lo, hi, a.s), ~upper};
    }
    // 2^(f / 2^64) 2^e
    __device__ __forceinline__ double exp2_parts(uint64_t f, int e) const {
        const uint64_t m = exp2_frac(f, __ldg(&t->exp_a[exp2_index_a(f)]), __ldg(&t->exp_b[exp2_index_b(f)]));
        return __longlong_as_double(static_cast<long long>(double_bits(m, e)));
    }
    __device__ __forceinline__ double exp2(int64_t y, int frac) const {
        return exp2_parts(static_cast<uint64_t>(y) << (64 - frac), static_cast<int>(y >> frac));
    }
};

// One date of an FP64 path: y is log2(S / S0) in the contract's units
// (LsmDev::frac > 0), else the reference's product (gbm.cpp:7-12).
struct LsmState64 {
    int64_t y = 0;
    double s;
    __device__ __forceinline__ explicit LsmState64(const LsmDev& c) : s(c.spot) {}
    __device__ __forceinline__ void advance(const LsmDev& c, uint32_t bits, uint32_t d, const GlobalTables& t) {
        if (c.frac > 0) {
            y += c.y_drift + drift_carry(d, c.y_drift_lo) + scaled_normal(t.normal(bits), c.y_vs);
            s = c.spot * t.exp2(y, c.frac);
        } else {
            s = s * exp(c.drift + c.vs * normal_from_bits_f64(bits));
        }
    }
};

// S on the paying side of K, by the order of positive doubles' bit patterns.
__device__ __forceinline__ bool in_the_money64(double s, double strike, int type) {
    const long long a = __double_as_longlong(s), b = __double_as_longlong(strike);
    return type == 0 ? a > b : a < b;
}

// e^{-x/2}, x = S/K >= 0: 2^y of y = -x / (2 ln 2) split into integer and
// fraction by integer operations on the double's bits, instead of the library's
// exponential (some fifteen FP64 operations; this takes one).
__device__ __forceinline__ double exp_half_neg(double x, const GlobalTables& t) {
    const double v = x * 0.72134752044448170368;  // 1 / (2 ln 2)
    const uint64_t b = static_cast<uint64_t>(__double_as_longlong(v));
    const int e = static_cast<int>(b >> 52) - 1023;
    if (e >= 9 || e < -60) return e < -60 ? 1.0 : exp(-0.5 * x);  // beyond 2^9 (or NaN), or nothing
    const uint64_t m = (b & 0xFFFFFFFFFFFFFull) | 1ull << 52;
    // v = whole + f / 2^64: the significand m 2^(e - 52) around the binary point
    const uint64_t f = e >= -12 ? m << (12 + e) : m >> (-12 - e);
    const int whole = e >= 0 ? static_cast<int>(m >> (52 - e)) : 0;
    // -v = -(whole + 1) + (2^64 - f) / 2^64
    return f == 0 ? t.exp2_parts(0, -whole) : t.exp2_parts(0ull - f, -whole - 1);
}

// Weighted Laguerre basis on x = S/K (src/pricers/lsm.cpp:21-25).
__device__ __forceinline__ void basis64(double s, double inv_strike, const GlobalTables& t, double (&b)[4]) {
    const double x = s * inv_strike;
    const double e = exp_half_neg(x, t);
    b[0] = e;
    b[1] = fma(-e, x, e);
    b[2] = e * fma(fma(0.5, x, -2.0), x, 1.0);
    b[3] = e * fma(fma(fma(-1.0 / 6.0, x, 1.5), x, -3.0), x, 1.0);
}

// The fitted combination in monomials of x (LsmReg::poly).
__device__ __forceinline__ double continuation64(double s, double inv_strike, const double (&p)[4],
                                                 const GlobalTables& t) {
    const double x = s * inv_strike;
    return exp_half_neg(x, t) * fma(fma(fma(p[3], x, p[2]), x, p[1]), x, p[0]);
}

}  // namespace mcdg
