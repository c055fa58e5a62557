// fp64_fast.cuh -- FP64 reciprocal and square root from an FP32 seed and one
// cubic iteration: three and five FP64 operations, against nine or more of the
// library's routines, on a GPU whose FP64 operations cost 68 FP32 ones each.
// The seed (MUFU, error below 2^-22) cubed is below 2^-64, so the results are
// within one unit in the last place.  The seed's conversions are integer
// operations on the bit patterns.
#pragma once

#include "device_common.cuh"

namespace mcdg {

// x > 0 in (2^-126, 2^127), truncated to FP32, and back.
__device__ __forceinline__ float seed_of(double x) {
    const uint32_t hi = static_cast<uint32_t>(__double2hiint(x)), lo = static_cast<uint32_t>(__double2loint(x));
    return __uint_as_float(__funnelshift_l(lo, hi, 3) - (384u << 23));
}
__device__ __forceinline__ double seed_wide(float y) {
    const uint32_t b = __float_as_uint(y);
    return __hiloint2double(static_cast<int>((b >> 3) + (896u << 20)), static_cast<int>(b << 29));
}
// Within the seed's range with room for the products below.
__device__ __forceinline__ bool seed_range(double x) {
    const int e = __double2hiint(x);
    return e > ((1023 - 100) << 20) && e < ((1023 + 100) << 20);  // 2^-100 < x < 2^100 (false for negative and NaN)
}

__device__ __forceinline__ double fast_rcp64(double x) {
    if (!seed_range(x)) return 1.0 / x;
    const double y = seed_wide(fast_rcp(seed_of(x)));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

__device__ __forceinline__ double fast_sqrt64(double x) {
    if (!seed_range(x)) return sqrt(x);
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(seed_of(x)));
    const double y = seed_wide(r);
    const double s = x * y;
    const double e = fma(-s, y, 1.0);
    return fma(s * e, fma(0.375, e, 0.5), s);
}

}  // namespace mcdg
