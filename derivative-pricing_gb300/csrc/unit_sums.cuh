// unit_sums.cuh -- a warp's samples as shifted sums: with d = sample - pivot, the
// pivot being the warp's first sample, the variance of a unit does not cancel,
// and three FP64 operations per sample (one division per unit) replace the
// reference's Welford update and its division (include/mcd/core/stats.hpp:29-36).
// FP64 operations are the scarce resource on this GPU.
#pragma once

#include <cuda_runtime.h>

#include "device_common.cuh"
#include "engine.hpp"

namespace mcdg {

// a = sum of d, b = sum of d^2 as a Welford triple.
__device__ __forceinline__ Welford unit_triple(uint32_t count, double pivot, double a, double b) {
    if (count == 0) return Welford{0ull, 0.0, 0.0};
    // every full unit has a power of two of samples: an exact product instead of
    // the division's 640 cycles
    const bool pow2 = (count & (count - 1u)) == 0u;
    const double inv = __hiloint2double((1023 - (31 - __clz(static_cast<int>(count)))) << 20, 0);
    const double m = pow2 ? a * inv : a / static_cast<double>(count);
    const double m2 = fma(-a, m, b);
    return Welford{count, pivot + m, m2 < 0.0 ? 0.0 : m2};  // (NaN stays)
}

// The triples of a CTA's four warps.  Whole items have a power of two of samples
// in every warp: the mean of the means and one term of the between-warps
// variance each, 18 FP64 operations; a chain of three Welford merges takes
// about 120 (three divisions), by one thread while its CTA waits.
__device__ __forceinline__ Welford merge_warps(const Welford& a, const Welford& b, const Welford& c, const Welford& d) {
    if (a.count != b.count || a.count != c.count || a.count != d.count || a.count == 0)
        return welford_merge(welford_merge(a, b), welford_merge(c, d));
    const double mean = 0.25 * ((a.mean + b.mean) + (c.mean + d.mean));
    const double da = a.mean - mean, db = b.mean - mean, dc = c.mean - mean, dd = d.mean - mean;
    const double between = fma(da, da, fma(db, db, fma(dc, dc, dd * dd)));
    return Welford{4 * a.count, mean,
                   fma(static_cast<double>(static_cast<uint32_t>(a.count)), between, (a.m2 + b.m2) + (c.m2 + d.m2))};
}

// One output.  first() once, by all lanes, with lane 0's sample valid (or no
// sample in the warp at all); reduce() by all lanes, valid in lane 0.
struct UnitSums {
    double pivot = 0.0, s1 = 0.0, s2 = 0.0;
    __device__ __forceinline__ void first(double v) { pivot = __shfl_sync(0xffffffffu, v, 0); }
    __device__ __forceinline__ void add(double v) {
        const double d = v - pivot;
        s1 += d;
        s2 = fma(d, d, s2);
    }
    __device__ __forceinline__ Welford reduce(uint32_t count) const {
        // the lower half-warp adds up s1, the upper one s2
        const bool high = threadIdx.x & 16;
        double a = (high ? s2 : s1) + __shfl_xor_sync(0xffffffffu, high ? s1 : s2, 16);
#pragma unroll
        for (int off = 8; off >= 1; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
        const double b = __shfl_xor_sync(0xffffffffu, a, 16);
        return unit_triple(count, pivot, a, b);  // lane 0: (s1, s2)
    }
};

// Sums v[i] over the warp for every i < 12 at once: each step halves the
// values a lane carries while it doubles the lanes they stand for (14 additions
// instead of 60); the additions of one value pair the same lanes as a shuffle
// tree's.  Returns the sum of output `index` (12 or more: none).
__device__ __forceinline__ double warp_sums(const double (&v)[12], int lane, int& index) {
    double a6[6], a3[3], a2[2];
    const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4, h2 = lane & 2;
#pragma unroll
    for (int i = 0; i < 6; ++i)
        a6[i] = (h16 ? v[i + 6] : v[i]) + __shfl_xor_sync(0xffffffffu, h16 ? v[i] : v[i + 6], 16);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        a3[i] = (h8 ? a6[i + 3] : a6[i]) + __shfl_xor_sync(0xffffffffu, h8 ? a6[i] : a6[i + 3], 8);
    // three values: lanes without bit 2 keep the first two, the others the third
    a2[0] = (h4 ? a3[2] : a3[0]) + __shfl_xor_sync(0xffffffffu, h4 ? a3[0] : a3[2], 4);
    const double other = __shfl_xor_sync(0xffffffffu, a3[1], 4);
    a2[1] = a3[1] + other;
    const double a1 = (h2 ? a2[1] : a2[0]) + __shfl_xor_sync(0xffffffffu, h2 ? a2[0] : a2[1], 2);
    index = (h16 ? 6 : 0) + (h8 ? 3 : 0) + (h4 ? 2 : 0) + (h2 ? 1 : 0);
    if ((h4 && h2) || (lane & 1)) index = 12;  // a duplicate or the other half of a pair
    return a1 + __shfl_xor_sync(0xffffffffu, a1, 1);
}

}  // namespace mcdg
