// merge.cuh -- the fold of a contract's item partials, shared by the pricer's
// and the sensitivities' merge kernels (whose prices agree bit for bit).
#pragma once

#include "engine.hpp"

namespace mcdg {

// A single contract of 1e5 paths has 3125 items, 25 per thread: four loads in
// flight and a short last tree take a call's merge from 16 to 9 us (cold); 256 or
// 512 threads measured the same.  The last division and root are IEEE's (0.3 us
// of a quote's 27 against ones from an FP32 seed, which err by up to a unit).
constexpr int kMergeThreads = 128;

struct MergedResult {
    double mean, standard_error;
    unsigned long long count;
};

// The first kMergeThreads threads of a CTA fold the Welford triples
// items[i * stride], i < count (every thread calls; read past the L1): thread t takes t, t + kMergeThreads, ... in order, as sums shifted by the
// first item's mean (four FP64 operations per item and no division: a chain of
// Welford merges takes about forty), then a fixed tree.  Valid in thread 0.
__device__ __forceinline__ MergedResult merge_items(const Welford* __restrict__ items, uint32_t count, int stride) {
    __shared__ double s_sum[2][kMergeThreads / 32];
    __shared__ unsigned long long s_count[kMergeThreads / 32];
    static_assert(sizeof(Welford) == 24 && offsetof(Welford, mean) == 8 && offsetof(Welford, m2) == 16, "three words");
    auto load = [&](uint32_t i) {
        const double* p = reinterpret_cast<const double*>(items + static_cast<size_t>(i) * stride);
        return Welford{static_cast<unsigned long long>(__double_as_longlong(__ldcg(p))), __ldcg(p + 1), __ldcg(p + 2)};
    };
    const double shift = count ? load(0).mean : 0.0;
    unsigned long long n = 0;
    double s1 = 0.0, s2 = 0.0;
    constexpr int kAhead = 4;
    for (uint32_t i0 = threadIdx.x; threadIdx.x < kMergeThreads && i0 < count; i0 += kAhead * kMergeThreads) {
        Welford w[kAhead];
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
            const uint32_t i = i0 + j * kMergeThreads;
            if (i < count) w[j] = load(i);
        }
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
            if (i0 + j * kMergeThreads >= count) break;
            const double d = w[j].mean - shift, nd = static_cast<double>(w[j].count) * d;
            n += w[j].count;
            s1 += nd;
            s2 += fma(nd, d, w[j].m2);
        }
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        n += __shfl_down_sync(0xffffffffu, n, off);
        s1 += __shfl_down_sync(0xffffffffu, s1, off);
        s2 += __shfl_down_sync(0xffffffffu, s2, off);
    }
    if ((threadIdx.x & 31) == 0 && threadIdx.x < kMergeThreads) {
        s_count[threadIdx.x >> 5] = n;
        s_sum[0][threadIdx.x >> 5] = s1;
        s_sum[1][threadIdx.x >> 5] = s2;
    }
    __syncthreads();
    MergedResult r{0.0, 0.0, 0ull};
    if (threadIdx.x >= 32) return r;
    constexpr int kWarps = kMergeThreads / 32;
    const int w = threadIdx.x & (kWarps - 1);
    n = s_count[w];
    s1 = s_sum[0][w];
    s2 = s_sum[1][w];
#pragma unroll
    for (int off = kWarps / 2; off >= 1; off >>= 1) {
        n += __shfl_down_sync(0xffffffffu, n, off);
        s1 += __shfl_down_sync(0xffffffffu, s1, off);
        s2 += __shfl_down_sync(0xffffffffu, s2, off);
    }
    if (threadIdx.x != 0) return r;
    r.count = n;
    if (n > 0) {
        const double nd = static_cast<double>(n);
        const double mean = s1 / nd;
        const double m2 = fma(-s1, mean, s2);
        r.mean = shift + mean;
        if (n > 1 && !(m2 <= 0.0)) r.standard_error = sqrt(m2 / ((nd - 1.0) * nd));
    }
    return r;
}

}  // namespace mcdg
