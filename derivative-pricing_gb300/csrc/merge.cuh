// merge.cuh -- the fold of a contract's item partials, shared by the pricer's
// and the sensitivities' merge kernels (whose prices agree bit for bit).
#pragma once

#include "engine.hpp"

namespace mcdg {

constexpr int kMergeThreads = 128;

struct MergedResult {
    double mean, standard_error;
    unsigned long long count;
};

// One CTA of kMergeThreads folds the Welford triples items[i * stride],
// i < count: thread t takes t, t + 128, ... in order, as sums shifted by the
// first item's mean (four FP64 operations per item and no division: a chain of
// Welford merges takes about forty), then a fixed tree.  Valid in thread 0.
__device__ __forceinline__ MergedResult merge_items(const Welford* __restrict__ items, uint32_t count, int stride) {
    __shared__ double s_sum[2][kMergeThreads / 32];
    __shared__ unsigned long long s_count[kMergeThreads / 32];
    const double shift = count ? items[0].mean : 0.0;
    unsigned long long n = 0;
    double s1 = 0.0, s2 = 0.0;
    for (uint32_t i = threadIdx.x; i < count; i += kMergeThreads) {
        const Welford w = items[static_cast<size_t>(i) * stride];
        const double d = w.mean - shift, nd = static_cast<double>(w.count) * d;
        n += w.count;
        s1 += nd;
        s2 += fma(nd, d, w.m2);
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        n += __shfl_down_sync(0xffffffffu, n, off);
        s1 += __shfl_down_sync(0xffffffffu, s1, off);
        s2 += __shfl_down_sync(0xffffffffu, s2, off);
    }
    if ((threadIdx.x & 31) == 0) {
        s_count[threadIdx.x >> 5] = n;
        s_sum[0][threadIdx.x >> 5] = s1;
        s_sum[1][threadIdx.x >> 5] = s2;
    }
    __syncthreads();
    MergedResult r{0.0, 0.0, 0ull};
    if (threadIdx.x != 0) return r;
    for (int w = 1; w < kMergeThreads / 32; ++w) {
        n += s_count[w];
        s1 += s_sum[0][w];
        s2 += s_sum[1][w];
    }
    r.count = n;
    if (n > 0) {
        const double mean = s1 / static_cast<double>(n);
        const double m2 = fma(-s1, mean, s2);
        r.mean = shift + mean;
        if (n > 1)
            r.standard_error = sqrt((m2 < 0.0 ? 0.0 : m2) / (static_cast<double>(n - 1) * static_cast<double>(n)));
    }
    return r;
}

}  // namespace mcdg
