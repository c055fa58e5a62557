// items.hpp -- into what a contract's paths are cut: slabs of 4096 (Sobol, FP32
// Heston), FP64 units, FP32 items.  By the contract alone, so that its result
// depends neither on the launch nor on the rest of the batch.
#pragma once

#include <cstdint>

namespace mcdg {

// FP64 units of 32 << unit_log paths: one path per lane up to 131,071 paths (a
// single call then has the most warps to spread over the GPU), doubling from there
// so that a contract keeps 2048 to 4096 units, up to a slab.
constexpr int unit_log(uint64_t paths) {
    int log = 0;
    while (log < 7 && (paths >> (17 + log)) != 0) ++log;
    return log;
}
constexpr uint64_t unit_count(uint64_t paths) {
    const uint64_t size = 32ull << unit_log(paths);
    return (paths + size - 1) / size;
}

// FP32 items of 128 << item_log paths: a CTA's 4096 paths, halved while the contract
// has at most 256 items of the half and those still hold 131,072 path-steps.  A
// small book's time is that of its longest item (4096 paths of 252 dates: 1.9 ms in
// a CTA by itself); contracts of more than 2^19 paths keep whole slabs.  Books of
// 3, 10, 30, 100, 300, 1000, 4096 contracts of 1e3 to 3e5 paths, ms, whole slabs
// against items: priced 1.11, 1.18, 1.78, 2.47, 4.35, 11.7, 54.4 and 0.72, 0.50,
// 0.85, 1.46, 4.12, 11.8, 54.7; sensitivities 2.72, 2.85, 3.34, 4.35, 7.75, 20.8,
// 93.4 and 1.60, 1.07, 1.52, 2.44, 7.43, 20.4, 91.6.
constexpr uint64_t kMaxCutItems = 256;
constexpr int item_log(uint64_t paths, int steps) {
    int log = 5;
    while (log > 1) {
        const uint64_t half = 64ull << log;
        if (paths > kMaxCutItems * half || half * static_cast<uint64_t>(steps) < 131072) break;
        --log;
    }
    return log;
}
constexpr uint64_t item_count(uint64_t paths, int steps) {
    const uint64_t size = 128ull << item_log(paths, steps);
    return (paths + size - 1) / size;
}

}  // namespace mcdg
