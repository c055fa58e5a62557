// paths64.cuh -- FP64 GBM paths of one contract: the per-path state in 64-bit
// fixed point, its step, and the payoff.  Shared by the pricer (gbm_paths64.cu)
// and the sensitivities (greeks64.cu), whose price output is the pricer's bit
// for bit.
//
// The reference multiplies the spot by exp(drift + vs z) per step
// (src/models/gbm.cpp:7-12).  Here y = log2(S / S0) is a sum of integers in
// units of 2^-F: no rounding accumulates over the steps, a barrier or a running
// extreme needs no exponential, and the geometric mean no logarithm.  Only the
// arithmetic average takes 2^y at every step (and one FP64 addition).
#pragma once

#include "engine.hpp"
#include "fixed_path.cuh"
#include "unit_sums.cuh"

namespace mcdg {

// A warp's contract and the Philox words of its next 32 steps.
struct WarpSlot {
    DevContract c;
    PhiloxStep step[32];
};

template <int KIND>
struct Path64 {
    int64_t y = 0;                // log2(S / S0), units of 2^-F
    int64_t hi = 0, lo = 0;       // running extremes of y (from the start value 0)
    int64_t lsum_hi = 0;          // sum of y as (sum of its high words, sum of its low words)
    uint64_t lsum_lo = 0;
    double sum = 0.0, last = 1.0; // sum of S / S0 and its last term (arithmetic averages)
    bool breached = false;

    // dy: this step's log2 increment; u: the bridge uniform's bits (kBarrierBridge)
    __device__ __forceinline__ void step(const DevContract& c, const FixedShared& s, int64_t dy, uint32_t ubits) {
        const int64_t y0 = y;
        y += dy;
        if constexpr (KIND == kAsianArith || KIND == kAsianCv) {
            last = exp2_units(y, c.frac, s);
            sum += last;
        }
        if constexpr (KIND == kAsianGeo || KIND == kAsianCv) add_log(y);
        if constexpr (KIND == kBarrier || KIND == kBarrierBridge)
            breached = breached || (c.up ? y >= c.y_barrier : y <= c.y_barrier);
        if constexpr (KIND == kBarrierBridge) {
            // crossing between the dates with probability
            // exp(-2 ln(H/S) ln(H/S') / (vol^2 dt)) (monte_carlo.cpp:184-230):
            // ln u against the exponent in FP32, in FP64 only where the two
            // are too close to tell
            if (!breached) {
                const int64_t d0 = c.y_barrier - y0, d1 = c.y_barrier - y;
                const float a = static_cast<float>(c.y_bridge) * static_cast<float>(d0) * static_cast<float>(d1);
                const float lu = __logf(uniform_from_bits_f32(ubits));
                if (fabsf(a - lu) > 1e-4f + 1e-5f * fabsf(a)) {
                    breached = lu < a;
                } else {
                    const double e = c.y_bridge * static_cast<double>(d0) * static_cast<double>(d1);
                    breached = uniform_open01_f64(ubits) < exp(e);
                }
            }
        }
        if constexpr (KIND == kLookbackFixed || KIND == kLookbackFloating) {
            hi = max(hi, y);
            lo = min(lo, y);
        }
    }

    __device__ __forceinline__ void add_log(int64_t v) {
        lsum_hi += v >> 32;
        lsum_lo += static_cast<uint32_t>(v);
    }
    __device__ __forceinline__ double log_sum() const {  // sum of y in units
        return fma(static_cast<double>(lsum_hi), 4294967296.0, static_cast<double>(lsum_lo));
    }
};

// (x < 0) ? 0 : x by the high word: from 0x80000000 (-0) to 0xFFF00000 (-infinity);
// a NaN above that stays, as in the comparison's form.
__device__ __forceinline__ double positive_part(double x) {
    return static_cast<uint32_t>(__double2hiint(x)) - 0x80000000u <= 0x7FF00000u ? 0.0 : x;
}
__device__ __forceinline__ double put_sign(double x, int type) { return type == 0 ? x : -x; }

// The average that an Asian pays on, from spot (or a bumped spot).
template <int KIND>
__device__ __forceinline__ double average64(const DevContract& c, double spot, const FixedShared& s,
                                            const Path64<KIND>& p) {
    if constexpr (KIND == kAsianGeo) return spot * exp2_units(__double2ll_rn(p.log_sum() * c.inv_n), c.frac, s);
    return spot * (p.sum * c.inv_n);
}

// The undiscounted payoff.
template <int KIND>
__device__ __forceinline__ double payoff64(const DevContract& c, double spot, const FixedShared& s,
                                           const Path64<KIND>& p) {
    if constexpr (KIND == kAsianArith || KIND == kAsianGeo) {
        const double avg = average64<KIND>(c, spot, s, p);
        const double x = c.floating ? spot * exp2_units(p.y, c.frac, s) - avg : avg - c.strike;
        return positive_part(put_sign(x, c.type));
    } else if constexpr (KIND == kLookbackFixed) {
        const double x = spot * exp2_units(c.type == 0 ? p.hi : p.lo, c.frac, s);
        return positive_part(put_sign(x - c.strike, c.type));
    } else {
        const double last = spot * exp2_units(p.y, c.frac, s);
        if constexpr (KIND == kLookbackFloating) {
            const double x = spot * exp2_units(c.type == 0 ? p.lo : p.hi, c.frac, s);
            return c.type == 0 ? last - x : x - last;
        }
        const double v = put_sign(last - c.strike, c.type);
        if constexpr (KIND == kDigital) return v > 0.0 ? (c.asset ? last : c.cash) : 0.0;
        if constexpr (KIND == kBarrier || KIND == kBarrierBridge) {
            const bool pays = c.out ? !p.breached : p.breached;
            return pays ? positive_part(v) : c.rebate;
        }
        return positive_part(v);
    }
}

// The control-variate Asian's sample; the anchor is discounted, so this one is too.
__device__ __forceinline__ double control_variate64(const DevContract& c, const FixedShared& s,
                                                    const Path64<kAsianCv>& p) {
    const double a = c.spot * (p.sum * c.inv_n);
    const double g = c.spot * exp2_units(__double2ll_rn(p.log_sum() * c.inv_n), c.frac, s);
    const double ap = c.discount * positive_part(put_sign(a - c.strike, c.type));
    const double gp = c.discount * positive_part(put_sign(g - c.strike, c.type));
    return ap - (gp - c.kv_anchor);
}

// The contract that holds an item: the largest index whose first item is <=
// item (empty contracts share their successor's first item and are skipped).
__device__ __forceinline__ int find_contract(const uint32_t* __restrict__ prefix, int n_contracts, uint32_t item) {
    int lo = 0, hi = n_contracts;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (prefix[mid] - prefix[0] <= item) lo = mid; else hi = mid;
    }
    return lo;
}

// A warp's copy of one record in 8-byte words.
template <class T>
__device__ __forceinline__ void copy_words(T* to, const T* from) {
    static_assert(sizeof(T) % 8 == 0, "records are copied in 8-byte words");
    for (int i = threadIdx.x & 31; i < static_cast<int>(sizeof(T) / 8); i += 32)
        reinterpret_cast<uint64_t*>(to)[i] = reinterpret_cast<const uint64_t*>(from)[i];
}

// The item that a warp works on next: the first round is dealt over the CTAs
// (a small batch then uses every SM), later items come from the ticket, a few
// at a time while many are left.
struct ItemSource {
    uint32_t item, left, total, dealt;
    __device__ __forceinline__ ItemSource(uint32_t total_items) {
        const uint32_t warps = blockDim.x >> 5;
        total = total_items;
        dealt = gridDim.x * warps;
        item = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
        left = 1;
    }
    __device__ __forceinline__ bool valid() const { return item < total; }
    __device__ __forceinline__ void next(uint32_t* ticket) {
        if (--left > 0) {
            ++item;
            return;
        }
        const uint32_t grab = total / dealt >= 64u ? 4u : 1u;
        uint32_t t = 0;
        if ((threadIdx.x & 31) == 0) t = atomicAdd(ticket, grab);
        t = __shfl_sync(0xffffffffu, t, 0);
        item = dealt + t;
        left = grab;
        if (item < total && left > total - item) left = total - item;
    }
};

}  // namespace mcdg
