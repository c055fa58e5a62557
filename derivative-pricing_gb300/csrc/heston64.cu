// heston64.cu -- Heston QE paths in FP64, priced against many strikes.
//
// Reference: heston_qe_european (src/pricers/heston.cpp:91-156), as heston.cu.
// Algebra.  With m = E[v'], psi = Var[v'] / m^2 and h = sqrt(1 - psi / 2), the
// quadratic branch's constants are b^2 = h / (1 - h) and a = m (1 - h), so
//     v' = a (b + z)^2 = m (sqrt(h) + z sqrt(1 - h))^2,  1 - h = (psi/2) / (1 + h),
// and, Var[v'] being linear in m, psi = r B (1 - r C / 2) with r = 1/m,
// B = xi^2 (1 - e) / kappa and C = theta (1 - e): one reciprocal where the
// reference divides three times.  The exponential branch is
// v' = -(m (1 + psi) / 2) ln((1 + psi)(1 - u) / 2), zero where u (1 + psi) <= psi - 1.
//
// Work: one warp per unit of 32 r paths (r a power of two fixed by the path
// count), the normals from the fixed-point quantile (fixed_path.cuh).  A path
// lives in one lane; its terminal spot is paid out against one strike in that
// lane, or, for several strikes, through shared memory with a strike per lane.
//
// Bound: the FP64 pipe, about 45 operations per step (the reference's form takes
// about 500, most of them in its two inverse normals).  One call of 1e5 paths and
// 252 steps: 410-441 ms (items of 4096 paths, 25 of 152 SMs) -> 2.7 to 5.2 ms,
// the longer the more often psi > 1.5; error against 64-bit values 1.5e-12 ->
// 1.2e-12.
//
// nvcc-flags: --fmad=false
#include <cuda_runtime.h>

#include "fp64_fast.cuh"
#include "heston.hpp"
#include "merge.cuh"
#include "paths64.cuh"

namespace mcdg {

namespace {

constexpr int kThreads = 512;
constexpr int kStrikesPerLane = kHestonMaxStrikes / 32;

struct HestonSlot {
    HestonSet set;
    PhiloxStep step[32];
    double terminal[32];
};
struct Shared {
    FixedShared tables;
    HestonSlot slot[kThreads / 32];
};

__device__ __forceinline__ double variance_step(double v, const HestonSet& h, uint32_t ubits, double z) {
    const double m = fma(v - h.theta, h.e, h.theta);
    const double r = fast_rcp64(m);
    const double psi = r * fma(-h.qe_a, r, h.qe_b);
    if (psi <= 1.5) {
        const double g = 0.5 * psi;
        const double s = fast_sqrt64(1.0 - g);
        const double w = fma(z, fast_sqrt64(g * fast_rcp64(1.0 + s)), fast_sqrt64(s));
        return m * (w * w);
    }
    const double q = psi + 1.0;
    if (uniform_open01_f64(ubits) * q <= psi - 1.0) return 0.0;
    // 1 - u = (~bits + 1/2) / 2^32, exact
    return positive_part(-0.5 * (m * q) * log(0.5 * q * uniform_open01_f64(~ubits)));
}

// ln(S_T / S_0) of one path.
__device__ __forceinline__ double log_return(HestonSlot& slot, const FixedShared& s, const FixedTables* __restrict__ t,
                                             const PhiloxKeys& k, uint32_t path_lo, uint32_t path_hi) {
    const HestonSet& h = slot.set;
    const int lane = threadIdx.x & 31;
    const PhiloxRow spot = philox_row(path_lo, 0u, k), variance = philox_row(path_lo, 1u, k);
    double v = h.v0, x = 0.0;
    for (int d0 = 0; d0 < h.n_steps; d0 += 32) {
        __syncwarp();
        slot.step[lane] = philox_step(static_cast<uint32_t>(d0 + lane), path_hi, k);
        __syncwarp();
        const int n = min(32, h.n_steps - d0);
        for (int d = 0; d < n; ++d) {
            const PhiloxStep st = slot.step[d];
            const double zs = normal_to_double(normal_fixed(philox_word0(spot, st, k), s, t));
            const uint32_t ubits = philox_word0(variance, st, k);
            const double zv = normal_to_double(normal_fixed(ubits, s, t));
            const double next = variance_step(v, h, ubits, zv);
            const double var = h.k3 * v + h.k4 * next;
            const double vol = var > 0.0 ? fast_sqrt64(var) : 0.0;
            x += fma(h.k1, v, fma(h.k2, next, fma(vol, zs, h.drift_k0)));
            v = next;
        }
    }
    return x;
}

__global__ void __launch_bounds__(kThreads, 1)
    heston64_kernel(const HestonSet* __restrict__ sets, const double* __restrict__ strikes, int n_strikes, int type,
                    uint32_t units_per_set, uint32_t total_items, int unit_log, uint32_t* __restrict__ ticket,
                    Welford* __restrict__ partials, const FixedTables* __restrict__ t) {
    extern __shared__ __align__(16) unsigned char smem[];
    Shared& sh = *reinterpret_cast<Shared*>(smem);
    load_fixed_tables(sh.tables, t);
    const FixedShared& s = sh.tables;
    const int lane = threadIdx.x & 31;
    HestonSlot& slot = sh.slot[threadIdx.x >> 5];
    uint32_t have = 0xFFFFFFFFu;
    for (ItemSource src(total_items); src.valid(); src.next(ticket)) {
        const uint32_t item = src.item, set = item / units_per_set;
        if (set != have) {
            have = set;
            __syncwarp();
            copy_words(&slot.set, &sets[set]);
            __syncwarp();
        }
        const HestonSet& h = slot.set;
        const uint64_t base = static_cast<uint64_t>(item % units_per_set) << (5 + unit_log);
        const uint64_t left = h.path_count - base;
        const uint32_t size = 32u << unit_log;
        const uint32_t count = left < size ? static_cast<uint32_t>(left) : size;
        const PhiloxKeys k = philox_keys(h.seed);
        UnitSums acc[kStrikesPerLane];
        auto payoff = [&](double spot, double strike) {
            return h.discount * positive_part(put_sign(spot - strike, type));
        };
        for (uint32_t o = 0; o < count; o += 32) {
            const uint32_t path_lo = static_cast<uint32_t>(base) + o + lane;
            const double spot = exp(h.log_s0 + log_return(slot, s, t, k, path_lo, static_cast<uint32_t>(base >> 32)));
            if (n_strikes == 1) {
                const double v = payoff(spot, strikes[0]);
                if (o == 0) acc[0].first(v);
                if (o + lane < count) acc[0].add(v);
                continue;
            }
            __syncwarp();
            slot.terminal[lane] = spot;
            __syncwarp();
            const int live = static_cast<int>(min(32u, count - o));
#pragma unroll
            for (int i = 0; i < kStrikesPerLane; ++i) {
                const int at = lane + 32 * i;
                if (at >= n_strikes) break;
                const double strike = strikes[at];
                if (o == 0) acc[i].pivot = payoff(slot.terminal[0], strike);
                for (int p = 0; p < live; ++p) acc[i].add(payoff(slot.terminal[p], strike));
            }
        }
        Welford* out = partials + static_cast<size_t>(item) * n_strikes;
        if (n_strikes == 1) {
            const Welford w = acc[0].reduce(count);
            if (lane == 0) out[0] = w;
        } else {
#pragma unroll
            for (int i = 0; i < kStrikesPerLane; ++i)
                if (lane + 32 * i < n_strikes) out[lane + 32 * i] = unit_triple(count, acc[i].pivot, acc[i].s1, acc[i].s2);
        }
    }
}

}  // namespace

cudaError_t launch_heston64(int grid, const HestonSet* sets, int n_sets, const double* strikes, int n_strikes,
                            int type, uint32_t units_per_set, int unit_log, uint32_t* ticket, Welford* partials,
                            const FixedTables* tables, cudaStream_t stream) {
    constexpr int bytes = static_cast<int>(sizeof(Shared));
    cudaError_t e = cudaFuncSetAttribute(heston64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    cudaGetLastError();
    heston64_kernel<<<grid, kThreads, bytes, stream>>>(sets, strikes, n_strikes, type, units_per_set,
                                                       units_per_set * static_cast<uint32_t>(n_sets), unit_log, ticket,
                                                       partials, tables);
    return cudaGetLastError();
}

}  // namespace mcdg
