// greeks64.cu -- the sensitivities of greeks.cu in FP64 accuracy: five states
// per path (base, spot +/- h, vol +/- h) evaluated literally on the same draws,
// in the fixed-point arithmetic of the FP64 pricer (paths64.cuh).  Units,
// sums and merge are the pricer's, so the price output is its price bit for bit.
//
// The spot states share the base's log-path (their spots differ by a factor),
// the vol states carry their own.  Estimators as in greeks.cu: finite
// differences (src/greeks/finite_difference.cpp:40-65), likelihood ratio
// (src/greeks/likelihood_ratio.cpp:33-73, :105-154), pathwise
// (src/greeks/pathwise.cpp:28-55, :64-147).  Sums that the reference takes per
// step follow from integer sums: W_i, the running sum of the draws, is one of its
// own (the log-spot's differs from it by vol sqrt(dt), and would have lost as many
// of its bits as that is small), the log-spots' derivatives are sqrt(dt) W_i - vol
// i dt, and sum i S_i follows from the prefix sums of S_i.
//
// Bound: issue and the FMA-heavy pipe for barriers, lookbacks and geometric
// Asians; the FP64 pipe for arithmetic Asians (five operations per step).  1024
// threads per CTA (64 registers): the twelve outputs' sums are then spilled
// between the rounds of a unit, but a call of 1e5 paths (3125 units) is one
// round of the 4864 resident warps, where 512 threads and 128 registers took
// two.  Measured: finite-difference European, likelihood-ratio barrier and
// pathwise Asian of 1e5 paths and 52 dates, one call each, 130 -> 0.40 ms in all
// (512, 640, 768, 1024 threads: 0.48, 0.48, 0.42, 0.41 before the units' sums
// lost their division); 16 contracts of 2e5 paths, Asian 3.09 -> 2.91 ms, barrier
// 1.91 -> 1.65, lookback 1.66 -> 1.61, European 0.81; largest error against
// 64-bit values 4.7e-13 -> 2.2e-14.
//
// nvcc-flags: --fmad=false
#include <cuda_runtime.h>

#include "engine.hpp"
#include "greeks.hpp"
#include "paths64.cuh"

namespace mcdg {

namespace {

constexpr int kThreads = 1024;

__device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; }

// Likelihood-ratio and pathwise estimators common to both path arithmetics,
// from the base state's numbers; v holds the five undiscounted payoffs.
struct BaseState {
    double z1, z_sum, zz_excess;             // first draw, sum of draws, sum of (z^2 - 1)
    double last, avg;                        // S_n and the average (Asians)
    double avg_dvol, avg_drate;              // derivatives of the average
    double last_dvol;                        // dS_n / dvol
};

__device__ __forceinline__ void estimators(const DevContract& c, const DevGreeks& g, const double (&v)[5],
                                           const BaseState& b, double (&o)[kNumGreeks]) {
    const double disc = c.discount, h = disc * v[0];
    o[kGPrice] = h;
    o[kGFdDelta] = disc * ((v[1] - v[2]) * g.inv_2hs);
    o[kGFdGamma] = disc * ((v[1] - 2.0 * v[0] + v[2]) * g.inv_hs2);
    o[kGFdVega] = disc * ((v[3] - v[4]) * g.inv_2hv);
    o[kGLrDelta] = h * (b.z1 * g.lr_delta_scale);
    o[kGLrGamma] = h * ((b.z1 * b.z1 - g.vol * g.sqrt_dt * b.z1 - 1.0) * g.lr_gamma_scale);
    o[kGLrVega] = h * (b.zz_excess * g.inv_vol - g.sqrt_dt * b.z_sum);
    o[kGLrRho] = h * (g.sqrt_dt_over_vol * b.z_sum - g.time);
    o[kGLrTheta] = o[kGPwDelta] = o[kGPwVega] = o[kGPwRho] = 0.0;
    const double phi = c.type == 0 ? 1.0 : -1.0;
    if (c.kind == kEuropean || c.kind == kDigital)
        o[kGLrTheta] = h * (g.rate - (b.zz_excess * g.inv_2t + g.mu_over_vol_sqrt_t * b.z1));
    if (c.kind == kEuropean) {
        const double slope = disc * (phi * (b.last - c.strike) > 0.0 ? phi : 0.0);
        o[kGPwDelta] = slope * (b.last * g.inv_spot);
        o[kGPwVega] = slope * (b.last * (g.sqrt_dt * b.z1 - g.vol * g.time));
        o[kGPwRho] = slope * (b.last * g.time) - g.time * h;
    } else if (c.kind == kAsianArith || c.kind == kAsianGeo) {
        const double ref = c.floating ? b.last - b.avg : b.avg - c.strike;
        const double slope = disc * (phi * ref > 0.0 ? phi : 0.0);
        const double nt = static_cast<double>(c.n_steps) * g.dt;
        const double s0 = c.floating ? b.last - b.avg : b.avg;
        o[kGPwDelta] = slope * (s0 * g.inv_spot);
        o[kGPwVega] = slope * (c.floating ? b.last_dvol - b.avg_dvol : b.avg_dvol);
        o[kGPwRho] = slope * (c.floating ? b.last * nt - b.avg_drate : b.avg_drate) - g.time * h;
    }
}

// ---------------------------------------------------------------------------
// Contracts outside the fixed-point range (DevGreeks::wide): the five states step
// by step in FP64.
// ---------------------------------------------------------------------------
__device__ __noinline__ void greeks_wide(const DevContract& c, const DevGreeks& g, uint64_t path,
                                         double (&o)[kNumGreeks]) {
    const PhiloxKeys k = philox_keys(c.seed);
    const PhiloxPath pp = philox_path(path, 0u, k);
    const double phi = c.type == 0 ? 1.0 : -1.0, n = static_cast<double>(c.n_steps);
    double s[5] = {c.spot, c.spot + g.h_spot, c.spot - g.h_spot, c.spot, c.spot}, v[5];
    double sum[5] = {}, lsum[5] = {}, hi[5], lo[5];
    bool hit[5] = {};
    for (int j = 0; j < 5; ++j) hi[j] = lo[j] = s[j];
    BaseState b{};
    double s_dvol = 0.0, l_dvol = 0.0, s_drate = 0.0, l_drate = 0.0;
    for (int step = 0; step < c.n_steps; ++step) {
        const double z = normal_from_bits_f64(philox_word0(pp, static_cast<uint32_t>(step), k));
        if (step == 0) b.z1 = z;
        b.z_sum += z;
        b.zz_excess += z * z - 1.0;
        const double m[3] = {exp(c.drift + c.vs * z), exp(g.drift_up + g.vs_up * z), exp(g.drift_dn + g.vs_dn * z)};
        for (int j = 0; j < 5; ++j) {
            s[j] = s[j] * m[j < 3 ? 0 : j - 2];
            sum[j] += s[j];
            lsum[j] += log(s[j]);
            hit[j] = hit[j] || (c.up ? s[j] >= c.barrier : s[j] <= c.barrier);
            hi[j] = dmax(hi[j], s[j]);
            lo[j] = s[j] < lo[j] ? s[j] : lo[j];
        }
        const double i = static_cast<double>(step + 1), d = g.sqrt_dt * b.z_sum - g.vol * i * g.dt;
        s_dvol += s[0] * d;
        l_dvol += d;
        s_drate += s[0] * (i * g.dt);
        l_drate += i * g.dt;
        b.last_dvol = s[0] * d;
    }
    for (int j = 0; j < 5; ++j) {
        const double avg = c.kind == kAsianGeo ? exp(lsum[j] / n) : sum[j] / n;
        if (j == 0) b.avg = avg;
        const double vanilla = dmax(phi * (s[j] - c.strike), 0.0);
        switch (c.kind) {
            case kEuropean: v[j] = vanilla; break;
            case kDigital: v[j] = phi * (s[j] - c.strike) > 0.0 ? (c.asset ? s[j] : c.cash) : 0.0; break;
            case kAsianArith:
            case kAsianGeo: v[j] = dmax(phi * (c.floating ? s[j] - avg : avg - c.strike), 0.0); break;
            case kBarrier: v[j] = (c.out ? !hit[j] : hit[j]) ? vanilla : c.rebate; break;
            case kLookbackFixed: v[j] = c.type == 0 ? dmax(hi[j] - c.strike, 0.0) : dmax(c.strike - lo[j], 0.0); break;
            default: v[j] = c.type == 0 ? s[j] - lo[j] : hi[j] - s[j]; break;
        }
    }
    b.last = s[0];
    b.avg_dvol = c.kind == kAsianGeo ? b.avg * (l_dvol / n) : s_dvol / n;
    b.avg_drate = c.kind == kAsianGeo ? b.avg * (l_drate / n) : s_drate / n;
    estimators(c, g, v, b, o);
}

// ---------------------------------------------------------------------------
// fixed point
// ---------------------------------------------------------------------------
struct GreeksSlot {
    WarpSlot w;
    DevGreeks g;
};

// A path's state beyond the pricer's: the barrier keeps its extreme instead of
// the flag, which then answers for every spot state.
template <int KIND>
struct State : Path64<KIND> {
    int64_t extreme = 0;
    __device__ __forceinline__ void advance(const DevContract& c, const FixedShared& s, int64_t dy, bool first) {
        if constexpr (KIND == kBarrier) {
            this->y += dy;
            extreme = first ? this->y : (c.up ? max(extreme, this->y) : min(extreme, this->y));
        } else {
            this->step(c, s, dy, 0u);
        }
    }
    __device__ __forceinline__ double payoff(const DevContract& c, double spot, int64_t barrier, const FixedShared& s) {
        if constexpr (KIND == kBarrier) this->breached = c.up ? extreme >= barrier : extreme <= barrier;
        return payoff64<KIND>(c, spot, s, *this);
    }
};

template <int KIND>
__device__ __forceinline__ void greeks_fixed(GreeksSlot& slot, const FixedShared& s, const FixedTables* __restrict__ t,
                                             const PhiloxKeys& k, uint32_t path_lo, uint32_t path_hi, bool refill,
                                             double (&o)[kNumGreeks]) {
    const DevContract& c = slot.w.c;
    const DevGreeks& g = slot.g;
    const int lane = threadIdx.x & 31;
    const int n = (KIND == kEuropean || KIND == kDigital) ? 1 : c.n_steps;
    const PhiloxRow row = philox_row(path_lo, 0u, k);
    State<KIND> p, up, dn;
    uint64_t zz_lo = 0, zz_hi = 0;  // sum of z^2, units of 2^-58, split at 32 bits
    int64_t w = 0;                   // W_i, units of 2^(z_shift - 61)
    int64_t wsum_hi = 0;             // geometric Asian: sum of W_i, as Path64's of y
    uint64_t wsum_lo = 0;
    double prefix = 0.0, e_w = 0.0;  // arithmetic Asian: sum of the running sums, sum of S_i / S0 times W_i
    FixedNormal z1{};
    for (int d0 = 0; d0 < n; d0 += 32) {
        if (refill || n > 32) {
            __syncwarp();
            const uint32_t d = static_cast<uint32_t>(d0 + lane);
            PhiloxStep st = philox_step(d, path_hi, k);
            st.carry = drift_carry(d, c.y_drift_lo) | drift_carry(d, g.y_drift_lo_up) << 1 |
                       drift_carry(d, g.y_drift_lo_dn) << 2;
            slot.w.step[lane] = st;
            __syncwarp();
        }
        const int m = min(32, n - d0);
        for (int d = 0; d < m; ++d) {
            const PhiloxStep st = slot.w.step[d];
            const FixedNormal z = normal_fixed(philox_word0(row, st, k), s, t);
            const bool first = d0 + d == 0;
            if (first) z1 = z;
            p.advance(c, s, c.y_drift + (st.carry & 1u) + scaled_normal(z, c.y_vs), first);
            up.advance(c, s, g.y_drift_up + (st.carry >> 1 & 1u) + scaled_normal(z, g.y_vs_up), first);
            dn.advance(c, s, g.y_drift_dn + (st.carry >> 2) + scaled_normal(z, g.y_vs_dn), first);
            const uint64_t zz = mul_hi64(z.mag, z.mag);
            zz_lo += static_cast<uint32_t>(zz);
            zz_hi += zz >> 32;
            if constexpr (KIND != kEuropean && KIND != kDigital) {
                const int64_t neg = z.neg;
                w += (static_cast<int64_t>(z.mag >> g.z_shift) ^ neg) - neg;
            }
            if constexpr (KIND == kAsianArith) {
                prefix += p.sum;
                e_w = fma(p.last, static_cast<double>(w), e_w);
            }
            if constexpr (KIND == kAsianGeo) {
                wsum_hi += w >> 32;
                wsum_lo += static_cast<uint32_t>(w);
            }
        }
    }
    const double nd = static_cast<double>(n);
    const double v[5] = {p.payoff(c, c.spot, c.y_barrier, s), p.payoff(c, c.spot + g.h_spot, g.y_barrier_su, s),
                         p.payoff(c, c.spot - g.h_spot, g.y_barrier_sd, s), up.payoff(c, c.spot, c.y_barrier, s),
                         dn.payoff(c, c.spot, c.y_barrier, s)};
    BaseState b{};
    b.z1 = normal_to_double(z1);
    b.last = c.spot * exp2_units(p.y, c.frac, s);
    if constexpr (KIND == kEuropean || KIND == kDigital) {
        b.z_sum = b.z1;
        b.zz_excess = b.z1 * b.z1 - 1.0;
    } else {
        b.z_sum = static_cast<double>(w) * g.z_unit;
        b.zz_excess = fma(fma(static_cast<double>(zz_hi), 4294967296.0, static_cast<double>(zz_lo)), 0x1p-58, -nd);
    }
    if constexpr (KIND == kAsianArith || KIND == kAsianGeo) {
        b.avg = average64<KIND>(c, c.spot, s, p);
        const double decay = g.vol * g.dt;  // dlnS_i/dvol = sqrt(dt) W_i - i decay
        b.last_dvol = b.last * fma(g.sqrt_dt, b.z_sum, -nd * decay);
        if constexpr (KIND == kAsianArith) {
            const double i_s = fma(nd + 1.0, p.sum, -prefix);  // sum of i S_i / S0
            b.avg_dvol = c.spot * (fma(g.sqrt_dt, e_w * g.z_unit, -i_s * decay) * c.inv_n);
            b.avg_drate = c.spot * (i_s * g.dt * c.inv_n);
        } else {
            const double i_mean = 0.5 * (nd + 1.0);
            const double w_mean = fma(static_cast<double>(wsum_hi), 4294967296.0, static_cast<double>(wsum_lo)) *
                                  (g.z_unit * c.inv_n);
            b.avg_dvol = b.avg * fma(g.sqrt_dt, w_mean, -i_mean * decay);
            b.avg_drate = b.avg * (i_mean * g.dt);
        }
    }
    estimators(c, g, v, b, o);
    // A floating-strike payoff is the spot times a number that does not depend
    // on it: its central differences are that number and zero, without the
    // rounding of three prices divided by h^2.
    if constexpr (KIND == kAsianArith || KIND == kAsianGeo || KIND == kLookbackFloating) {
        if (KIND == kLookbackFloating || c.floating) {
            o[kGFdDelta] = c.discount * p.payoff(c, 1.0, c.y_barrier, s);
            o[kGFdGamma] = 0.0;
        }
    }
}

// The pricer's sample where its contract is in the fixed-point range but a bumped
// state is not.
template <int KIND>
__device__ __forceinline__ double price_sample(const DevContract& c, const FixedShared& s,
                                               const FixedTables* __restrict__ t, uint64_t path) {
    const PhiloxKeys k = philox_keys(c.seed);
    const PhiloxRow row = philox_row(static_cast<uint32_t>(path), 0u, k);
    const uint32_t n = KIND == kEuropean || KIND == kDigital ? 1u : static_cast<uint32_t>(c.n_steps);
    Path64<KIND> p;
    for (uint32_t d = 0; d < n; ++d) {
        const uint32_t bits = philox_word0(row, philox_step(d, static_cast<uint32_t>(path >> 32), k), k);
        p.step(c, s, c.y_drift + drift_carry(d, c.y_drift_lo) + scaled_normal(normal_fixed(bits, s, t), c.y_vs), 0u);
    }
    return c.discount * payoff64<KIND>(c, c.spot, s, p);
}
__device__ __noinline__ double price_fixed(const DevContract& c, const FixedShared& s,
                                           const FixedTables* __restrict__ t, uint64_t path) {
    switch (c.kind) {
        case kEuropean: return price_sample<kEuropean>(c, s, t, path);
        case kDigital: return price_sample<kDigital>(c, s, t, path);
        case kAsianArith: return price_sample<kAsianArith>(c, s, t, path);
        case kAsianGeo: return price_sample<kAsianGeo>(c, s, t, path);
        case kBarrier: return price_sample<kBarrier>(c, s, t, path);
        case kLookbackFixed: return price_sample<kLookbackFixed>(c, s, t, path);
        default: return price_sample<kLookbackFloating>(c, s, t, path);
    }
}

struct SharedGreeks {
    FixedShared tables;
    GreeksSlot slot[kThreads / 32];
};

__global__ void __launch_bounds__(kThreads, 1)
    greeks64_kernel(const DevContract* __restrict__ contracts, const DevGreeks* __restrict__ greeks, int n_contracts,
                    const uint32_t* __restrict__ prefix, uint32_t* __restrict__ ticket, Welford* __restrict__ partials,
                    uint32_t* __restrict__ error_flag, const FixedTables* __restrict__ t) {
    extern __shared__ __align__(16) unsigned char smem[];
    SharedGreeks& sh = *reinterpret_cast<SharedGreeks*>(smem);
    load_fixed_tables(sh.tables, t);
    const FixedShared& s = sh.tables;
    const int lane = threadIdx.x & 31;
    GreeksSlot& slot = sh.slot[threadIdx.x >> 5];
    const uint32_t first = prefix[0];
    int have = -1;
    uint32_t lo_item = 0, hi_item = 0;
    for (ItemSource src(prefix[n_contracts] - first); src.valid(); src.next(ticket)) {
        const uint32_t item = src.item;
        if (have < 0 || item - lo_item >= hi_item - lo_item) {
            have = find_contract(prefix, n_contracts, item);
            lo_item = prefix[have] - first;
            hi_item = prefix[have + 1] - first;
            __syncwarp();
            copy_words(&slot.w.c, &contracts[have]);
            copy_words(&slot.g, &greeks[have]);
            __syncwarp();
        }
        const DevContract& c = slot.w.c;
        const uint64_t base = static_cast<uint64_t>(item - lo_item) << (5 + c.unit_log);
        if (base >= c.path_count) {  // planning invariant broken: record, skip the item
            if (lane == 0) atomicOr(error_flag, 1u);
            continue;
        }
        const uint64_t left = c.path_count - base;
        const uint32_t size = 32u << c.unit_log;
        const uint32_t count = left < size ? static_cast<uint32_t>(left) : size;
        const int rounds = static_cast<int>((count + 31u) / 32u);
        const PhiloxKeys k = philox_keys(c.seed);
        double pivot[kNumGreeks], s1[kNumGreeks], s2[kNumGreeks], o[kNumGreeks];
        for (int j = 0; j < rounds; ++j) {
            const uint32_t at = static_cast<uint32_t>(j) * 32u + lane;
            const uint32_t path_lo = static_cast<uint32_t>(base) + at, path_hi = static_cast<uint32_t>(base >> 32);
#define MCD_GREEKS(K) case K: greeks_fixed<K>(slot, s, t, k, path_lo, path_hi, j == 0, o); break;
            if (slot.g.wide) {
                greeks_wide(c, slot.g, base + at, o);
                if (c.frac != 0) o[kGPrice] = price_fixed(c, s, t, base + at);
            } else {
                switch (c.kind) {
                    MCD_GREEKS(kEuropean)
                    MCD_GREEKS(kDigital)
                    MCD_GREEKS(kAsianArith)
                    MCD_GREEKS(kAsianGeo)
                    MCD_GREEKS(kBarrier)
                    MCD_GREEKS(kLookbackFixed)
                    default: MCD_GREEKS(kLookbackFloating)
                }
            }
#undef MCD_GREEKS
#pragma unroll
            for (int i = 0; i < kNumGreeks; ++i) {  // as UnitSums
                if (j == 0) {
                    pivot[i] = __shfl_sync(0xffffffffu, o[i], 0);
                    s1[i] = s2[i] = 0.0;
                }
                if (at < count) {
                    const double d = o[i] - pivot[i];
                    s1[i] += d;
                    s2[i] = fma(d, d, s2[i]);
                }
            }
        }
        int index;
        const double a = warp_sums(s1, lane, index);
        const double b = warp_sums(s2, lane, index);
        double p = 0.0;
#pragma unroll
        for (int i = 0; i < kNumGreeks; ++i) p = index == i ? pivot[i] : p;
        if (index < kNumGreeks)
            partials[static_cast<size_t>(item) * kNumGreeks + index] =
                unit_triple(count, p, a, b);
    }
}

}  // namespace

cudaError_t launch_greeks64_kernel(int grid, const DevContract* contracts, const DevGreeks* greeks, int n_contracts,
                                   const uint32_t* item_prefix, uint32_t* ticket, Welford* partials,
                                   uint32_t* error_flag, const FixedTables* tables, cudaStream_t stream) {
    constexpr int bytes = static_cast<int>(sizeof(SharedGreeks));
    cudaError_t e = cudaFuncSetAttribute(greeks64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    cudaGetLastError();
    greeks64_kernel<<<grid, kThreads, bytes, stream>>>(contracts, greeks, n_contracts, item_prefix, ticket, partials,
                                                       error_flag, tables);
    return cudaGetLastError();
}

}  // namespace mcdg
