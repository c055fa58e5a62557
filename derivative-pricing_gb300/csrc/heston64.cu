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
// Square roots, the reciprocal and the logarithm are integer operations on the
// doubles' significands (fixed_root.hpp), and psi / 2, the two roots of the
// quadratic branch and b + z are 64-bit fractions: 1 - sqrt(1 - psi / 2) keeps
// 60 fraction bits where the regrouped FP64 form needs a second reciprocal.  Of
// the log-spot only sum(v) and sum(z sqrt(v + v')) are carried along the path:
// K1 and K2 act on sum(v) and on the end points, and K3 = K4 leaves the root's
// factor out of the loop.  Eight FP64 operations per step remain (E[v'], psi,
// the product of the new variance, the two sums).
//
// Bound: issue and the multiply pipe, about 400 instructions per step.  One call
// of 1e5 paths and 252 steps: 410-441 ms for the reference's form in items of
// 4096 paths, 2.7 to 5.2 ms (the longer the more often psi > 1.5) with 46 or
// more FP64 operations per step, which held the FP64 pipe at 83 %, 0.65 to 1.1 ms
// in integers.  24 warps per SM (80 registers): 16 warps 0.79, 32 warps 0.65.
//
// nvcc-flags: --fmad=false
#include <cuda_runtime.h>

#include "fixed_root.hpp"
#include "fp64_fast.cuh"
#include "heston.hpp"
#include "merge.cuh"
#include "paths64.cuh"

namespace mcdg {

namespace {

constexpr int kThreads = 768;
constexpr int kStrikesPerLane = kHestonMaxStrikes / 32;

struct HestonSlot {
    HestonSet set;
    PhiloxStep step[32];
    double terminal[32];
};
struct HestonTables : QuantTables {
    uint64_t log_l[kLogEntries];
    uint32_t log_c[kLogEntries];
};
struct Shared {
    HestonTables tables;
    HestonSlot slot[kThreads / 32];
};

// Steps outside the integer forms' range (E[v'] beyond 2^+-100, psi below 2^-13,
// where 1 - sqrt(1 - psi / 2) has too few bits, or above 2^60), in FP64.
__device__ __noinline__ double variance_step_wide(double m, double qe_a, double qe_b, uint32_t ubits, double z) {
    const double r = fast_rcp64(m);
    const double psi = r * fma(-qe_a, r, qe_b);
    if (psi <= 1.5) {
        const double g = 0.5 * psi;
        const double s = fast_sqrt64(1.0 - g);
        if (psi < 0x1p-13) {
            // With t = 1 - s, (sqrt(s) + z sqrt(t))^2 - 1 = 2 z sqrt(s t) + t (z^2 - 1).  The
            // square itself, rounded next to 1 in the same way at every step, adds up:
            // at xi = 0.0013, 252 steps and rho / xi = 223, 4e-13 in ln S against 2e-14.
            const double t = g * fast_rcp64(1.0 + s);
            return fma(m, fma(z + z, fast_sqrt64(s * t), t * fma(z, z, -1.0)), m);
        }
        const double w = fma(z, fast_sqrt64(g * fast_rcp64(1.0 + s)), fast_sqrt64(s));
        return m * (w * w);
    }
    const double q = psi + 1.0;
    if (uniform_open01_f64(ubits) * q <= psi - 1.0) return 0.0;
    // 1 - u = (~bits + 1/2) / 2^32, exact
    return positive_part(-0.5 * (m * q) * log(0.5 * q * uniform_open01_f64(~ubits)));
}

__device__ __forceinline__ double variance_step(double v, const HestonSet& h, uint32_t ubits, const HestonTables& s,
                                                const FixedTables* __restrict__ t) {
    const double m = fma(v, h.e, h.reversion);
    constexpr uint32_t kLow = (1023u - 100u) << 20, kSpan = 200u << 20;
    const bool m_ok = static_cast<uint32_t>(__double2hiint(m)) - kLow < kSpan;
    const double r = m_ok ? rcp_int(m) : 1.0;
    const double psi = r * fma(-h.qe_a, r, h.qe_b);
    const uint32_t psi_hi = static_cast<uint32_t>(__double2hiint(psi));
    if (!m_ok || psi_hi - ((1023u - 13u) << 20) >= (73u << 20))
        return variance_step_wide(m, h.qe_a, h.qe_b, ubits, normal_to_double(normal_fixed(ubits, s, t)));
    const uint64_t pb = bits_of(psi);
    if (pb <= 0x3FF8000000000000ull) {  // psi <= 1.5
        const FixedNormal z = normal_fixed(ubits, s, t);
        const uint64_t g = significand(pb) >> (1023 - static_cast<int>(psi_hi >> 20));  // psi / 2, units of 2^-64
        const uint64_t root = sqrt_frac(0u - g);                                        // sqrt(1 - psi / 2)
        const uint64_t rest = 0u - root;
        const int half = __clz(static_cast<int>(rest >> 32)) >> 1;
        const uint64_t b = sqrt_frac(rest << (2 * half)) >> half;  // sqrt(1 - root)
        const uint64_t zb = mul_hi64(z.mag, b), a = sqrt_frac(root) >> 3;  // units of 2^-61
        const int64_t w = static_cast<int64_t>(z.neg ? a - zb : a + zb);
        const double d = scaled_double(static_cast<uint64_t>(w < 0 ? -w : w) | 1u, 2);
        return m * (d * d);
    }
    // y = (1 + psi) / 2 (1 - u), 1 - u = (~bits + 1/2) / 2^32: zero from y = 1 on
    const double q = psi + 1.0;
    const uint64_t qb = bits_of(q);
    const uint32_t nb = ~ubits;
    const int lz = __clz(static_cast<int>(nb));
    uint64_t y = mul_hi64(significand(qb), ((static_cast<uint64_t>(nb) << 32) | 0x80000000u) << lz);
    int e = lz + 1 - exponent_of(qb);
    if (static_cast<int64_t>(y) >= 0) {
        y <<= 1;
        ++e;
    }
    if (e <= 0) return 0.0;
    const uint32_t i = log_index(y);
    const uint64_t l = neg_log(y, e, s.log_c[i], s.log_l[i]);
    return 0.5 * (m * q) * scaled_double(l | 1u, 4);
}

// ln(S_T / S_0) of one path.
__device__ __forceinline__ double log_return(HestonSlot& slot, const HestonTables& s,
                                             const FixedTables* __restrict__ t, const PhiloxKeys& k, uint32_t path_lo,
                                             uint32_t path_hi) {
    const HestonSet& h = slot.set;
    const int lane = threadIdx.x & 31;
    const PhiloxRow spot = philox_row(path_lo, 0u, k), variance = philox_row(path_lo, 1u, k);
    double v = h.v0, sum = 0.0, x = 0.0;
    for (int d0 = 0; d0 < h.n_steps; d0 += 32) {
        __syncwarp();
        slot.step[lane] = philox_step(static_cast<uint32_t>(d0 + lane), path_hi, k);
        __syncwarp();
        const int n = min(32, h.n_steps - d0);
        for (int d = 0; d < n; ++d) {
            const PhiloxStep st = slot.step[d];
            const double next = variance_step(v, h, philox_word0(variance, st, k), s, t);
            const double both = v + next;
            const uint32_t hi = static_cast<uint32_t>(__double2hiint(both));
            // zero (both variances are), subnormal or beyond FP64's range: the library's
            const double root = hi - 0x00100000u < 0x7FE00000u ? sqrt_int(both) : sqrt(both);
            x = fma(root, normal_to_double(normal_fixed(philox_word0(spot, st, k), s, t)), x);
            sum += v;
            v = next;
        }
    }
    return fma(h.root_k3, x, fma(h.k2, v - h.v0, fma(h.k12, sum, h.drift_sum)));
}

__global__ void __launch_bounds__(kThreads, 1)
    heston64_kernel(const HestonSet* __restrict__ sets, const double* __restrict__ strikes, int n_strikes, int type,
                    uint32_t units_per_set, uint32_t total_items, int unit_log, uint32_t* __restrict__ ticket,
                    Welford* __restrict__ partials, const FixedTables* __restrict__ t) {
    extern __shared__ __align__(16) unsigned char smem[];
    Shared& sh = *reinterpret_cast<Shared*>(smem);
    copy_quantile(sh.tables, t);
    copy_table(sh.tables.log_l, t->log_l, sizeof sh.tables.log_l);
    copy_table(sh.tables.log_c, t->log_c, sizeof sh.tables.log_c);
    wait_tables();
    const HestonTables& s = sh.tables;
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
