// gbm_paths64.cu -- the batched GBM path engine in FP64 accuracy: one
// persistent kernel for every product, paths in 64-bit fixed point
// (paths64.cuh, fixed_math.hpp).
//
// Work.  A contract's paths are cut into units of 32 r paths, r a power of two
// that depends on the contract's path count alone (convert_contract): one warp
// prices one unit, lane l taking paths l, l + 32, ...  A call with few paths
// therefore spreads over all SMs (10,000 paths: 313 warps), and a unit's result
// does not depend on the grid or on the rest of the batch.
//
// Bound: issue slots and the FMA-heavy pipe (integer multiplies); a path-step
// of a barrier takes 13 wide products for Philox, 6 for the quantile and 3 for
// the log-spot, and one gather of 32 bytes per lane from the quantile table in
// shared memory.  One CTA per SM shares that table among 32 warps.
//
// Measured on one GB300 against the reference's operations in FP64 (about 200
// FP64 operations per path-step, slabs of 4096 paths as items): a
// control-variate antithetic Asian of 1e5 paths and 252 dates 842-1035 ms ->
// 0.31 ms per call, a European of 1e4 paths 0.55 -> 0.026 ms, a mixed book of
// 64 contracts (1e4 to 3e5 paths, 12 to 252 dates) 750-990 -> 3.3-3.9 ms; error
// of the book's prices against 64-bit values 5.9e-16 -> 2.7e-16 relative.
//
// nvcc-flags: --fmad=false
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "engine.hpp"
#include "fixed_tables.hpp"
#include "lsm_math.cuh"
#include "merge.cuh"
#include "paths64.cuh"

namespace mcdg {

namespace {

__device__ FixedTables g_fixed_tables;

constexpr int kQuoteThreads = 128, kQuoteCtas = 6;

// ---------------------------------------------------------------------------
// Contracts whose log-spot does not fit the fixed-point range (|log2(S/S0)|
// could reach 2^9 on some path): the reference's arithmetic step by step.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double dmin(double a, double b) { return (b < a) ? b : a; }

__device__ __noinline__ double payoff_wide(const DevContract& c, uint64_t path, bool neg) {
    const PhiloxKeys k = philox_keys(c.seed);
    const double phi = c.type == 0 ? 1.0 : -1.0;
    const PhiloxPath pp = philox_path(path, 0u, k), pu = philox_path(path, 1u, k);
    double s = c.spot, sum = 0.0, log_sum = 0.0, rmax = c.spot, rmin = c.spot;
    bool breached = false;
    for (int step = 0; step < c.n_steps; ++step) {
        const uint32_t d = static_cast<uint32_t>(step);
        double z = normal_from_bits_f64(philox_word0(pp, d, k));
        if (neg) z = -z;
        const double s_next = s * exp(c.drift + c.vs * z);
        breached = breached || (c.up ? s_next >= c.barrier : s_next <= c.barrier);
        if (c.kind == kBarrierBridge && !breached) {
            const double p = exp(-2.0 * (c.log_barrier - log(s)) * (c.log_barrier - log(s_next)) / c.bb_denom);
            breached = uniform_open01_f64(philox_word0(pu, d, k)) < p;
        }
        s = s_next;
        if (c.kind == kAsianArith || c.kind == kAsianCv) sum += s;
        if (c.kind == kAsianGeo || c.kind == kAsianCv) log_sum += log(s);
        rmax = dmax(rmax, s);
        rmin = dmin(rmin, s);
    }
    const double n = static_cast<double>(c.n_steps);
    const double vanilla = dmax(phi * (s - c.strike), 0.0);
    switch (c.kind) {
        case kEuropean: return vanilla;
        case kDigital: return phi * (s - c.strike) > 0.0 ? (c.asset ? s : c.cash) : 0.0;
        case kAsianArith:
        case kAsianGeo: {
            const double avg = c.kind == kAsianArith ? sum / n : exp(log_sum / n);
            return dmax(phi * (c.floating ? s - avg : avg - c.strike), 0.0);
        }
        case kAsianCv:
            return c.discount * dmax(phi * (sum / n - c.strike), 0.0) -
                   (c.discount * dmax(phi * (exp(log_sum / n) - c.strike), 0.0) - c.kv_anchor);
        case kBarrier:
        case kBarrierBridge: return (c.out ? !breached : breached) ? vanilla : c.rebate;
        case kLookbackFixed: return c.type == 0 ? dmax(rmax - c.strike, 0.0) : dmax(c.strike - rmin, 0.0);
        default: return c.type == 0 ? s - rmin : rmax - s;
    }
}

__device__ __noinline__ Welford unit_wide(const DevContract& c, uint64_t base, uint32_t count, int rounds) {
    UnitSums acc;
    for (int j = 0; j < rounds; ++j) {
        const uint32_t o = static_cast<uint32_t>(j) * 32u + (threadIdx.x & 31u);
        double v = 0.0;
        if (o < count) {
            const double scale = c.kind == kAsianCv ? 1.0 : c.discount;
            v = scale * payoff_wide(c, base + o, false);
            if (c.antithetic) v = 0.5 * (v + scale * payoff_wide(c, base + o, true));
        }
        if (j == 0) acc.first(v);
        if (o < count) acc.add(v);
    }
    return acc.reduce(count);
}

// ---------------------------------------------------------------------------
// one unit in fixed point; ANTI: both halves of an antithetic sample
// ---------------------------------------------------------------------------
template <int KIND, bool ANTI>
__device__ __forceinline__ Welford unit_fixed(WarpSlot& w, const FixedShared& s, const FixedTables* __restrict__ g,
                                              uint64_t base, uint32_t count, int rounds) {
    const DevContract& c = w.c;
    const int lane = threadIdx.x & 31;
    const PhiloxKeys k = philox_keys(c.seed);
    const uint32_t path_hi = static_cast<uint32_t>(base >> 32);  // a unit is aligned to its size
    const int n = (KIND == kEuropean || KIND == kDigital) ? 1 : c.n_steps;
    UnitSums acc;
    for (int j = 0; j < rounds; ++j) {
        const uint32_t o = static_cast<uint32_t>(j) * 32u + lane;
        const uint32_t path_lo = static_cast<uint32_t>(base) + o;
        const PhiloxRow row = philox_row(path_lo, 0u, k);
        PhiloxRow row_u{};
        if constexpr (KIND == kBarrierBridge) row_u = philox_row(path_lo, 1u, k);
        Path64<KIND> p, q;
        for (int d0 = 0; d0 < n; d0 += 32) {
            if (j == 0 || n > 32) {  // the words of the next 32 steps, one per lane
                __syncwarp();
                PhiloxStep st = philox_step(static_cast<uint32_t>(d0 + lane), path_hi, k);
                st.carry = drift_carry(static_cast<uint32_t>(d0 + lane), c.y_drift_lo);
                w.step[lane] = st;
                __syncwarp();
            }
            const int m = min(32, n - d0);
            for (int d = 0; d < m; ++d) {
                const PhiloxStep st = w.step[d];
                const int64_t x = scaled_normal(normal_fixed(philox_word0(row, st, k), s, g), c.y_vs);
                uint32_t ubits = 0;
                if constexpr (KIND == kBarrierBridge) ubits = philox_word0(row_u, st, k);
                const int64_t drift = c.y_drift + st.carry;
                p.step(c, s, drift + x, ubits);
                if constexpr (ANTI) q.step(c, s, drift - x, ubits);
            }
        }
        auto sample = [&](const Path64<KIND>& path) {
            if constexpr (KIND == kAsianCv) return control_variate64(c, s, path);
            else return c.discount * payoff64<KIND>(c, c.spot, s, path);
        };
        double v = sample(p);
        if constexpr (ANTI) v = 0.5 * (v + sample(q));
        if (j == 0) acc.first(v);
        if (o < count) acc.add(v);
    }
    return acc.reduce(count);
}

struct Shared64 {
    FixedShared tables;
    WarpSlot slot[1];  // one per warp
};

// A call of one European or digital contract, latency above all: the contract is
// a launch parameter, the tables are read through the L1 cache (a CTA would copy
// 176 KB of them for a few hundred lookups), and the last CTA folds the units
// and writes the result to pinned host memory.  So a call is one launch, without
// copies.  Microseconds per call by number of paths, against upload, path
// kernel, merge kernel and read-back: 32: 36.3 -> 23.4, 1e4: 35.9 -> 27.5, 1e5:
// 48.3 -> 38.2, 1e6: 60.6 -> 57.8, 3e6: 85 -> 79, 1e7: 196 -> 203 (where the
// table in shared memory pays).  With several contracts the last CTA's folds
// follow one another: nine of 1e5 paths took 70 us longer.
__global__ void __launch_bounds__(kQuoteThreads, kQuoteCtas)
    quote64_kernel(const __grid_constant__ DevContract c, Welford* __restrict__ partials,
                    uint32_t* __restrict__ done, DevMcResult* __restrict__ result,
                    const FixedTables* __restrict__ g) {
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (kQuoteThreads / 32);
    const GlobalTables tables{g};
    for (uint32_t item = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; item < c.n_units; item += warps) {
        const uint64_t base = static_cast<uint64_t>(item) << (5 + c.unit_log);
        const uint64_t left = c.path_count - base;
        const uint32_t size = 32u << c.unit_log;
        const uint32_t count = left < size ? static_cast<uint32_t>(left) : size;
        const int rounds = static_cast<int>((count + 31u) / 32u);
        Welford r;
        if (c.frac == 0) {
            r = unit_wide(c, base, count, rounds);
        } else {  // unit_fixed of one step
            const PhiloxKeys k = philox_keys(c.seed);
            const PhiloxStep st = philox_step(0u, static_cast<uint32_t>(base >> 32), k);
            UnitSums acc;
            for (int j = 0; j < rounds; ++j) {
                const uint32_t o = static_cast<uint32_t>(j) * 32u + lane;
                const PhiloxRow row = philox_row(static_cast<uint32_t>(base) + o, 0u, k);
                const int64_t x = scaled_normal(tables.normal(philox_word0(row, st, k)), c.y_vs);
                auto sample = [&](int64_t y) {
                    const double last = c.spot * tables.exp2(y, c.frac), v = put_sign(last - c.strike, c.type);
                    const double pay = c.kind == kDigital ? (v > 0.0 ? (c.asset ? last : c.cash) : 0.0) : positive_part(v);
                    return c.discount * pay;
                };
                double v = sample(c.y_drift + x);
                if (c.antithetic) v = 0.5 * (v + sample(c.y_drift - x));
                if (j == 0) acc.first(v);
                if (o < count) acc.add(v);
            }
            r = acc.reduce(count);
        }
        if (lane == 0) partials[item] = r;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(done, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const MergedResult m = merge_items(partials, c.n_units, 1);
    if (threadIdx.x == 0) {
        *result = DevMcResult{m.mean, m.standard_error, m.count};
        *done = 0u;  // for the next call
    }
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1)
    path64_kernel(const DevContract* __restrict__ contracts, int n_contracts, const uint32_t* __restrict__ prefix,
                  uint32_t* __restrict__ ticket, Welford* __restrict__ partials, uint32_t* __restrict__ error_flag,
                  const FixedTables* __restrict__ g) {
    extern __shared__ __align__(16) unsigned char smem[];
    Shared64& sh = *reinterpret_cast<Shared64*>(smem);
    load_fixed_tables(sh.tables, g);
    const FixedShared& s = sh.tables;
    const int lane = threadIdx.x & 31;
    WarpSlot& w = sh.slot[threadIdx.x >> 5];
    const uint32_t first = prefix[0];
    int have = -1;
    uint32_t lo_item = 0, hi_item = 0;  // items of the contract in the slot
    for (ItemSource src(prefix[n_contracts] - first); src.valid(); src.next(ticket)) {
        const uint32_t item = src.item;
        if (have < 0 || item - lo_item >= hi_item - lo_item) {
            have = find_contract(prefix, n_contracts, item);
            lo_item = prefix[have] - first;
            hi_item = prefix[have + 1] - first;
            __syncwarp();
            copy_words(&w.c, &contracts[have]);
            __syncwarp();
        }
        const DevContract& c = w.c;
        const uint64_t base = static_cast<uint64_t>(item - lo_item) << (5 + c.unit_log);
        if (base >= c.path_count) {  // planning invariant broken: record, skip the item
            if (lane == 0) atomicOr(error_flag, 1u);
            continue;
        }
        const uint64_t left = c.path_count - base;
        const uint32_t size = 32u << c.unit_log;
        const uint32_t count = left < size ? static_cast<uint32_t>(left) : size;
        const int rounds = static_cast<int>((count + 31u) / 32u);
        Welford r;
#define MCD_UNIT(K)                                                          \
    case K:                                                                  \
        r = c.antithetic ? unit_fixed<K, true>(w, s, g, base, count, rounds) \
                         : unit_fixed<K, false>(w, s, g, base, count, rounds); \
        break;
        if (c.frac == 0) {
            r = unit_wide(c, base, count, rounds);
        } else {
            switch (c.kind) {
                MCD_UNIT(kEuropean)
                MCD_UNIT(kDigital)
                MCD_UNIT(kAsianArith)
                MCD_UNIT(kAsianGeo)
                MCD_UNIT(kAsianCv)
                MCD_UNIT(kBarrier)
                MCD_UNIT(kBarrierBridge)
                MCD_UNIT(kLookbackFixed)
                default:
                MCD_UNIT(kLookbackFloating)
            }
        }
#undef MCD_UNIT
        if (lane == 0) partials[item] = r;
    }
}

template <int THREADS>
cudaError_t launch_threads(int grid, const DevContract* c, int n, const uint32_t* prefix, uint32_t* ticket,
                           Welford* partials, uint32_t* err, const FixedTables* tables, cudaStream_t stream) {
    constexpr int bytes = static_cast<int>(sizeof(FixedShared) + sizeof(WarpSlot) * (THREADS / 32));
    cudaError_t e = cudaFuncSetAttribute(path64_kernel<THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    cudaGetLastError();  // report this launch only
    path64_kernel<THREADS><<<grid, THREADS, bytes, stream>>>(c, n, prefix, ticket, partials, err, tables);
    return cudaGetLastError();
}

__global__ void draws64_kernel(uint64_t seed, uint64_t path_begin, uint64_t n_paths, uint32_t draw_begin,
                               uint32_t n_draws, const FixedTables* __restrict__ g, double* __restrict__ out) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n_paths * n_draws) return;
    const uint64_t path = path_begin + i / n_draws;
    const PhiloxKeys k = philox_keys(seed);
    const PhiloxStep st = philox_step(draw_begin + static_cast<uint32_t>(i % n_draws), static_cast<uint32_t>(path >> 32), k);
    const uint32_t bits = philox_word0(philox_row(static_cast<uint32_t>(path), 0u, k), st, k);
    const int32_t upper = static_cast<int32_t>(bits) >> 31;
    const QuantArg a = quant_arg(2u * (bits ^ static_cast<uint32_t>(upper)) + 1u);
    out[i] = normal_to_double(FixedNormal{quant_eval(g->lo[a.entry], g->hi[a.entry], a.s), ~upper});
}

}  // namespace

cudaError_t fixed_tables_device(const FixedTables** out, cudaStream_t stream) {
    constexpr int kDevices = 64;
    static std::mutex lock;
    static void* address[kDevices] = {};
    static unsigned long long context[kDevices] = {};  // in which the address holds the tables
    int device = 0;
    unsigned long long id = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = device_context_id(&id);
    if (e != cudaSuccess) return e;
    if (device < 0 || device >= kDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> hold(lock);
    if (!address[device] || context[device] != id) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_fixed_tables);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(p, &fixed_tables(), sizeof(FixedTables), cudaMemcpyHostToDevice, stream);
        // A copy from pageable memory may return before its last part has arrived,
        // and launches on other streams do not wait for it.
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess) return e;
        address[device] = p;
        context[device] = id;
    }
    *out = static_cast<const FixedTables*>(address[device]);
    return cudaSuccess;
}

cudaError_t launch_path64_kernel(int variant, int grid, const DevContract* contracts, int n_contracts,
                                 const uint32_t* item_prefix, uint32_t* ticket, Welford* partials,
                                 uint32_t* error_flag, const FixedTables* tables, cudaStream_t stream) {
    switch (variant) {
        case 0: return launch_threads<512>(grid, contracts, n_contracts, item_prefix, ticket, partials, error_flag,
                                           tables, stream);
        case 4: return launch_threads<768>(grid, contracts, n_contracts, item_prefix, ticket, partials, error_flag,
                                           tables, stream);
        default: return launch_threads<1024>(grid, contracts, n_contracts, item_prefix, ticket, partials, error_flag,
                                             tables, stream);
    }
}

cudaError_t launch_quote64(int sm_count, const DevContract& c, Welford* partials, uint32_t* done, DevMcResult* result,
                           const FixedTables* tables, cudaStream_t stream) {
    constexpr uint32_t kWarps = kQuoteThreads / 32;
    const uint32_t ctas = std::max(1u, std::min((c.n_units + kWarps - 1) / kWarps, static_cast<uint32_t>(sm_count) * kQuoteCtas));
    cudaGetLastError();
    quote64_kernel<<<ctas, kQuoteThreads, 0, stream>>>(c, partials, done, result, tables);
    return cudaGetLastError();
}

cudaError_t launch_draws64_kernel(uint64_t seed, uint64_t path_begin, uint64_t n_paths, uint32_t draw_begin,
                                  uint32_t n_draws, const FixedTables* tables, double* out, cudaStream_t stream) {
    const uint64_t total = n_paths * n_draws;
    if (total == 0) return cudaSuccess;
    const unsigned blocks = static_cast<unsigned>((total + 255) / 256);
    cudaGetLastError();
    draws64_kernel<<<blocks, 256, 0, stream>>>(seed, path_begin, n_paths, draw_begin, n_draws, tables, out);
    return cudaGetLastError();
}

}  // namespace mcdg
