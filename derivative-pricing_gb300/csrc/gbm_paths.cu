// gbm_paths.cu -- the batched GBM path engine (European, digital, Asian,
// barrier, lookback) in FP32 as one persistent kernel, and the merge of both
// precisions (the FP64 paths are gbm_paths64.cu).
//
// Work decomposition.  Every contract's paths are cut into items of 128 << item_log
// paths, 4096 or fewer (items.hpp); one (contract, item) pair is one work item.  The
// host orders contracts longest-first and passes the running item count per
// contract (item_prefix).  A CTA of 128 threads claims items from a ticket
// counter (one atomicAdd per item, no waiting) until the list is exhausted.
// Inside an item, thread t simulates paths base + j*128 + t for j = 0, 1, ...,
// so the Philox counters of a warp are consecutive path indices.
//
// Determinism.  An item's Welford triple depends only on the item: per-thread
// shifted sums in j order (unit_sums.cuh), then a fixed warp shuffle tree and a
// fixed 4-warp tree.  The merge kernel folds a contract's items in a fixed tree (merge.cuh).
// Grid size and kernel variant (register budget) only decide who
// computes an item, never the arithmetic, so results are bitwise identical
// across launch shapes.
//
// Bound: the FMA pipes.  A 32x32->64 product occupies them for 4.3 cycles of a
// scheduler (measured; an FFMA 1.1, and the two do not overlap), so a
// path-step's 12 wide products, three half products and 16 FP32 operations
// take 82 cycles; measured 94 on the 4096-contract book.  Products that depend
// on the draw alone come from a table per item, those of the path alone are
// taken once per path (PhiloxStep, PhiloxRow): 18 products -> 14.5.  The book
// 313 -> 253 ms at 8 CTAs per SM (294 before at its best launch shape), of
// which 7 ms from sums instead of Welford merges in the reductions.  Logarithm
// and exponentials without their range tests (fp32_fast.cuh) left 248 ms at 7
// CTAs per SM (68 registers); one call, host side included, at 4, 5, 6, 7, 8, 12
// CTAs: 265, 257, 254, 253, 258, 272 ms.
//
// Reference semantics restated per kind (src/pricers/monte_carlo.cpp):
//   terminal products :135-149, path-dependent loop :154-177, Brownian-bridge
//   barrier :184-230, control-variate Asian :275-302, antithetic pairing
//   :73-79; payoffs include/mcd/payoffs/{european,digital,asian,barrier,
//   lookback}.hpp.
// nvcc-flags: --fmad=false
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "engine.hpp"
#include "merge.cuh"
#include "unit_sums.cuh"

namespace mcdg {

namespace {

// ===========================================================================
// FP32: log-space paths x = ln(S/S0), FP32 payoffs, FP64 accumulation.
// ===========================================================================
// Path-dependent products (Asians, barriers, lookbacks), two paths at once (or
// the two halves of an antithetic sample, which share their draws): two
// independent dependency chains per thread.  Each path's arithmetic does not
// depend on its partner.
template <int KIND>
struct Pair32 {
    float x[2], acc[2], acc2[2], xmax[2], xmin[2];  // log path, sum of S/S0, sum of x, extrema
    bool breached[2];

    __device__ __forceinline__ Pair32() {
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            x[p] = acc[p] = acc2[p] = xmax[p] = xmin[p] = 0.0f;
            breached[p] = false;
        }
    }

    template <bool ANTI>
    __device__ __forceinline__ void advance(const DevContract& c, const PhiloxKeys& k, const PhiloxStep* table,
                                            int count, const PhiloxRow (&row)[2], const PhiloxRow (&row_u)[2]) {
        const float mu = static_cast<float>(c.drift), sg = static_cast<float>(c.vs);
        const float lnh = static_cast<float>(c.log_h_rel);
        const float inv_denom = KIND == kBarrierBridge ? static_cast<float>(-2.0 / c.bb_denom) : 0.0f;
#pragma unroll 1
        for (int d = 0; d < count; ++d) {
            const PhiloxStep st = table[d];
            float z[2];
            if constexpr (ANTI) {
                const uint32_t bits[1] = {philox_word0(row[0], st, k)};
                float one[1];
                normals_from_bits_f32<1>(bits, one);
                z[0] = one[0];
                z[1] = -one[0];
            } else {
                const uint32_t bits[2] = {philox_word0(row[0], st, k), philox_word0(row[1], st, k)};
                normals_from_bits_f32<2>(bits, z);
            }
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const float x0 = x[p];
                x[p] = __fmaf_rn(sg, z[p], x[p] + mu);
                if constexpr (KIND == kAsianArith || KIND == kAsianCv) acc[p] += fast_exp(x[p]);
                if constexpr (KIND == kAsianGeo || KIND == kAsianCv) acc2[p] += x[p];
                if constexpr (KIND == kBarrier || KIND == kBarrierBridge) {
                    const bool crossed = c.up ? x[p] >= lnh : x[p] <= lnh;
                    breached[p] = breached[p] || crossed;
                }
                if constexpr (KIND == kBarrierBridge) {
                    if (!breached[p]) {
                        const float p_cross = fast_exp(inv_denom * (lnh - x0) * (lnh - x[p]));
                        breached[p] = uniform_from_bits_f32(philox_word0(row_u[p], st, k)) < p_cross;
                    }
                }
                if constexpr (KIND == kLookbackFixed || KIND == kLookbackFloating) {
                    xmax[p] = fmaxf(xmax[p], x[p]);
                    xmin[p] = fminf(xmin[p], x[p]);
                }
            }
        }
    }

    // The discounted sample in FP64 (the payoff itself is FP32).
    __device__ __forceinline__ double sample(const DevContract& c, int p) const {
        const float phi = c.type == 0 ? 1.0f : -1.0f;
        const float s0 = static_cast<float>(c.spot), strike = static_cast<float>(c.strike);
        const float inv_n = 1.0f / static_cast<float>(c.n_steps);
        const float last = s0 * __expf(x[p]);
        if constexpr (KIND == kAsianArith || KIND == kAsianGeo) {
            const float avg = KIND == kAsianArith ? s0 * (acc[p] * inv_n) : s0 * __expf(acc2[p] * inv_n);
            const float ref = c.floating ? (last - avg) : (avg - strike);
            return c.discount * static_cast<double>(fmaxf(phi * ref, 0.0f));
        } else if constexpr (KIND == kAsianCv) {
            const float a = s0 * (acc[p] * inv_n);
            const float g = s0 * __expf(acc2[p] * inv_n);
            const double ap = c.discount * static_cast<double>(fmaxf(phi * (a - strike), 0.0f));
            const double gp = c.discount * static_cast<double>(fmaxf(phi * (g - strike), 0.0f));
            return ap - (gp - c.kv_anchor);
        } else if constexpr (KIND == kBarrier || KIND == kBarrierBridge) {
            const float vanilla = fmaxf(phi * (last - strike), 0.0f);
            const bool pays = c.out ? !breached[p] : breached[p];
            return c.discount * static_cast<double>(pays ? vanilla : static_cast<float>(c.rebate));
        } else if constexpr (KIND == kLookbackFixed) {
            const float v = c.type == 0 ? fmaxf(s0 * __expf(xmax[p]) - strike, 0.0f)
                                        : fmaxf(strike - s0 * __expf(xmin[p]), 0.0f);
            return c.discount * static_cast<double>(v);
        } else {
            const float v = c.type == 0 ? (last - s0 * __expf(xmin[p])) : (s0 * __expf(xmax[p]) - last);
            return c.discount * static_cast<double>(v);
        }
    }
};

// European and digital: the discounted sample of one draw.
template <int KIND>
__device__ __forceinline__ double terminal32(const DevContract& c, uint32_t bits, bool neg) {
    const float phi = c.type == 0 ? 1.0f : -1.0f;
    const float mu = static_cast<float>(c.drift), sg = static_cast<float>(c.vs);
    const float s0 = static_cast<float>(c.spot), strike = static_cast<float>(c.strike);
    const float z0 = normal_from_bits_f32(bits);
    const float z = neg ? -z0 : z0;
    const float s = s0 * __expf(__fmaf_rn(sg, z, mu));
    float payoff;
    if constexpr (KIND == kEuropean) {
        payoff = fmaxf(phi * (s - strike), 0.0f);
    } else {
        const bool itm = phi * (s - strike) > 0.0f;
        payoff = itm ? (c.asset ? s : static_cast<float>(c.cash)) : 0.0f;
    }
    return c.discount * static_cast<double>(payoff);
}

// A warp's share of an item (valid in lane 0), from path base on, `rounds` paths
// per thread; table: the CTA's step table.
// Every thread runs every round (the table's refills are CTA barriers); a path
// past the contract's last one is simulated or skipped, and not counted.
template <int KIND>
__device__ Welford slab32(const DevContract& c, const PhiloxKeys& k, PhiloxStep* table, const uint64_t& base,
                          const int& rounds) {
    unsigned count = 0;
    UnitSums acc;
    auto add = [&](double v) {
        ++count;
        acc.add(v);
    };
    const uint32_t path_hi = static_cast<uint32_t>(base >> 32);  // a slab is aligned to its size
    if constexpr (KIND == kEuropean || KIND == kDigital) {
        const PhiloxStep st = philox_step(0u, path_hi, k);
        for (int j = 0; j < rounds; ++j) {
            const uint64_t path = base + static_cast<uint64_t>(j * kSlabThreads) + threadIdx.x;
            const uint32_t bits = philox_word0(philox_row(static_cast<uint32_t>(path), 0u, k), st, k);
            double v = terminal32<KIND>(c, bits, false);
            if (c.antithetic) v = 0.5 * (v + terminal32<KIND>(c, bits, true));
            if (j == 0) acc.first(v);
            if (path < c.path_count) add(v);
        }
    } else {
        const int n = c.n_steps;
        const bool once = n <= kStepTable;
        if (once) {
            fill_steps(table, 0, path_hi, k);
            __syncthreads();
        }
        const int stride = c.antithetic ? 1 : 2;  // paths of a thread per round, in path order
        for (int j = 0; j < rounds; j += stride) {
            const uint64_t path = base + static_cast<uint64_t>(j * kSlabThreads) + threadIdx.x;
            const bool live = path < c.path_count;
            double v0 = 0.0, v1 = 0.0;
            if (live || !once) {
                const uint32_t lo = static_cast<uint32_t>(path);
                const PhiloxRow row[2] = {philox_row(lo, 0u, k), philox_row(lo + kSlabThreads, 0u, k)};
                PhiloxRow row_u[2] = {};
                if constexpr (KIND == kBarrierBridge) {
                    row_u[0] = philox_row(lo, 1u, k);
                    row_u[1] = philox_row(c.antithetic ? lo : lo + kSlabThreads, 1u, k);
                }
                Pair32<KIND> pair;
                for (int d0 = 0; d0 < n; d0 += kStepTable) {
                    if (!once) {
                        __syncthreads();
                        fill_steps(table, d0, path_hi, k);
                        __syncthreads();
                    }
                    const int m = min(kStepTable, n - d0);
                    if (c.antithetic) pair.template advance<true>(c, k, table, m, row, row_u);
                    else pair.template advance<false>(c, k, table, m, row, row_u);
                }
                v0 = pair.sample(c, 0);
                v1 = pair.sample(c, 1);
                if (c.antithetic) v0 = 0.5 * (v0 + v1);
            }
            if (j == 0) acc.first(v0);
            if (live) add(v0);
            if (!c.antithetic && path + kSlabThreads < c.path_count) add(v1);
        }
    }
    return acc.reduce(__reduce_add_sync(0xffffffffu, count));
}

__device__ Welford run_slab(const DevContract& c, PhiloxStep* table, const uint64_t& base, const int& rounds) {
    const PhiloxKeys k = philox_keys(c.seed);
    switch (c.kind) {
        case kEuropean: return slab32<kEuropean>(c, k, table, base, rounds);
        case kDigital: return slab32<kDigital>(c, k, table, base, rounds);
        case kAsianArith: return slab32<kAsianArith>(c, k, table, base, rounds);
        case kAsianGeo: return slab32<kAsianGeo>(c, k, table, base, rounds);
        case kAsianCv: return slab32<kAsianCv>(c, k, table, base, rounds);
        case kBarrier: return slab32<kBarrier>(c, k, table, base, rounds);
        case kBarrierBridge: return slab32<kBarrierBridge>(c, k, table, base, rounds);
        case kLookbackFixed: return slab32<kLookbackFixed>(c, k, table, base, rounds);
        default: return slab32<kLookbackFloating>(c, k, table, base, rounds);
    }
}

template <int MINB>
__global__ void __launch_bounds__(kSlabThreads, MINB)
    path_kernel(const DevContract* __restrict__ contracts, int n_contracts,
                const uint32_t* __restrict__ item_prefix, uint32_t* __restrict__ ticket,
                Welford* __restrict__ partials, uint32_t* __restrict__ error_flag) {
    __shared__ uint32_t s_item, s_total;
    // an item's first path and its paths per thread: in registers they cost the
    // step loop 1.5 % (72 registers instead of 68)
    __shared__ uint64_t s_base;
    __shared__ int s_rounds;
    __shared__ Welford s_warp[kSlabThreads / 32];
    __shared__ DevContract s_contract;
    __shared__ PhiloxStep s_step[kStepTable];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    // The batch's items are read from the prefix (modulo 2^32, from its first
    // entry on), so a captured launch serves every path count of the same
    // contract count.
    const uint32_t first = item_prefix[0];
    if (threadIdx.x == 0) s_total = item_prefix[n_contracts] - first;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(ticket, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= s_total) return;
        // Largest contract index c with item_prefix[c] <= item (empty
        // contracts share their successor's prefix and are skipped).
        int lo = 0, hi = n_contracts;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (item_prefix[mid] - first <= item) lo = mid; else hi = mid;
        }
        static_assert(sizeof(DevContract) % 4 == 0 && sizeof(DevContract) / 4 <= kSlabThreads,
                      "contract staging assumes one word per thread");
        if (threadIdx.x < sizeof(DevContract) / 4)
            reinterpret_cast<uint32_t*>(&s_contract)[threadIdx.x] =
                reinterpret_cast<const uint32_t*>(&contracts[lo])[threadIdx.x];
        __syncthreads();
        const DevContract& c = s_contract;
        const uint32_t slab = item - (item_prefix[lo] - first);
        if (slab >= c.n_items) {  // planning invariant broken: record, skip the item
            if (threadIdx.x == 0) atomicOr(error_flag, 1u);
            __syncthreads();
            continue;
        }
        if (threadIdx.x == 0) {
            s_base = static_cast<uint64_t>(slab) * kSlabThreads << c.item_log;
            const uint64_t left = c.path_count - s_base, size = static_cast<uint64_t>(kSlabThreads) << c.item_log;
            s_rounds = static_cast<int>(((left < size ? left : size) + kSlabThreads - 1) / kSlabThreads);
        }
        __syncthreads();
        const Welford w = run_slab(c, s_step, s_base, s_rounds);
        if (lane == 0) s_warp[warp] = w;
        __syncthreads();
        if (threadIdx.x == 0) partials[item] = merge_warps(s_warp[0], s_warp[1], s_warp[2], s_warp[3]);
        __syncthreads();
    }
}

// One CTA per contract; results go to the caller's positions.
__global__ void __launch_bounds__(kMergeThreads)
    merge_kernel(const DevContract* __restrict__ contracts, const uint32_t* __restrict__ item_prefix,
                 const Welford* __restrict__ partials, DevMcResult* __restrict__ results) {
    const int ci = blockIdx.x;
    const MergedResult m =
        merge_items(partials + (item_prefix[ci] - item_prefix[0]), item_prefix[ci + 1] - item_prefix[ci], 1);
    if (threadIdx.x == 0) results[contracts[ci].orig_index] = DevMcResult{m.mean, m.standard_error, m.count};
}

// ---- parity kernels ----------------------------------------------------------
__global__ void philox_kernel(const uint4* __restrict__ counters, const uint2* __restrict__ keys,
                              size_t n, uint4* __restrict__ out) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint2 k = keys[i];
    out[i] = philox4x32_10(counters[i], k.x, k.y);
}

__global__ void draws_kernel(uint64_t seed, uint64_t path_begin, uint64_t n_paths,
                             uint32_t draw_begin, uint32_t n_draws, int stream_id, int precision,
                             double* __restrict__ out) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n_paths * n_draws) return;
    const uint64_t p = i / n_draws;
    const uint32_t d = static_cast<uint32_t>(i % n_draws);
    const PhiloxKeys k = philox_keys(seed);
    const PhiloxPath pp = philox_path(path_begin + p, static_cast<uint32_t>(stream_id), k);
    const uint32_t bits = philox_word0(pp, draw_begin + d, k);
    // (FP64 normals: draws64_kernel)
    out[i] = stream_id == 0   ? static_cast<double>(normal_from_bits_f32(bits))
             : precision == 0 ? uniform_open01_f64(bits)
                              : static_cast<double>(uniform_from_bits_f32(bits));
}

template <int MINB>
cudaError_t launch_one(int grid, const DevContract* c, int n, const uint32_t* prefix, uint32_t* ticket,
                       Welford* partials, uint32_t* err, cudaStream_t stream) {
    cudaGetLastError();  // report this launch only
    path_kernel<MINB><<<grid, kSlabThreads, 0, stream>>>(c, n, prefix, ticket, partials, err);
    return cudaGetLastError();
}

// Digest of a word array: sum over i of splitmix64's finaliser (Steele, Lea
// and Flood, OOPSLA 2014) applied to word_i + (i + 1) * golden-ratio constant.
// Integer sums do not depend on the order of the additions, so the digest is
// the same for any grid; one CTA suffices for a contract list.
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__global__ void __launch_bounds__(256) words_digest_kernel(const uint64_t* __restrict__ words, size_t n,
                                                           uint64_t* __restrict__ out) {
    __shared__ uint64_t part[8];
    uint64_t acc = 0;
    for (size_t i = threadIdx.x; i < n; i += blockDim.x) acc += mix64(words[i] + (i + 1) * 0x9E3779B97F4A7C15ull);
    for (int off = 16; off >= 1; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint64_t total = 0;
        for (int w = 0; w < 8; ++w) total += part[w];
        *out = total;
    }
}

}  // namespace

cudaError_t launch_words_digest(const uint64_t* words, size_t n_words, uint64_t* out, cudaStream_t stream) {
    cudaGetLastError();
    words_digest_kernel<<<1, 256, 0, stream>>>(words, n_words, out);
    return cudaGetLastError();
}

cudaError_t launch_path_kernel(int precision, int variant, int grid, const DevContract* contracts,
                               int n_contracts, const uint32_t* item_prefix, uint32_t* ticket,
                               Welford* partials, uint32_t* error_flag, const FixedTables* tables,
                               cudaStream_t stream) {
    if (precision == 0)
        return launch_path64_kernel(variant, grid, contracts, n_contracts, item_prefix, ticket, partials, error_flag,
                                    tables, stream);
    switch (variant) {
        case 0: return launch_one<4>(grid, contracts, n_contracts, item_prefix, ticket, partials, error_flag, stream);
        case 1: return launch_one<8>(grid, contracts, n_contracts, item_prefix, ticket, partials, error_flag, stream);
        case 2: return launch_one<12>(grid, contracts, n_contracts, item_prefix, ticket, partials, error_flag, stream);
        case 3: return launch_one<16>(grid, contracts, n_contracts, item_prefix, ticket, partials, error_flag, stream);
        default: return launch_one<7>(grid, contracts, n_contracts, item_prefix, ticket, partials, error_flag, stream);
    }
}

cudaError_t path_kernel_occupancy(int precision, int variant, int* blocks) {
    if (precision == 0) {  // one CTA per SM shares the fixed-point tables
        *blocks = 1;
        return cudaSuccess;
    }
    switch (variant) {
        case 0: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, path_kernel<4>, kSlabThreads, 0);
        case 1: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, path_kernel<8>, kSlabThreads, 0);
        case 2: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, path_kernel<12>, kSlabThreads, 0);
        case 3: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, path_kernel<16>, kSlabThreads, 0);
        default: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, path_kernel<7>, kSlabThreads, 0);
    }
}

cudaError_t launch_merge_kernel(const DevContract* contracts, int n_contracts,
                                const uint32_t* item_prefix, const Welford* partials,
                                void* results, cudaStream_t stream) {
    if (n_contracts == 0) return cudaSuccess;
    cudaGetLastError();
    merge_kernel<<<n_contracts, kMergeThreads, 0, stream>>>(contracts, item_prefix, partials,
                                                            static_cast<DevMcResult*>(results));
    return cudaGetLastError();
}

cudaError_t launch_philox_kernel(const uint32_t* counters, const uint32_t* keys, size_t n,
                                 uint32_t* out, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    const int threads = 256;
    const unsigned blocks = static_cast<unsigned>((n + threads - 1) / threads);
    cudaGetLastError();
    philox_kernel<<<blocks, threads, 0, stream>>>(reinterpret_cast<const uint4*>(counters),
                                                  reinterpret_cast<const uint2*>(keys), n,
                                                  reinterpret_cast<uint4*>(out));
    return cudaGetLastError();
}

cudaError_t launch_draws_kernel(uint64_t seed, uint64_t path_begin, uint64_t n_paths,
                                uint32_t draw_begin, uint32_t n_draws, int stream_id,
                                int precision, double* out, cudaStream_t stream) {
    const uint64_t total = n_paths * n_draws;
    if (total == 0) return cudaSuccess;
    const int threads = 256;
    const unsigned blocks = static_cast<unsigned>((total + threads - 1) / threads);
    cudaGetLastError();
    draws_kernel<<<blocks, threads, 0, stream>>>(seed, path_begin, n_paths, draw_begin, n_draws,
                                                 stream_id, precision, out);
    return cudaGetLastError();
}

}  // namespace mcdg
