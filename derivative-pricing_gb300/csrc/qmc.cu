// qmc.cu -- Sobol quasi-Monte Carlo pricing of a batch of GBM contracts with
// Brownian-bridge paths, as one persistent kernel per precision.
//
// Reference semantics: src/core/sobol.cpp:83-97 (Gray-code point, indices
// 1..N as in src/pricers/qmc.cpp:20-25), src/models/brownian_bridge_path.cpp
// :20-77 (bisection bridge: terminal point from dimension 0, then breadth-
// first midpoints, dimension = draw number), src/pricers/qmc.cpp:15-57
// (European: one dimension and the exact terminal spot; Asian: dims =
// monitoring points, price = mean of discounted payoffs, no standard error).
// The same bridge paths also price the other batch products (geometric Asian,
// discrete barrier, lookback), which the reference prices by Monte Carlo only.
//
// Work decomposition, slab reduction and merge are the path engine's
// (gbm_paths.cu): (contract, 4096-path slab) items claimed from a ticket,
// fixed trees, so results do not depend on the launch shape.
//
// Per path, the bridge program (qmc.hpp) is walked in depth-first pre-order:
// each node takes its Sobol coordinate (XOR of the direction numbers of the
// set bits of the Gray code), the inverse normal, and the bridge update from
// the two ancestor values it sits between; spots are folded into the payoff
// aggregates at once (sum, log-sum, extrema, barrier test, terminal spot), so
// no path array is kept: one value per tree depth.
//
// nvcc-flags: --fmad=false
#include <cuda_runtime.h>

#include <type_traits>

#include "device_common.cuh"
#include "engine.hpp"
#include "qmc.hpp"
#include "unit_sums.cuh"

namespace mcdg {

namespace {

__device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double dmin(double a, double b) { return (b < a) ? b : a; }

// Sobol coordinate bits of `dim` for Gray code `gray` (sobol.cpp:87-94;
// directions[dim * 32 + b] is the reference's v[b + 1]).
__device__ __forceinline__ uint32_t sobol_x(const uint32_t* __restrict__ dirs, uint32_t dim, uint32_t gray) {
    const uint32_t* v = dirs + dim * kSobolBits;
    uint32_t x = 0;
    while (gray != 0u) {
        const int b = __ffs(gray) - 1;
        x ^= __ldg(v + b);
        gray &= gray - 1u;
    }
    return x;
}

// Sobol coordinates of a warp's 32 consecutive indices.  Path p has index
// I = p + 1; a warp's paths are B .. B+31 with B a multiple of 32, so
// I = B' + low with B' in {B, B + 32} (B + 32 for the last lane only) and
// low < 32, and gray(B' + low) = gray(B') ^ gray(low).  The coordinate is
// linear in the Gray-code bits over GF(2): x(I) = X(B') ^ Y(low).  X is
// computed once per warp and dimension (lanes share the dimensions) into
// shared memory; Y depends on the lane and dimension only and is a table
// (kSobolDims x 32, uploaded with the directions).  A draw is then one XOR
// of two loads instead of a loop over the set bits of the index.
struct SobolLane {
    const uint32_t* x;  // this warp's X for this lane's B' (indexed by dimension)
    const uint32_t* y;  // Y table column of this lane (stride 32)
    __device__ __forceinline__ uint32_t operator()(uint32_t dim) const { return x[dim] ^ __ldg(y + dim * 32u); }
};

constexpr int kSxStride = kSobolDims + 1;  // +1 word: the last lane's row sits in another bank
constexpr int kSxPerWarp = 2 * kSxStride;
constexpr int kQuad = 4;  // FP32: paths per thread at a time

// Bridge coefficients of one contract in program order, FP64 kernel.
struct QmcTables64 {
    BridgeNode node[kSobolDims];
    double a[kSobolDims], sd[kSobolDims], drift[kSobolDims];
};

// FP32 kernel: one 16-byte record per node, read with one shared-memory load
// (the same address across the warp): the FP32 coefficients and the node's
// Sobol dimension and slots packed into the last word.
struct QmcTables32 {
    float4 node[kSobolDims];     // {a, sd, drift, bits(meta)}
    uint4 mask[kSobolDims][2];   // quad_qmc32: of lanes 0..30, of lane 31
};
__device__ __forceinline__ uint32_t meta_dim(uint32_t m) { return m & 0xFFu; }
__device__ __forceinline__ uint32_t meta_left(uint32_t m) { return (m >> 8) & 0xFu; }
__device__ __forceinline__ uint32_t meta_right(uint32_t m) { return (m >> 12) & 0xFu; }
__device__ __forceinline__ uint32_t meta_out(uint32_t m) { return (m >> 16) & 0xFu; }

template <int PREC>
using QmcTables = typename std::conditional<PREC == 0, QmcTables64, QmcTables32>::type;

// FP32: a thread's four paths are 32 indices apart, B + 32 p + lane with B a
// multiple of 128, so the indices' high parts differ in bits 5 and 6 only:
// X(B + 32 p) = X(B) ^ M_p, M_p the directions of the bits of gray(32 p), one
// row X(B) for all four.  Lane 31's low part is 0 of the next 32: its masks are
// M_1, M_2, M_3 and, for its last path, the row X(B + 128).
__device__ __forceinline__ uint3 quad_masks(const uint32_t* __restrict__ by_bit, uint32_t dim) {
    const uint32_t v4 = __ldg(by_bit + 4 * kSobolDims + dim), v5 = __ldg(by_bit + 5 * kSobolDims + dim),
                   v6 = __ldg(by_bit + 6 * kSobolDims + dim);
    return make_uint3(v4 ^ v5, v5 ^ v6, v4 ^ v6);  // gray(32), gray(64), gray(96)
}

// Bridge coefficients of one contract in program order, with the reference's
// operations (brownian_bridge_path.cpp:29-31, :52-62, :71-74): t_i = i T / n.
template <int PREC>
__device__ void fill_tables(const DevContract& c, const DevQmc& q, const BridgeNode* __restrict__ programs,
                            const uint32_t* __restrict__ by_bit, QmcTables<PREC>& S) {
    const int n = c.n_steps;
    const double nd = static_cast<double>(n);
    auto t_of = [&](int i) { return static_cast<double>(i) * q.time / nd; };
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        const BridgeNode b = programs[q.prog_offset + e];
        const double tm = t_of(b.t_mid + 1);
        const bool root = b.t_left < 0 && b.t_right < 0;
        double a, sd;
        if (root) {
            a = 0.0;
            sd = sqrt(t_of(n));
        } else {
            const double tl = b.t_left < 0 ? 0.0 : t_of(b.t_left + 1);
            const double tr = t_of(b.t_right + 1);
            a = (tm - tl) / (tr - tl);
            sd = sqrt((tm - tl) * (tr - tm) / (tr - tl));
        }
        const double drift = q.drift_rate * tm;
        if constexpr (PREC == 0) {
            S.node[e] = b;
            S.a[e] = a;
            S.sd[e] = sd;
            S.drift[e] = drift;
        } else {
            const uint32_t meta = static_cast<uint32_t>(b.dim) | (static_cast<uint32_t>(b.slot_left) << 8) |
                                  (static_cast<uint32_t>(b.slot_right) << 12) |
                                  (static_cast<uint32_t>(b.slot_out) << 16);
            S.node[e] = make_float4(static_cast<float>(a), static_cast<float>(sd), static_cast<float>(drift),
                                    __uint_as_float(meta));
            const uint3 m = quad_masks(by_bit, b.dim);
            S.mask[e][0] = make_uint4(0u, m.x, m.y, m.z);
            S.mask[e][1] = make_uint4(m.x, m.y, m.z, 0u);
        }
    }
}

template <int KIND>
__device__ double sample_qmc64(const DevContract& c, const DevQmc& q, const QmcTables64& S, const SobolLane& sob) {
    const double phi = c.type == 0 ? 1.0 : -1.0;
    if constexpr (KIND == kEuropean || KIND == kDigital) {  // qmc.cpp:20-27
        const double z = inv_normal_cdf_f64(static_cast<double>(sob(0u)) * (1.0 / 4294967296.0));
        const double s = c.spot * exp(c.drift + c.vs * z);
        if constexpr (KIND == kEuropean) {
            return c.discount * dmax(phi * (s - c.strike), 0.0);
        } else {
            const bool itm = phi * (s - c.strike) > 0.0;
            return c.discount * (itm ? (c.asset ? s : c.cash) : 0.0);
        }
    } else {
        const int n = c.n_steps;
        double w[kBridgeSlots];
        w[0] = 0.0;
        double sum = 0.0, lsum = 0.0, last = c.spot, hi = c.spot, lo = c.spot;
        bool breached = false;
        for (int e = 0; e < n; ++e) {
            const BridgeNode& b = S.node[e];
            const double z = inv_normal_cdf_f64(static_cast<double>(sob(b.dim)) * (1.0 / 4294967296.0));
            double val;
            if (b.t_left < 0 && b.t_right < 0) {
                val = S.sd[e] * z;
            } else {
                const double wl = w[b.slot_left], wr = w[b.slot_right];
                val = wl + S.a[e] * (wr - wl) + S.sd[e] * z;
            }
            w[b.slot_out] = val;
            const double s = c.spot * exp(S.drift[e] + q.vol * val);
            if (b.t_mid == n - 1) last = s;
            if constexpr (KIND == kAsianArith) {
                sum += s;
            } else if constexpr (KIND == kAsianGeo) {
                lsum += log(s);
            } else if constexpr (KIND == kBarrier) {
                breached = breached || (c.up ? s >= c.barrier : s <= c.barrier);
            } else {
                hi = dmax(hi, s);
                lo = dmin(lo, s);
            }
        }
        const double nd = static_cast<double>(n);
        if constexpr (KIND == kAsianArith || KIND == kAsianGeo) {  // qmc.cpp:44-53
            const double avg = KIND == kAsianArith ? sum / nd : exp(lsum / nd);
            const double ref = c.floating ? (last - avg) : (avg - c.strike);
            return c.discount * dmax(phi * ref, 0.0);
        } else if constexpr (KIND == kBarrier) {
            const double vanilla = dmax(phi * (last - c.strike), 0.0);
            const bool pays = c.out ? !breached : breached;
            return c.discount * (pays ? vanilla : c.rebate);
        } else if constexpr (KIND == kLookbackFixed) {
            return c.discount * (c.type == 0 ? dmax(hi - c.strike, 0.0) : dmax(c.strike - lo, 0.0));
        } else {
            return c.discount * (c.type == 0 ? (last - lo) : (hi - last));
        }
    }
}

// FP32: log-space spots x = ln(S/S0), FP32 payoff, FP64 accumulation.
__device__ __forceinline__ double terminal_qmc32(const DevContract& c, uint32_t x) {  // European, digital
    const float phi = c.type == 0 ? 1.0f : -1.0f;
    const float s0 = static_cast<float>(c.spot), strike = static_cast<float>(c.strike);
    const float z = normal_from_sobol_f32(x);
    const float s = s0 * __expf(__fmaf_rn(static_cast<float>(c.vs), z, static_cast<float>(c.drift)));
    float payoff;
    if (c.kind == kEuropean) {
        payoff = fmaxf(phi * (s - strike), 0.0f);
    } else {
        const bool itm = phi * (s - strike) > 0.0f;
        payoff = itm ? (c.asset ? s : static_cast<float>(c.cash)) : 0.0f;
    }
    return c.discount * static_cast<double>(payoff);
}

// The four paths of a thread: they share the program's records, their slots'
// addresses, the row X and the lane's Y word, and their chains interleave.
// Bound by issue.  A book of 4096 mixed contracts of 1e4 to 1e6 paths: one path
// at a time 282 ms, two 277 (both waiting on bank conflicts of the directions,
// see add_x), with the bit-major directions and the node fetched one ahead 173,
// the root taken out of the loop 165, four paths from one row 149 (47
// instructions per path-step instead of 59, issue 83 % at 5 CTAs per SM); 146
// with subnormals flushed in ex2 and lg2 alone (fp32_fast.cuh).
// The bridge values live in shared memory, one column per thread and path
// (w[slot * 512 + 128 p]): a node's slots are known only at run time, so a
// register array would be spilled to local memory.
template <int KIND>
__device__ __forceinline__ void quad_qmc32(const DevContract& c, const DevQmc& q, const QmcTables32& S,
                                           const uint32_t* row, const uint32_t* row_last,
                                           const uint32_t* __restrict__ y, float* __restrict__ w,
                                           double (&out)[kQuad]) {
    const float phi = c.type == 0 ? 1.0f : -1.0f;
    const float s0 = static_cast<float>(c.spot);
    const float strike = static_cast<float>(c.strike);
    const int n = c.n_steps;
    const float vol = static_cast<float>(q.vol);
    const float lnh = static_cast<float>(c.log_h_rel);
    float acc[kQuad], xlast[kQuad], xmax[kQuad], xmin[kQuad];
    bool breached[kQuad];
#pragma unroll
    for (int p = 0; p < kQuad; ++p) {
        w[p * kSlabThreads] = 0.0f;
        acc[p] = xmax[p] = xmin[p] = 0.0f;
        breached[p] = false;
    }
    auto observe = [&](int p, float x) {
        if constexpr (KIND == kAsianArith) {
            acc[p] += fast_exp(x);
        } else if constexpr (KIND == kAsianGeo) {
            acc[p] += x;
        } else if constexpr (KIND == kBarrier) {
            breached[p] = breached[p] || (c.up ? x >= lnh : x <= lnh);
        } else {
            xmax[p] = fmaxf(xmax[p], x);
            xmin[p] = fminf(xmin[p], x);
        }
    };
    auto offset = [&](uint32_t slot) { return w + slot * (kQuad * kSlabThreads); };
    const uint4* mask = &S.mask[0][(threadIdx.x & 31) == 31 ? 1 : 0];
    // the next node's record and draws are fetched a node ahead
    float4 ahead;
    uint4 bits;
    auto fetch = [&](int e) {
        ahead = S.node[e];
        const uint32_t dim = meta_dim(__float_as_uint(ahead.w));
        const uint32_t yw = __ldg(y + dim * 32u), x = row[dim];
        const uint4 m = mask[2 * e];
        bits = make_uint4(x ^ yw ^ m.x, x ^ yw ^ m.y, x ^ yw ^ m.z, row_last[dim] ^ yw ^ m.w);
    };
    fetch(0);
    {  // the program starts at its root, the terminal point, which has no ancestors
        const float4 nd = ahead;
        const uint32_t u[kQuad] = {bits.x, bits.y, bits.z, bits.w};
        fetch(n > 1 ? 1 : 0);
        float z[kQuad];
        normals_from_sobol_f32<kQuad>(u, z);
        float* at = offset(meta_out(__float_as_uint(nd.w)));
#pragma unroll
        for (int p = 0; p < kQuad; ++p) {
            const float val = nd.y * z[p];
            at[p * kSlabThreads] = val;
            xlast[p] = __fmaf_rn(vol, val, nd.z);
            observe(p, xlast[p]);
        }
    }
    for (int e = 1; e < n; ++e) {
        const float4 nd = ahead;
        const uint32_t meta = __float_as_uint(nd.w);
        const uint32_t u[kQuad] = {bits.x, bits.y, bits.z, bits.w};
        fetch(min(e + 1, n - 1));
        float z[kQuad];
        normals_from_sobol_f32<kQuad>(u, z);
        const float *left = offset(meta_left(meta)), *right = offset(meta_right(meta));
        float* at = offset(meta_out(meta));
#pragma unroll
        for (int p = 0; p < kQuad; ++p) {
            const float wl = left[p * kSlabThreads], wr = right[p * kSlabThreads];
            const float val = __fmaf_rn(nd.y, z[p], __fmaf_rn(nd.x, wr - wl, wl));
            at[p * kSlabThreads] = val;
            observe(p, __fmaf_rn(vol, val, nd.z));
        }
    }
    const float inv_n = 1.0f / static_cast<float>(n);
#pragma unroll
    for (int p = 0; p < kQuad; ++p) {
        const float last = s0 * __expf(xlast[p]);
        float v;
        if constexpr (KIND == kAsianArith || KIND == kAsianGeo) {
            const float avg = KIND == kAsianArith ? s0 * (acc[p] * inv_n) : s0 * __expf(acc[p] * inv_n);
            v = fmaxf(phi * (c.floating ? (last - avg) : (avg - strike)), 0.0f);
        } else if constexpr (KIND == kBarrier) {
            const float vanilla = fmaxf(phi * (last - strike), 0.0f);
            v = (c.out ? !breached[p] : breached[p]) ? vanilla : static_cast<float>(c.rebate);
        } else if constexpr (KIND == kLookbackFixed) {
            v = c.type == 0 ? fmaxf(s0 * __expf(xmax[p]) - strike, 0.0f) : fmaxf(strike - s0 * __expf(xmin[p]), 0.0f);
        } else {
            v = c.type == 0 ? (last - s0 * __expf(xmin[p])) : (s0 * __expf(xmax[p]) - last);
        }
        out[p] = c.discount * static_cast<double>(v);
    }
}

// Adds (over GF(2)) the directions of the set bits of `gray` to a row of X, the
// dimensions spread over the lanes; start: from zero.  From one group of paths
// to the next only one to three bits of the Gray code change, so the rows are
// updated rather than computed anew.  The directions are read bit-major: from
// the dimension-major table a warp's 32 loads were 128 bytes apart, and their
// wavefronts held the L1 for half of the kernel's cycles.
__device__ __forceinline__ void add_x(uint32_t* row, const uint32_t* __restrict__ by_bit, uint32_t ndims, uint32_t gray,
                                      bool start) {
    for (uint32_t d = threadIdx.x & 31; d < ndims; d += 32) {
        uint32_t x = start ? 0u : row[d];
        for (uint32_t g = gray; g != 0u; g &= g - 1u) x ^= __ldg(by_bit + (__ffs(g) - 1) * kSobolDims + d);
        row[d] = x;
    }
}

__device__ __forceinline__ uint32_t gray_code(uint64_t i) { return static_cast<uint32_t>(i ^ (i >> 1)); }

// Rows X(b0) and X(b0 + span) of a warp's paths from b0 on (the second for the
// last lane).  They hold those of the paths from `before` on, or nothing yet.
__device__ __forceinline__ void fill_x(uint32_t* xw, const uint32_t* __restrict__ by_bit, uint32_t ndims, uint64_t b0,
                                       uint64_t span, uint64_t before, bool start) {
    const uint32_t g0 = gray_code(b0), g1 = gray_code(b0 + span);
    add_x(xw, by_bit, ndims, start ? g0 : g0 ^ gray_code(before), start);
    add_x(xw + kSxStride, by_bit, ndims, start ? g1 : g1 ^ gray_code(before + span), start);
}

// A warp's share of a slab; valid in lane 0 (FP32: shifted sums, FP64: a
// Welford triple per lane, merged in a fixed tree).
template <int PREC, int KIND>
__device__ Welford slab_qmc(const DevContract& c, const DevQmc& q, const QmcTables<PREC>& S,
                            const uint32_t* __restrict__ by_bit, const uint32_t* __restrict__ ytab, uint32_t* sx,
                            float* bridge_w, uint64_t base) {
    constexpr bool kTerminal = KIND == kEuropean || KIND == kDigital;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t ndims = kTerminal ? 1u : static_cast<uint32_t>(c.n_steps);
    uint32_t* xw = sx + warp * kSxPerWarp;
    const uint32_t* my_x = xw + (lane == 31 ? kSxStride : 0);
    if constexpr (PREC == 0) {
        const SobolLane sob{my_x, ytab + lane};
        Welford w{0ull, 0.0, 0.0};
        for (int j = 0; j < kPathsPerThread; ++j) {
            const uint64_t b0 = base + static_cast<uint64_t>(j * kSlabThreads) + 32u * warp;  // this warp's first path
            if (b0 >= c.path_count) break;  // uniform per warp
            __syncwarp();
            fill_x(xw, by_bit, ndims, b0, 32, b0 - kSlabThreads, j == 0);
            __syncwarp();
            if (b0 + lane < c.path_count) welford_add(w, sample_qmc64<KIND>(c, q, S, sob));
        }
        return welford_warp_reduce(w);
    } else {
        UnitSums acc;
        unsigned count = 0;
        uint3 m0 = make_uint3(0u, 0u, 0u);
        if constexpr (kTerminal) m0 = quad_masks(by_bit, 0u);
        for (int j = 0; j < kPathsPerThread; j += kQuad) {  // 128 paths of a warp at a time
            const uint64_t b0 = base + static_cast<uint64_t>(j * kSlabThreads) + kQuad * 32u * warp;
            if (b0 >= c.path_count) break;  // uniform per warp
            __syncwarp();
            fill_x(xw, by_bit, ndims, b0, kQuad * 32u, b0 - kQuad * kSlabThreads, j == 0);
            __syncwarp();
            double v[kQuad];
            if constexpr (kTerminal) {
                const uint32_t x = xw[0] ^ __ldg(ytab + lane);
                const bool end = lane == 31;
                v[0] = terminal_qmc32(c, end ? x ^ m0.x : x);
                v[1] = terminal_qmc32(c, x ^ (end ? m0.y : m0.x));
                v[2] = terminal_qmc32(c, x ^ (end ? m0.z : m0.y));
                v[3] = terminal_qmc32(c, end ? xw[kSxStride] ^ __ldg(ytab + lane) : x ^ m0.z);
            } else {
                quad_qmc32<KIND>(c, q, S, xw, my_x, ytab + lane, bridge_w + threadIdx.x, v);
            }
            if (j == 0) acc.first(v[0]);
#pragma unroll
            for (int p = 0; p < kQuad; ++p) {
                if (b0 + 32u * p + lane < c.path_count) {
                    ++count;
                    acc.add(v[p]);
                }
            }
        }
        return acc.reduce(__reduce_add_sync(0xffffffffu, count));
    }
}

template <int PREC>
__device__ Welford run_qmc_slab(const DevContract& c, const DevQmc& q, const QmcTables<PREC>& S,
                                const uint32_t* __restrict__ by_bit, const uint32_t* __restrict__ ytab, uint32_t* sx,
                                float* bridge_w, uint64_t base) {
    switch (c.kind) {
        case kEuropean: return slab_qmc<PREC, kEuropean>(c, q, S, by_bit, ytab, sx, bridge_w, base);
        case kDigital: return slab_qmc<PREC, kDigital>(c, q, S, by_bit, ytab, sx, bridge_w, base);
        case kAsianArith: return slab_qmc<PREC, kAsianArith>(c, q, S, by_bit, ytab, sx, bridge_w, base);
        case kAsianGeo: return slab_qmc<PREC, kAsianGeo>(c, q, S, by_bit, ytab, sx, bridge_w, base);
        case kBarrier: return slab_qmc<PREC, kBarrier>(c, q, S, by_bit, ytab, sx, bridge_w, base);
        case kLookbackFixed: return slab_qmc<PREC, kLookbackFixed>(c, q, S, by_bit, ytab, sx, bridge_w, base);
        default: return slab_qmc<PREC, kLookbackFloating>(c, q, S, by_bit, ytab, sx, bridge_w, base);
    }
}

template <int PREC>
__global__ void __launch_bounds__(kSlabThreads)
    qmc_kernel(const DevContract* __restrict__ contracts, const DevQmc* __restrict__ qmc, int n_contracts,
               const uint32_t* __restrict__ item_prefix, uint32_t total_items,
               const BridgeNode* __restrict__ programs, const uint32_t* __restrict__ dirs,
               uint32_t* __restrict__ ticket, Welford* __restrict__ partials, uint32_t* __restrict__ error_flag) {
    const uint32_t* ytab = dirs + kSobolDims * kSobolBits;  // Y table, then the directions bit-major
    const uint32_t* by_bit = ytab + kSobolDims * 32;
    __shared__ uint32_t s_sx[(kSlabThreads / 32) * kSxPerWarp];
    __shared__ uint32_t s_item;
    __shared__ Welford s_warp[kSlabThreads / 32];
    __shared__ DevContract s_c;
    __shared__ DevQmc s_q;
    __shared__ QmcTables<PREC> S;
    __shared__ float s_bridge[PREC == 0 ? 1 : kQuad * kBridgeSlots * kSlabThreads];  // FP32 bridge values, per thread and path
    __shared__ int s_loaded;  // sorted index of the contract whose tables are in S
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_loaded = -1;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(ticket, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= total_items) return;
        int lo = 0, hi = n_contracts;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (item_prefix[mid] <= item) lo = mid; else hi = mid;
        }
        const bool reload = s_loaded != lo;
        __syncthreads();
        if (reload) {
            for (int i = threadIdx.x; i < static_cast<int>(sizeof(DevContract) / 4); i += kSlabThreads)
                reinterpret_cast<uint32_t*>(&s_c)[i] = reinterpret_cast<const uint32_t*>(&contracts[lo])[i];
            for (int i = threadIdx.x; i < static_cast<int>(sizeof(DevQmc) / 4); i += kSlabThreads)
                reinterpret_cast<uint32_t*>(&s_q)[i] = reinterpret_cast<const uint32_t*>(&qmc[lo])[i];
            __syncthreads();
            if (s_c.kind != kEuropean && s_c.kind != kDigital) {
                if (s_c.n_steps > kSobolDims) {  // planning invariant broken
                    if (threadIdx.x == 0) atomicOr(error_flag, 2u);
                    continue;
                }
                fill_tables<PREC>(s_c, s_q, programs, by_bit, S);
            }
            if (threadIdx.x == 0) s_loaded = lo;
            __syncthreads();
        }
        const uint32_t slab = item - item_prefix[lo];
        if (slab >= s_c.n_slabs) {
            if (threadIdx.x == 0) atomicOr(error_flag, 1u);
            continue;
        }
        const Welford w = run_qmc_slab<PREC>(s_c, s_q, S, by_bit, ytab, s_sx, s_bridge, static_cast<uint64_t>(slab) * kSlabPaths);
        if (lane == 0) s_warp[warp] = w;
        __syncthreads();
        if (threadIdx.x == 0)
            partials[item] = welford_merge(welford_merge(s_warp[0], s_warp[1]), welford_merge(s_warp[2], s_warp[3]));
    }
}

__global__ void sobol_points_kernel(const uint32_t* __restrict__ dirs, uint32_t dim0, uint32_t n_dims,
                                    uint64_t index0, uint64_t n_idx, double* __restrict__ out) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n_idx * n_dims) return;
    const uint64_t index = index0 + i / n_dims;
    const uint32_t d = dim0 + static_cast<uint32_t>(i % n_dims);
    const uint32_t gray = static_cast<uint32_t>(index ^ (index >> 1));
    out[i] = index == 0 ? 0.0 : static_cast<double>(sobol_x(dirs, d, gray)) * (1.0 / 4294967296.0);
}

}  // namespace

cudaError_t launch_qmc_kernel(int precision, int grid, const DevContract* contracts, const DevQmc* qmc,
                              int n_contracts, const uint32_t* item_prefix, uint32_t total_items,
                              const BridgeNode* programs, const uint32_t* directions, uint32_t* ticket,
                              Welford* partials, uint32_t* error_flag, cudaStream_t stream) {
    cudaGetLastError();
    if (precision == 0)
        qmc_kernel<0><<<grid, kSlabThreads, 0, stream>>>(contracts, qmc, n_contracts, item_prefix, total_items,
                                                         programs, directions, ticket, partials, error_flag);
    else
        qmc_kernel<1><<<grid, kSlabThreads, 0, stream>>>(contracts, qmc, n_contracts, item_prefix, total_items,
                                                         programs, directions, ticket, partials, error_flag);
    return cudaGetLastError();
}

cudaError_t qmc_kernel_occupancy(int precision, int* blocks) {
    return precision == 0 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, qmc_kernel<0>, kSlabThreads, 0)
                          : cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, qmc_kernel<1>, kSlabThreads, 0);
}

cudaError_t launch_sobol_points(const uint32_t* directions, uint32_t dim0, uint32_t n_dims, uint64_t index0,
                                uint64_t n_idx, double* out, cudaStream_t stream) {
    cudaGetLastError();
    const uint64_t total = n_idx * n_dims;
    if (total == 0) return cudaSuccess;
    const uint64_t blocks = (total + 255) / 256;
    sobol_points_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(directions, dim0, n_dims, index0, n_idx,
                                                                           out);
    return cudaGetLastError();
}

}  // namespace mcdg
