// lsm_frozen.cu -- replay of a frozen Longstaff-Schwartz exercise policy,
// streamed: no path storage, one pass, several scenarios per path.
//
// Reference: reprice_against_frozen_policy (src/pricers/lsm.cpp:151-213)
// simulates the paths, seeds the cash flows with the terminal intrinsic and
// walks dates n-1..1 backwards: discount, then exercise where the frozen
// coefficients say so.  With the coefficients fixed, the cash flow a path ends
// with is the exercise value at the EARLIEST date whose test passes (later
// overwrites are earlier dates), or the terminal intrinsic, multiplied by the
// one-date discount once per date before it.  So a path can be priced
// forwards, stopping at its first exercise: the same multiplications in the
// same order give the same bits, and nothing is stored.  Frozen-boundary
// Greeks need the same replay at bumped inputs on the same draws (the
// reference's tests/lsm_test.cpp:138-185 calls the replay at S +/- h): each
// thread carries every scenario's state along one path, sharing the draws.
//
// Work layout, reductions and per-chunk partials are those of the backward
// pass's last date (lsm.cu): chunks of 1024 paths, 256 threads, a fixed
// reduction tree per chunk (FP64 Welford on the FP64 path, compensated FP32
// sums up to the warp on the FP32 path), chunks merged in order per contract
// -- the base scenario reproduces the fitted price bit for bit.
//
// nvcc-flags: --fmad=false
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "lsm.hpp"
#include "lsm_math.cuh"
#include "merge.cuh"

namespace mcdg {

namespace {

__device__ __forceinline__ double intrinsic(double s, double k, int type) {
    const double x = (type == 0 ? 1.0 : -1.0) * (s - k);
    return (x < 0.0) ? 0.0 : x;
}

// Scenarios by volatility: {base, spot+h, spot-h} share the base's GBM step
// constants (and so its growth factors), vol+h and vol-h have their own.
template <int NS>
constexpr int kGroups = NS == 1 ? 1 : 3;
__device__ __forceinline__ constexpr int group_of(int q) { return q < 3 ? 0 : q - 2; }
__device__ __forceinline__ constexpr int group_lead(int gi) { return gi == 0 ? 0 : gi + 2; }
template <int NS>
__device__ __forceinline__ bool group_live(const bool (&live)[NS], int gi) {
    bool any = false;
#pragma unroll
    for (int q = 0; q < NS; ++q) any = any || (group_of(q) == gi && live[q]);
    return any;
}

// One path, NS scenarios: cash flow of each scenario, discounted to t = 0.
template <int NS>
__device__ void replay64(const LsmDev& c, const FrozenDev& f, const LsmReg* __restrict__ rg, uint64_t path,
                         const PhiloxKeys& k, const GlobalTables& tables, double (&v)[NS]) {
    // per volatility group: the log-spot (units of 2^-frac), or the product of
    // growth factors outside the fixed-point range
    int64_t y[kGroups<NS>];
    double growth[kGroups<NS>], s[NS];
    int stop[NS];
    bool live[NS];
#pragma unroll
    for (int gi = 0; gi < kGroups<NS>; ++gi) {
        y[gi] = 0;
        growth[gi] = 1.0;
    }
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        s[q] = f.sc[q].spot;
        stop[q] = c.n_steps;
        live[q] = true;
        v[q] = 0.0;
    }
    const uint32_t path_hi = static_cast<uint32_t>(path >> 32);
    const PhiloxRow row = philox_row(static_cast<uint32_t>(path), 0u, k);
    int n_live = NS;
    for (int d = 0; d < c.n_steps && n_live > 0; ++d) {
        const uint32_t du = static_cast<uint32_t>(d);
        const uint32_t bits = philox_word0(row, philox_step(du, path_hi, k), k);
        const int date = d + 1;
        const bool test = date < c.n_steps && rg[date].has == 1;
        double p[4] = {0.0, 0.0, 0.0, 0.0};
        if (test) {
#pragma unroll
            for (int q = 0; q < 4; ++q) p[q] = rg[date].poly[q];
        }
        if (c.frac > 0) {  // the spot scenarios share the base's growth
            const FixedNormal z = tables.normal(bits);
#pragma unroll
            for (int gi = 0; gi < kGroups<NS>; ++gi) {
                const FrozenScenario& sc = f.sc[group_lead(gi)];
                y[gi] += sc.y_drift + drift_carry(du, sc.y_drift_lo) + scaled_normal(z, sc.y_vs);
                growth[gi] = tables.exp2(y[gi], c.frac);
            }
        } else {
            const double z = normal_from_bits_f64(bits);
#pragma unroll
            for (int gi = 0; gi < kGroups<NS>; ++gi)
                if (group_live<NS>(live, gi)) growth[gi] = exp(f.sc[group_lead(gi)].drift + f.sc[group_lead(gi)].vs * z);
        }
#pragma unroll
        for (int q = 0; q < NS; ++q) {
            if (!live[q]) continue;
            s[q] = (c.frac > 0 ? f.sc[q].spot : s[q]) * growth[group_of(q)];
            if (test) {
                const double ex = intrinsic(s[q], c.strike, c.type);
                if (ex > 0.0 && ex > continuation64(s[q], c.inv_strike, p, tables)) {
                    v[q] = ex;
                    stop[q] = date;
                    live[q] = false;
                    --n_live;
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        if (live[q]) v[q] = intrinsic(s[q], c.strike, c.type);
        for (int t = 0; t < stop[q]; ++t) v[q] *= c.disc;
    }
}

template <int NS>
__device__ void replay32(const LsmDev& c, const FrozenDev& f, const LsmReg* __restrict__ rg, const PhiloxPath& pp,
                         const PhiloxKeys& k, float (&v)[NS]) {
    float x[kGroups<NS>], s[NS];
    int stop[NS];
    bool live[NS];
#pragma unroll
    for (int gi = 0; gi < kGroups<NS>; ++gi) x[gi] = 0.0f;
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        s[q] = f.sc[q].spot_f;
        stop[q] = c.n_steps;
        live[q] = true;
        v[q] = 0.0f;
    }
    const float phi = c.phi_f, strike = c.strike_f, inv_k = c.inv_strike_f;
    int n_live = NS;
    for (int d = 0; d < c.n_steps && n_live > 0; ++d) {
        const float z = normal_from_bits_f32(philox_word0(pp, static_cast<uint32_t>(d), k));
        const int date = d + 1;
        const bool test = date < c.n_steps && rg[date].has == 1;
        float g[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (test) {
            g[0] = rg[date].poly_f[0];
            g[1] = rg[date].poly_f[1];
            g[2] = rg[date].poly_f[2];
            g[3] = rg[date].poly_f[3];
        }
        // the FP32 forward pass's log-space step (lsm.cu, lsm_forward), one
        // log path per volatility group
        float e[kGroups<NS>];
#pragma unroll
        for (int gi = 0; gi < kGroups<NS>; ++gi) {
            e[gi] = 1.0f;
            if (group_live<NS>(live, gi)) {
                const FrozenScenario& g0 = f.sc[group_lead(gi)];
                x[gi] = __fmaf_rn(g0.sg_f, z, x[gi] + g0.mu_f);
                e[gi] = fast_exp(x[gi]);
            }
        }
#pragma unroll
        for (int q = 0; q < NS; ++q) {
            if (!live[q]) continue;
            s[q] = f.sc[q].spot_f * e[group_of(q)];
            if (test) {
                const float ex = phi * (s[q] - strike);
                if (ex > 0.0f && ex > continuation_poly32(s[q], inv_k, g)) {
                    v[q] = ex;
                    stop[q] = date;
                    live[q] = false;
                    --n_live;
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        if (live[q]) v[q] = fmaxf(phi * (s[q] - strike), 0.0f);
        for (int t = 0; t < stop[q]; ++t) v[q] *= c.disc_f;
    }
}

// Per chunk: NS scenario averages (and, for the five-scenario form, the
// per-path central differences of delta, gamma and vega) as Welford partials.
// The FP32 five-scenario form runs 384 threads per SM at most 85 registers
// each (measured 1.3x faster than 512 threads at 106 registers on the 20-put
// grid: paths that exercise early leave the pass latency-bound).
template <int PREC, int NS>
__global__ void __launch_bounds__(kChunkThreads<PREC>, ((PREC == 1 && NS > 1) ? 3 : 2) * (256 / kChunkThreads<PREC>))
    lsm_frozen_stream(const LsmDev* __restrict__ cs, const FrozenDev* __restrict__ fz,
                      const uint32_t* __restrict__ chunk_contract, uint32_t total_chunks,
                      const LsmReg* __restrict__ reg, Welford* __restrict__ part,
                      const FixedTables* __restrict__ fixed) {
    constexpr int NW = NS == 1 ? 1 : kFrozenOutputs;
    __shared__ Welford swf[kLsmThreads64 / 32][NW];
    __shared__ Sum64 s64[NW][kLsmThreads / 32];
    const uint32_t chunk = blockIdx.x;
    if (chunk >= total_chunks) return;
    const uint32_t ci = chunk_contract[chunk];
    const LsmDev c = cs[ci];
    const FrozenDev& f = fz[ci];
    const LsmReg* rg = reg + c.reg_offset;
    const PhiloxKeys k = philox_keys(c.seed);
    const uint32_t local = chunk - c.chunk_begin;
    if constexpr (PREC == 0) {
        Welford w[NW];
#pragma unroll
        for (int q = 0; q < NW; ++q) w[q] = Welford{0ull, 0.0, 0.0};
        for (int j = 0; j < kLsmChunk / kLsmThreads64; ++j) {
            const uint64_t i = static_cast<uint64_t>(local) * kLsmChunk + j * kLsmThreads64 + threadIdx.x;
            if (i >= c.path_count) break;
            double v[NS];
            replay64<NS>(c, f, rg, i, k, GlobalTables{fixed}, v);
#pragma unroll
            for (int q = 0; q < NS; ++q) welford_add(w[q], v[q]);
            if constexpr (NS == kFrozenScenarios) {
                welford_add(w[5], (v[1] - v[2]) * f.inv_2hs);
                welford_add(w[6], ((v[1] - v[0]) - (v[0] - v[2])) * f.inv_hs2);
                welford_add(w[7], (v[3] - v[4]) * f.inv_2hv);
            }
        }
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            const Welford r = welford_warp_reduce(w[q]);
            if ((threadIdx.x & 31) == 0) swf[threadIdx.x >> 5][q] = r;
        }
        __syncthreads();
        if (threadIdx.x < NW) {
            const int q = threadIdx.x;
            Welford m = swf[0][q];
            for (int wi = 1; wi < kLsmThreads64 / 32; ++wi) m = welford_merge(m, swf[wi][q]);
            part[static_cast<uint64_t>(chunk) * NW + q] = m;
        }
    } else {
        // FP32 cash flows; compensated FP32 sums per thread and over the
        // warp tree (Sum32, as the backward pass's last date, so the base
        // scenario keeps its bits), FP64 from the warp sums on.
        Sum32 acc[NW];
#pragma unroll
        for (int q = 0; q < NW; ++q) acc[q] = Sum32{0u, 0.0f, 0.0f, 0.0f, 0.0f};
        for (int j = 0; j < kLsmChunk / kLsmThreads; ++j) {
            const uint64_t i = static_cast<uint64_t>(local) * kLsmChunk + j * kLsmThreads + threadIdx.x;
            if (i >= c.path_count) break;
            float v[NS];
            replay32<NS>(c, f, rg, philox_path(i, 0u, k), k, v);
#pragma unroll
            for (int q = 0; q < NS; ++q) sum32_add(acc[q], v[q]);
            if constexpr (NS == kFrozenScenarios) {
                sum32_add(acc[5], (v[1] - v[2]) * f.inv_2hs_f);
                sum32_add(acc[6], ((v[1] - v[0]) - (v[0] - v[2])) * f.inv_hs2_f);
                sum32_add(acc[7], (v[3] - v[4]) * f.inv_2hv_f);
            }
        }
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            const Sum32 r = sum32_warp_reduce(acc[q]);
            if ((threadIdx.x & 31) == 0) s64[q][threadIdx.x >> 5] = sum32_wide(r);
        }
        __syncthreads();
        if (threadIdx.x < NW)
            part[static_cast<uint64_t>(chunk) * NW + threadIdx.x] = sum64_fold<kLsmThreads / 32>(s64[threadIdx.x]);
    }
}

// The FP32 replay with lanes that move on by themselves (contracts of at most
// kCompactDates dates; the kernel above serves longer ones).  A path ends at its
// last scenario's exercise, so lanes that start together finish far apart: in
// lockstep 18.5 of 32 lanes were active.  Here a lane whose path is done takes
// the chunk's next one, each lane at a date of its own; the dates' Philox words
// and policies are gathered from shared memory.  Finished cash flows wait there
// undiscounted; a second phase discounts and sums them in path order, with the
// operations and the order of the kernel above, so every output keeps its bits.
//
// A date's test is branch-free: with ex = max(intrinsic, 0) a live scenario
// exercises where ex > max(continuation, floor); the floor is 0 at a test date,
// +inf at a date without coefficients, and -1 at maturity, whose polynomial
// makes the continuation -inf, so that every scenario still live ends there.
//
// Bound: issue (73 % of the slots) and the ALU pipe (56 %: selects, minima and
// Philox's XORs), about 180 instructions per path-date with five scenarios.
// 20 puts, 2^20 paths, 50 dates: 11.96 ms in lockstep, 9.2 with a list of paths
// per lane, 7.8 with one list per chunk (25.6 of 32 lanes active); 252 dates is
// what the tables, and a stop in eight bits, hold.
constexpr int kCompactDates = 252;
constexpr int kCompactStride = 4;  // dates between two looks at finished lanes
constexpr int kCompactPaths = kLsmChunk / kLsmThreads;

template <int NS>
__global__ void __launch_bounds__(kLsmThreads, 6)
    lsm_frozen_compact(const LsmDev* __restrict__ cs, const FrozenDev* __restrict__ fz,
                       const uint32_t* __restrict__ chunk_contract, const LsmReg* __restrict__ reg,
                       Welford* __restrict__ part) {
    constexpr int NW = NS == 1 ? 1 : kFrozenOutputs;
    __shared__ PhiloxStep s_step[256];   // date d + 1: Philox words, floor in the fourth
    __shared__ float4 s_poly[256];       // and its polynomial
    __shared__ float s_v[kCompactPaths][NS][kLsmThreads];
    __shared__ uint8_t s_stop[kCompactPaths][NS][kLsmThreads];
    __shared__ Sum64 s64[NW][kLsmThreads / 32];
    __shared__ int s_next;               // next path of the chunk that no lane has taken
    const uint32_t chunk = blockIdx.x, ci = chunk_contract[chunk];
    const LsmDev& c = cs[ci];
    const FrozenDev& f = fz[ci];
    const int t = threadIdx.x, n = c.n_steps;
    if (t == 0) s_next = kLsmThreads;
    const PhiloxKeys k = philox_keys(c.seed);
    const uint64_t base = static_cast<uint64_t>(chunk - c.chunk_begin) * kLsmChunk;
    const float inf = __int_as_float(0x7f800000);
    for (int d = t; d < 256; d += kLsmThreads) {  // dates past maturity repeat it
        PhiloxStep st = philox_step(static_cast<uint32_t>(d), static_cast<uint32_t>(base >> 32), k);
        float4 p = make_float4(-inf, 0.0f, 0.0f, 0.0f);
        float floor = -1.0f;
        if (d + 1 < n) {
            const LsmReg& r = reg[c.reg_offset + d + 1];
            floor = r.has == 1 ? 0.0f : inf;
            if (r.has == 1) p = make_float4(r.poly_f[0], r.poly_f[1], r.poly_f[2], r.poly_f[3]);
        }
        st.carry = __float_as_uint(floor);
        s_step[d] = st;
        s_poly[d] = p;
    }
    __syncthreads();
    const uint64_t left = c.path_count - base;
    const int in_chunk = static_cast<int>(left < kLsmChunk ? left : kLsmChunk);
    const int mine = in_chunk > t ? (in_chunk - t + kLsmThreads - 1) / kLsmThreads : 0;  // this thread's paths
    const float phi = c.phi_f, pk = -c.phi_f * c.strike_f, inv_k = c.inv_strike_f;
    float mu[kGroups<NS>], sg[kGroups<NS>], spot[NS];
#pragma unroll
    for (int gi = 0; gi < kGroups<NS>; ++gi) {
        mu[gi] = f.sc[group_lead(gi)].mu_f;
        sg[gi] = f.sc[group_lead(gi)].sg_f;
    }
#pragma unroll
    for (int q = 0; q < NS; ++q) spot[q] = f.sc[q].spot_f;

    constexpr uint32_t kAll = (1u << NS) - 1u;
    int at = t, d = 0;  // this lane's path within the chunk, its next date's index
    uint32_t live = kAll;
    float x[kGroups<NS>], v[NS];
    int stop[NS];
#pragma unroll
    for (int gi = 0; gi < kGroups<NS>; ++gi) x[gi] = 0.0f;
    PhiloxRow row = philox_row(static_cast<uint32_t>(base) + t, 0u, k);
    while (at < in_chunk) {
#pragma unroll 1
        for (int u = 0; u < kCompactStride; ++u) {
            const PhiloxStep st = s_step[d];
            const float4 p4 = s_poly[d];
            const float p[4] = {p4.x, p4.y, p4.z, p4.w};
            const float floor = __uint_as_float(st.carry);
            const float z = normal_from_bits_f32(philox_word0(row, st, k));
            ++d;
            float e[kGroups<NS>];
#pragma unroll
            for (int gi = 0; gi < kGroups<NS>; ++gi) {
                x[gi] = __fmaf_rn(sg[gi], z, x[gi] + mu[gi]);
                e[gi] = fast_exp(x[gi]);
            }
#pragma unroll
            for (int q = 0; q < NS; ++q) {
                const float s = spot[q] * e[group_of(q)];
                const float ex = fmaxf(__fmaf_rn(phi, s, pk), 0.0f);  // phi (s - strike), one rounding either way
                const bool hit = (live >> q & 1u) != 0u && ex > fmaxf(continuation_poly32(s, inv_k, p), floor);
                v[q] = hit ? ex : v[q];
                stop[q] = hit ? d : stop[q];
                live = hit ? live & ~(1u << q) : live;
            }
        }
        if (live == 0u) {
#pragma unroll
            for (int q = 0; q < NS; ++q) {
                s_v[at / kLsmThreads][q][at % kLsmThreads] = v[q];
                s_stop[at / kLsmThreads][q][at % kLsmThreads] = static_cast<uint8_t>(stop[q]);
            }
            at = atomicAdd(&s_next, 1);
            d = 0;
            live = kAll;
#pragma unroll
            for (int gi = 0; gi < kGroups<NS>; ++gi) x[gi] = 0.0f;
            row = philox_row(static_cast<uint32_t>(base) + at, 0u, k);
        }
    }
    __syncthreads();
    const float disc = c.disc_f;
    Sum32 acc[NW];
#pragma unroll
    for (int q = 0; q < NW; ++q) acc[q] = Sum32{0u, 0.0f, 0.0f, 0.0f, 0.0f};
    for (int j = 0; j < mine; ++j) {
        int first = 255;
#pragma unroll
        for (int q = 0; q < NS; ++q) {
            v[q] = s_v[j][q][t];
            stop[q] = s_stop[j][q][t];
            first = min(first, stop[q]);
        }
        // one multiplication per date: all scenarios up to the earliest stop,
        // then each on its own (most stop within a few dates of one another)
#pragma unroll 4
        for (int i = 0; i < first; ++i) {
#pragma unroll
            for (int q = 0; q < NS; ++q) v[q] *= disc;
        }
#pragma unroll
        for (int q = 0; q < NS; ++q)
            for (int i = first; i < stop[q]; ++i) v[q] *= disc;
#pragma unroll
        for (int q = 0; q < NS; ++q) sum32_add(acc[q], v[q]);
        if constexpr (NS == kFrozenScenarios) {
            sum32_add(acc[5], (v[1] - v[2]) * f.inv_2hs_f);
            sum32_add(acc[6], ((v[1] - v[0]) - (v[0] - v[2])) * f.inv_hs2_f);
            sum32_add(acc[7], (v[3] - v[4]) * f.inv_2hv_f);
        }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < NW; ++q) {
        const Sum32 r = sum32_warp_reduce(acc[q]);
        if ((t & 31) == 0) s64[q][t >> 5] = sum32_wide(r);
    }
    __syncthreads();
    if (t < NW) part[static_cast<uint64_t>(chunk) * NW + t] = sum64_fold<kLsmThreads / 32>(s64[t]);
}

// One CTA per (contract, output), the merge of lsm_finish: mean, standard
// error, count.
__global__ void __launch_bounds__(kMergeThreads)
    lsm_frozen_finish(const LsmDev* __restrict__ cs, const Welford* __restrict__ part, double* __restrict__ out) {
    const int ci = blockIdx.x, q = blockIdx.y, nw = gridDim.y;
    const LsmDev& c = cs[ci];
    const MergedResult m = merge_items(part + static_cast<size_t>(c.chunk_begin) * nw + q, c.n_chunks, nw);
    if (threadIdx.x != 0) return;
    double* o = out + (static_cast<size_t>(ci) * nw + q) * 3;
    o[0] = m.mean;
    o[1] = m.standard_error;
    o[2] = static_cast<double>(m.count);
}

}  // namespace

cudaError_t launch_lsm_frozen(int precision, int n_scenarios, int max_steps, const LsmDev* c, const FrozenDev* f,
                              int n_contracts, const uint32_t* chunk_contract, uint32_t total_chunks,
                              const LsmReg* reg, Welford* partials, double* out, const FixedTables* tables,
                              cudaStream_t stream) {
    cudaGetLastError();
    if (n_scenarios != 1 && n_scenarios != kFrozenScenarios) return cudaErrorInvalidValue;
    if (total_chunks) {
        const bool five = n_scenarios == kFrozenScenarios;
        if (precision == 0) {
            if (five) lsm_frozen_stream<0, kFrozenScenarios><<<total_chunks, kLsmThreads64, 0, stream>>>(c, f, chunk_contract, total_chunks, reg, partials, tables);
            else lsm_frozen_stream<0, 1><<<total_chunks, kLsmThreads64, 0, stream>>>(c, f, chunk_contract, total_chunks, reg, partials, tables);
        } else if (max_steps <= kCompactDates) {
            if (five) lsm_frozen_compact<kFrozenScenarios><<<total_chunks, kLsmThreads, 0, stream>>>(c, f, chunk_contract, reg, partials);
            else lsm_frozen_compact<1><<<total_chunks, kLsmThreads, 0, stream>>>(c, f, chunk_contract, reg, partials);
        } else {
            if (five) lsm_frozen_stream<1, kFrozenScenarios><<<total_chunks, kLsmThreads, 0, stream>>>(c, f, chunk_contract, total_chunks, reg, partials, tables);
            else lsm_frozen_stream<1, 1><<<total_chunks, kLsmThreads, 0, stream>>>(c, f, chunk_contract, total_chunks, reg, partials, tables);
        }
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    const int nw = n_scenarios == 1 ? 1 : kFrozenOutputs;
    if (n_contracts > 0) lsm_frozen_finish<<<dim3(n_contracts, nw), kMergeThreads, 0, stream>>>(c, partials, out);
    return cudaGetLastError();
}

}  // namespace mcdg
