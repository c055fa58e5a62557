// heston.cu -- Heston QE paths priced against many strikes in one pass.
//
// Reference: heston_qe_european (src/pricers/heston.cpp:120-156) with the
// Andersen QE variance step (:91-116, psi_c = 1.5) and the K0..K4 log-spot
// update (gamma1 = gamma2 = 1/2, :125-129).  Each (path, step) consumes the
// stream-0 normal for the spot and the stream-1 uniform for the variance,
// both keyed (seed, path, step) exactly as the reference.
//
// The reference prices one strike per call; calling it for K strikes with one
// seed re-simulates identical paths K times (common random numbers).  Here a
// path is simulated once and its terminal spot is paid out against all K
// strikes, which gives the same K results (to rounding) for 1/K of the
// simulation work.
//
// Work items are (parameter set, 4096-path slab).  A CTA of 128 threads
// simulates one path per thread per round (32 rounds per slab), stages the
// terminal values in shared memory, then pays them out: thread t serves
// strike t % K over the paths of group t / K (G = 128 / K groups), so every
// thread is busy when K <= 128; for 128 < K <= 256, thread t serves strikes t
// and t + 128 over all paths.  FP32 payoffs are summed per round with Kahan
// compensation, then added in FP64; the groups and slabs are merged in fixed
// order.  (The FP64 paths are heston64.cu.)
//
// Bound: issue (68 % of the slots) and the FMA-heavy pipe (69 %), 158
// thread-instructions per path-step.  64 sets of 64 strikes, 252 steps, 2^20
// paths: 110 ms -> 106 with the Philox products of the draw and of the path
// taken out of the step, 100-104 with one branch region for both paths'
// exponential steps, 97.5 at 5 CTAs per SM with every subnormal flushed, 0.7 %
// more with the exponential and logarithm alone doing so (fp32_fast.cuh).
//
// nvcc-flags: --fmad=false
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "heston.hpp"
#include "merge.cuh"

namespace mcdg {

namespace {

// FP32 QE step of two paths: the reference's scheme, 1-u formed from the bits.
// z holds the normals of the same bits.  Both paths take the quadratic branch's
// value, then one branch for the pair replaces it where psi > 1.5: in most
// warps some lane has such a path, and a branch region per path would run both
// sides one after the other.
__device__ __forceinline__ void qe_pair32(const float (&v)[2], const HestonSet32& h, const uint32_t (&ubits)[2],
                                          const float (&z)[2], float (&out)[2]) {
    float m[2], psi[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        m[i] = __fmaf_rn(v[i] - h.theta, h.e, h.theta);
        const float s2 = __fmaf_rn(v[i], h.s2_lin, h.s2_const);
        psi[i] = s2 * fast_rcp(m[i] * m[i]);
        const float inv_psi = fast_rcp(psi[i]);
        const float two = 2.0f * inv_psi;
        const float b2 = two - 1.0f + fast_sqrt(two) * fast_sqrt(two - 1.0f);
        const float a = m[i] * fast_rcp(1.0f + b2);
        const float bz = fast_sqrt(b2) + z[i];
        out[i] = a * bz * bz;
    }
    if (!(psi[0] <= 1.5f) || !(psi[1] <= 1.5f)) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float p = (psi[i] - 1.0f) * fast_rcp(psi[i] + 1.0f);
            const float u = uniform_from_bits_f32(ubits[i]);
            // 1 - u = (~bits + 0.5) / 2^32, exact relative precision near u = 1
            const float one_minus_u = __fmaf_rn(__uint2float_rn(~ubits[i]), 2.3283064365386963e-10f,
                                                1.1641532182693481e-10f);
            const float beta = (1.0f - p) * fast_rcp(m[i]);
            const float e = fast_log((1.0f - p) * fast_rcp(one_minus_u)) * fast_rcp(beta);
            if (!(psi[i] <= 1.5f)) out[i] = u <= p ? 0.0f : e;
        }
    }
}

struct KahanF {
    float s = 0.0f, c = 0.0f;
    __device__ __forceinline__ void add(float x) {
        const float y = x - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
};

// Two paths per thread in flight, 5 CTAs of 128 threads per SM (92 registers): 64
// sets of 2^20 paths and 252 steps at 3, 4, 5, 6, 7, 8 CTAs: 107.7, 99.7, 97.5,
// 99.9, 104.4, 105.8 ms.
__global__ void __launch_bounds__(128, 5)
    heston_kernel(const HestonSet* __restrict__ sets, const double* __restrict__ strikes,
                  int n_strikes, int type, uint32_t items_per_set, uint32_t total_items,
                  uint32_t* __restrict__ ticket, Welford* __restrict__ partials) {
    __shared__ uint32_t s_item;
    __shared__ float s_terminal32[128], s_terminal32b[128];
    __shared__ Welford s_acc[256];
    __shared__ HestonSet s_set;
    __shared__ PhiloxStep s_step[kStepTable];
    const int t = threadIdx.x;
    const int groups = n_strikes <= 128 ? 128 / n_strikes : 1;
    const int my_group = n_strikes <= 128 ? t / n_strikes : 0;
    const int k0 = n_strikes <= 128 ? t % n_strikes : t;
    const bool serves0 = (n_strikes <= 128) ? (my_group < groups) : (k0 < n_strikes);
    const bool serves1 = n_strikes > 128 && (t + 128) < n_strikes;
    const double phi = type == 0 ? 1.0 : -1.0;
    for (;;) {
        if (t == 0) s_item = atomicAdd(ticket, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= total_items) return;
        const int set = static_cast<int>(item / items_per_set);
        const uint32_t slab = item % items_per_set;
        static_assert(sizeof(HestonSet) % 4 == 0 && sizeof(HestonSet) / 4 <= 128, "one word per thread");
        if (t < static_cast<int>(sizeof(HestonSet) / 4))
            reinterpret_cast<uint32_t*>(&s_set)[t] = reinterpret_cast<const uint32_t*>(&sets[set])[t];
        __syncthreads();
        const HestonSet& h = s_set;
        const PhiloxKeys k = philox_keys(h.seed);
        const uint64_t base = static_cast<uint64_t>(slab) * 4096;
        const uint32_t path_hi = static_cast<uint32_t>(base >> 32);
        const bool once = h.n_steps <= kStepTable;  // the step table serves the whole slab
        if (once) {
            fill_steps(s_step, 0, path_hi, k);
            __syncthreads();
        }
        const double strike0 = serves0 ? strikes[k0] : 0.0;
        const double strike1 = serves1 ? strikes[t + 128] : 0.0;
        unsigned cnt0 = 0, cnt1 = 0;
        double a0 = 0.0, q0 = 0.0, a1 = 0.0, q1 = 0.0;
        const HestonSet32 h32 = make_set32(h);
        {
            // Two rounds per pass: each thread simulates the paths of rounds j
            // and j + 1 together (independent dependency chains), then both
            // rounds are paid out in order, so the sums are those of one round
            // at a time.
            const float fphi = static_cast<float>(phi);
            const float fk0 = static_cast<float>(strike0), fk1 = static_cast<float>(strike1);
            auto payout = [&](int j, const float* terminal) {
                const uint64_t round_base = static_cast<uint64_t>(slab) * 4096 + static_cast<uint64_t>(j * 128);
                const uint64_t left = round_base >= h.path_count ? 0 : h.path_count - round_base;
                const int round_live = left > 128 ? 128 : static_cast<int>(left);
                KahanF s0a, s0b, s1a, s1b;
                unsigned n_here = 0;
                for (int p = my_group; p < round_live; p += groups) {
                    const float s_t = terminal[p];
                    const float y0 = fmaxf(fphi * (s_t - fk0), 0.0f);
                    s0a.add(y0);
                    s0b.add(y0 * y0);
                    if (serves1) {
                        const float y1 = fmaxf(fphi * (s_t - fk1), 0.0f);
                        s1a.add(y1);
                        s1b.add(y1 * y1);
                    }
                    ++n_here;
                }
                if (serves0) {
                    cnt0 += n_here;
                    a0 += static_cast<double>(s0a.s) + static_cast<double>(-s0a.c);
                    q0 += static_cast<double>(s0b.s) + static_cast<double>(-s0b.c);
                }
                if (serves1) {
                    cnt1 += n_here;
                    a1 += static_cast<double>(s1a.s) + static_cast<double>(-s1a.c);
                    q1 += static_cast<double>(s1b.s) + static_cast<double>(-s1b.c);
                }
            };
            for (int j = 0; j < 32; j += 2) {
                const uint64_t path_a = base + static_cast<uint64_t>(j * 128 + t);
                // (a table refill is a CTA barrier: every thread then runs every round)
                if (path_a < h.path_count || !once) {
                    const uint32_t lo = static_cast<uint32_t>(path_a);
                    const PhiloxRow ra = philox_row(lo, 0u, k), rb = philox_row(lo + 128, 0u, k);
                    const PhiloxRow ua = philox_row(lo, 1u, k), ub = philox_row(lo + 128, 1u, k);
                    float v[2] = {h32.v0, h32.v0}, x[2] = {0.0f, 0.0f};  // variance, ln(S/S0)
                    for (int d0 = 0; d0 < h.n_steps; d0 += kStepTable) {
                        if (!once) {
                            __syncthreads();
                            fill_steps(s_step, d0, path_hi, k);
                            __syncthreads();
                        }
                        const int m = min(kStepTable, h.n_steps - d0);
                        for (int d = 0; d < m; ++d) {
                            const PhiloxStep st = s_step[d];
                            const uint32_t bits[4] = {philox_word0(ra, st, k), philox_word0(rb, st, k),
                                                      philox_word0(ua, st, k), philox_word0(ub, st, k)};
                            float z[4], next[2];
                            normals_from_bits_f32<4>(bits, z);
                            const uint32_t ubits[2] = {bits[2], bits[3]};
                            const float zv[2] = {z[2], z[3]};
                            qe_pair32(v, h32, ubits, zv, next);
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                const float dv = fmaxf(__fmaf_rn(h32.k3, v[i], h32.k4 * next[i]), 0.0f);
                                const float inc = __fmaf_rn(h32.k1, v[i], __fmaf_rn(h32.k2, next[i], h32.c0));
                                x[i] = __fmaf_rn(fast_sqrt(dv), z[i], x[i] + inc);
                                v[i] = next[i];
                            }
                        }
                    }
                    s_terminal32[t] = h32.s0 * __expf(x[0]);
                    s_terminal32b[t] = h32.s0 * __expf(x[1]);
                }
                __syncthreads();
                payout(j, s_terminal32);
                payout(j + 1, s_terminal32b);
                __syncthreads();
            }
        }
        // discount applied once: mean scales by D, M2 by D^2
        const double disc = h.discount;
        const Welford w0 = welford_from_sums(cnt0, a0 * disc, q0 * disc * disc);
        const Welford w1 = welford_from_sums(cnt1, a1 * disc, q1 * disc * disc);
        // Merge the groups of each strike in group order (fixed tree).
        if (serves0) s_acc[n_strikes <= 128 ? my_group * n_strikes + k0 : k0] = w0;
        if (serves1) s_acc[t + 128] = w1;
        __syncthreads();
        if (n_strikes <= 128) {
            if (t < n_strikes) {
                Welford m = s_acc[t];
                for (int g = 1; g < groups; ++g) m = welford_merge(m, s_acc[g * n_strikes + t]);
                partials[static_cast<size_t>(item) * n_strikes + t] = m;
            }
        } else {
            for (int kk = t; kk < n_strikes; kk += 128)
                partials[static_cast<size_t>(item) * n_strikes + kk] = s_acc[kk];
        }
        __syncthreads();
    }
}

// One CTA per (set, strike).
__global__ void __launch_bounds__(kMergeThreads)
    heston_merge_kernel(int n_strikes, uint32_t items_per_set, const Welford* __restrict__ partials,
                        double* __restrict__ out /* n_sets*n_strikes x {price, se, count} */) {
    const size_t w = blockIdx.x, set = w / n_strikes, strike = w % n_strikes;
    const MergedResult m = merge_items(partials + set * items_per_set * n_strikes + strike, items_per_set, n_strikes);
    if (threadIdx.x == 0) {
        out[3 * w] = m.mean;
        out[3 * w + 1] = m.standard_error;
        reinterpret_cast<unsigned long long*>(out)[3 * w + 2] = m.count;
    }
}

}  // namespace

cudaError_t launch_heston32(int grid, const HestonSet* sets, int n_sets, const double* strikes, int n_strikes,
                            int type, uint32_t items_per_set, uint32_t* ticket, Welford* partials,
                            cudaStream_t stream) {
    cudaGetLastError();
    heston_kernel<<<grid, 128, 0, stream>>>(sets, strikes, n_strikes, type, items_per_set,
                                            items_per_set * static_cast<uint32_t>(n_sets), ticket, partials);
    return cudaGetLastError();
}

cudaError_t launch_heston_merge(int n_sets, int n_strikes, uint32_t items_per_set, const Welford* partials,
                                double* out, cudaStream_t stream) {
    cudaGetLastError();
    heston_merge_kernel<<<static_cast<unsigned>(n_sets) * n_strikes, kMergeThreads, 0, stream>>>(
        n_strikes, items_per_set, partials, out);
    return cudaGetLastError();
}

cudaError_t heston32_occupancy(int* blocks) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, heston_kernel, 128, 0);
}

}  // namespace mcdg
