// lsm.cu -- batched Longstaff-Schwartz American pricing (QR regression).
//
// Reference: monte_carlo_lsm_american (src/pricers/lsm.cpp:62-149; the frozen
// replay of :151-213 is the streaming kernel of lsm_frozen.cu): forward-simulated
// GBM paths, cash flows seeded with the terminal intrinsic, backward over dates
// n-1..1 (discount
// the cash flows, regress them on the weighted Laguerre basis of S/K over the
// in-the-money paths -- skipped below 4 such paths --, exercise where
// intrinsic > continuation), a final discount, Welford, and the inception check.
//
// Layout.  Every contract's paths live in HBM for the whole backward pass,
// date-major (S[d-1][i], coalesced per date for the forward stores and the
// backward column reads), FP32 or FP64; cash flows likewise.  Paths are cut
// into fixed chunks of 1024 (the reduction unit); a chunk is one CTA of 128
// threads (FP32, 8 paths per thread) or 256 (FP64, 4 paths per thread).
//
// Backward pass.  All contracts of a batch step back in lockstep: iteration k
// handles date e = n_c - k of contract c, in one pass over the date's columns
// (lsm_step): exercise at date e with that date's coefficients, discount, and
// either the regression sums of date e-1 -- Gram matrix and right-hand side
// in the basis b T_e, T_e being date e's preconditioner (adjacent dates'
// in-the-money populations are alike, so b T_e is already close to
// orthonormal on date e-1) -- or, when e = 1, the final Welford partial.  The
// last CTA of a contract to finish folds the chunk partials in chunk order
// and solves date e-1 (no separate launch; no CTA waits for another): the
// Cholesky factor R of the lagged Gram matrix gives date e-1's own
// preconditioner T = T_e R^{-1}; when that matrix is well conditioned the 4x4
// Householder solve of the preconditioned normal equations gives the
// coefficients at once.  Otherwise -- always on the first regression date,
// whose lag is the identity (cond of the raw Laguerre Gram matrix reaches
// ~4e12) -- lsm_refine makes a second pass in the basis b T and solves it:
// Cholesky-QR2 for that date.  Either way the coefficients agree with the
// reference's Householder QR to the limit set by the least-squares
// conditioning (its own algorithm moves them that much when the rows are
// reordered), and the fitted continuation values, hence the exercise
// decisions, coincide.  Every reduction tree is fixed by chunk index.
// Precision: the FP64 path keeps FP64 accuracy throughout (paths in fixed point,
// fused products, e^{-x/2} from the fixed-point tables).  The
// FP32 path evaluates the basis, the exercise tests and the Gram products in
// FP32 (FP64 runs at a small fraction of the FP32 rate here), keeps the cash
// flows and continuation values in FP32 and accumulates the Gram products
// with compensated FP32 sums per chunk (per thread, then one warp per sum
// over the chunk's threads); the final payoffs are summed in compensated
// FP32 per thread and over the warp tree (Sum32); warp sums, chunk partials
// and the Cholesky-QR2 solves are FP64.  (The FP32 discount factor
// carries a relative error below 3e-8 per date, a bias under 2e-6 of the
// price after 50 dates.)
//
// Bound of a single FP64 contract: the chain of dates.  Per date of a put with
// 131,072 paths and 50 dates: 92 us before; the FP64 pipe (about 150 -> 41
// operations per path) and the tail (folds by transposed warp sums, the 4x4
// algebra one element per lane: an FP64 operation holds a scheduler for 64
// cycles with one lane or 32) -> 37 us; every date in one launch with the cash
// flows and basis values kept on the SM (lsm_chain64) and in-the-money paths
// packed before the products -> 17 us.  Forward simulation of that put 2.9 ms
// -> 55 us (one warp per 32 paths instead of 8 paths per thread in 128 CTAs).
// The call 7.35 -> 1.92 -> 1.0 ms.  FP32 pass of two contracts 62 -> 28 us, of
// ten 100 -> 70 us.
//
// nvcc-flags: --fmad=false
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "fp64_fast.cuh"
#include "lsm.hpp"
#include "lsm_math.cuh"
#include "merge.cuh"
#include "paths64.cuh"

namespace mcdg {

namespace {

// FP32 path: the same basis evaluated in FP32.  FP64 arithmetic runs at a
// small fraction of the FP32 rate on this GPU, and with FP32 paths the basis
// carries FP32 inputs anyway; the regression is fitted to exactly this
// evaluated basis and the sums that need the range stay compensated (below).
__device__ __forceinline__ float sixth(float x) {  // x / 6, correctly rounded (Markstein), without the division's slow path
    constexpr float y = 1.0f / 6.0f;
    const float q = x * y;
    return __fmaf_rn(__fmaf_rn(-6.0f, q, x), y, q);
}
__device__ __forceinline__ void basis32(float s, float inv_strike, bool use, float b[4]) {  // use: else zeros
    const float x = s * inv_strike;
    const float e = use ? fast_exp(-0.5f * x) : 0.0f;
    b[0] = e;
    b[1] = e * (1.0f - x);
    b[2] = e * __fmaf_rn(0.5f * x, x, __fmaf_rn(-2.0f, x, 1.0f));
    b[3] = e * __fmaf_rn(__fmaf_rn(-sixth(x), x, 1.5f * x), x, __fmaf_rn(-3.0f, x, 1.0f));
}

// Compensated FP32 accumulation (Knuth's TwoSum): hi + lo carries ~44 bits,
// enough for Gram sums of a chunk; chunk partials are then merged in FP64.
__device__ __forceinline__ void df_add(float& hi, float& lo, float x) {
    const float s = hi + x;
    const float bp = s - hi;
    lo += (hi - (s - bp)) + (x - bp);
    hi = s;
}

// Fixed-shape block reduction of N compensated sums (256 threads): every
// thread's (hi, lo) pairs go to shared memory, then warp w folds sums w,
// w + 8, ...: lane l takes threads l, l + 32, ..., l + 224 in that order
// (compensated), then a compensated shuffle tree; the FP64 value hi + lo of
// each sum lands in res.
template <int N>
__device__ void block_sum_df(const float (&hi)[N], const float (&lo)[N], float2 (*scratch)[kLsmThreads],
                             double* res) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll
    for (int i = 0; i < N; ++i) scratch[i][t] = make_float2(hi[i], lo[i]);
    __syncthreads();
    for (int i = warp; i < N; i += kLsmThreads / 32) {
        float h = 0.0f, l = 0.0f;
#pragma unroll
        for (int u = 0; u < kLsmThreads / 32; ++u) {
            const float2 v = scratch[i][lane + 32 * u];
            df_add(h, l, v.x);
            l += v.y;
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            const float oh = __shfl_down_sync(0xffffffffu, h, off);
            const float ol = __shfl_down_sync(0xffffffffu, l, off);
            df_add(h, l, oh);
            l += ol;
        }
        if (lane == 0) res[i] = static_cast<double>(h) + static_cast<double>(l);
    }
    __syncthreads();
}

// Chunk reduction of plain FP32 per-thread sums (the FP32 step's sums in a
// well-conditioned basis): thread partials go to shared memory, warp w folds
// sums w, w + W, ... (W warps): lane l adds threads l, l + 32, ... in that
// order, then a shuffle tree; lane 0 widens the chunk's sum to FP64 in res.
// FP32 up to the chunk (1024 paths), FP64 above.
template <int N>
__device__ void block_sum_f32(const float (&v)[N], float (*scratch)[kLsmThreads], double* res) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll
    for (int i = 0; i < N; ++i) scratch[i][t] = v[i];
    __syncthreads();
    for (int i = warp; i < N; i += kLsmThreads / 32) {
        float x = scratch[i][lane];
#pragma unroll
        for (int u = 1; u < kLsmThreads / 32; ++u) x += scratch[i][lane + 32 * u];
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
        if (lane == 0) res[i] = static_cast<double>(x);
    }
    __syncthreads();
}

// The 15 sums of a chunk or fold over a warp, transposed: each step halves the
// values a lane carries (16 additions instead of 75; an FP64 operation holds a
// scheduler for 64 cycles, however many lanes are active).  The additions of
// one value pair the lanes of a shuffle tree, so the bits are the tree's.
// Lanes 2 i return sum i.
__device__ __forceinline__ double warp_sums15(const double (&v)[15]) {
    const int lane = threadIdx.x & 31;
    const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4, h2 = lane & 2;
    auto at = [&](int i) { return i < 15 ? v[i < 15 ? i : 0] : 0.0; };
    double a[8], b[4], c[2];
#pragma unroll
    for (int i = 0; i < 8; ++i)
        a[i] = (h16 ? at(i + 8) : at(i)) + __shfl_xor_sync(0xffffffffu, h16 ? at(i) : at(i + 8), 16);
#pragma unroll
    for (int i = 0; i < 4; ++i)
        b[i] = (h8 ? a[i + 4] : a[i]) + __shfl_xor_sync(0xffffffffu, h8 ? a[i] : a[i + 4], 8);
#pragma unroll
    for (int i = 0; i < 2; ++i)
        c[i] = (h4 ? b[i + 2] : b[i]) + __shfl_xor_sync(0xffffffffu, h4 ? b[i] : b[i + 2], 4);
    const double d = (h2 ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, h2 ? c[0] : c[1], 2);
    return d + __shfl_xor_sync(0xffffffffu, d, 1);
}

// Fixed-shape block reduction of the 15 sums of the first `warps` warps (the
// others hold zeros): warp trees, then the warps in order.  Result in res for
// every thread after the closing barrier.
__device__ __forceinline__ void block_sum15(const double (&v)[15], int warps, double (*smem)[15], double* res) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < warps) {
        const double x = warp_sums15(v);
        // lane = 16 b3 + 8 b2 + 4 b1 + 2 b0 holds sum b3 b2 b1 b0
        if ((lane & 1) == 0 && lane < 30) smem[warp][lane >> 1] = x;
    }
    __syncthreads();
    if (threadIdx.x < 15) {
        double x = smem[0][threadIdx.x];
        for (int w = 1; w < warps; ++w) x += smem[w][threadIdx.x];
        res[threadIdx.x] = x;
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// forward simulation (src/pricers/lsm.cpp:35-58), date-major stores
// ---------------------------------------------------------------------------
// FP64: one warp per 32 paths, the fixed-point tables shared by the SM's one
// CTA; every warp takes every (number of warps)-th unit.
struct ForwardSlot {
    LsmDev c;
    PhiloxStep step[32];
};
struct ForwardShared {
    FixedShared tables;
    ForwardSlot slot[32];
};

__global__ void __launch_bounds__(1024, 1)
    lsm_forward64(const LsmDev* __restrict__ cs, const uint32_t* __restrict__ chunk_contract, uint32_t chunk_first,
                  uint32_t chunk_end, double* __restrict__ store, const FixedTables* __restrict__ t) {
    extern __shared__ __align__(16) unsigned char smem[];
    ForwardShared& sh = *reinterpret_cast<ForwardShared*>(smem);
    load_fixed_tables(sh.tables, t);
    const FixedShared& s = sh.tables;
    const int lane = threadIdx.x & 31;
    ForwardSlot& slot = sh.slot[threadIdx.x >> 5];
    const LsmDev& c = slot.c;
    constexpr uint32_t kUnits = kLsmChunk / 32;  // units of a chunk
    const uint64_t units = static_cast<uint64_t>(chunk_end - chunk_first) * kUnits;
    uint32_t have = 0xFFFFFFFFu;
    for (uint64_t u = static_cast<uint64_t>(threadIdx.x >> 5) * gridDim.x + blockIdx.x; u < units; u += 32ull * gridDim.x) {
        const uint32_t chunk = chunk_first + static_cast<uint32_t>(u / kUnits), ci = chunk_contract[chunk];
        if (ci != have) {
            have = ci;
            __syncwarp();
            copy_words(&slot.c, &cs[ci]);
            __syncwarp();
        }
        const uint64_t base = static_cast<uint64_t>(chunk - c.chunk_begin) * kLsmChunk + (u % kUnits) * 32;
        const uint64_t i = base + lane;
        const bool live = i < c.path_count;
        double* out = store + c.s_offset + i;
        const PhiloxKeys k = philox_keys(c.seed);
        const PhiloxRow row = philox_row(static_cast<uint32_t>(i), 0u, k);
        int64_t y = 0;
        double spot = c.spot;
        for (int d0 = 0; d0 < c.n_steps; d0 += 32) {
            __syncwarp();
            PhiloxStep st = philox_step(static_cast<uint32_t>(d0 + lane), static_cast<uint32_t>(base >> 32), k);
            st.carry = drift_carry(static_cast<uint32_t>(d0 + lane), c.y_drift_lo);
            slot.step[lane] = st;
            __syncwarp();
            const int n = min(32, c.n_steps - d0);
            for (int d = 0; d < n; ++d) {
                const PhiloxStep w = slot.step[d];
                const uint32_t bits = philox_word0(row, w, k);
                if (c.frac > 0) {  // as LsmState64
                    y += c.y_drift + w.carry + scaled_normal(normal_fixed(bits, s, t), c.y_vs);
                    spot = c.spot * exp2_units(y, c.frac, s);
                } else {
                    spot = spot * exp(c.drift + c.vs * normal_from_bits_f64(bits));
                }
                if (live) *out = spot;
                out += c.path_count;
            }
        }
    }
}

// Two paths from table step 0 to n, from log-spots x, storing S0 e^x per date.
__device__ __forceinline__ void forward_pair32(const PhiloxStep* table, int n, const PhiloxKeys& k, uint32_t path_lo,
                                               float mu, float sg, float s0, uint64_t column, bool both,
                                               float (&x)[2], float* __restrict__ out) {
    const PhiloxRow row[2] = {philox_row(path_lo, 0u, k), philox_row(path_lo + kLsmThreads, 0u, k)};
    for (int d = 0; d < n; ++d) {
        const PhiloxStep st = table[d];
        const uint32_t bits[2] = {philox_word0(row[0], st, k), philox_word0(row[1], st, k)};
        float z[2];
        normals_from_bits_f32<2>(bits, z);
        x[0] = gbm_log_step_f32(x[0], z[0], mu, sg);
        x[1] = gbm_log_step_f32(x[1], z[1], mu, sg);
        out[0] = gbm_spot_f32(s0, x[0]);
        if (both) out[kLsmThreads] = gbm_spot_f32(s0, x[1]);
        out += column;  // one column per date
    }
}

// FP32: one CTA per chunk, two paths per thread at a time (independent Philox
// chains), the step table of the path engine.  A contract of more dates than
// the table holds keeps its chunk's log-spots in shared memory between refills.
__global__ void __launch_bounds__(kLsmThreads, 8)
    lsm_forward32(const LsmDev* __restrict__ cs, const uint32_t* __restrict__ chunk_contract, uint32_t chunk_first,
                  uint32_t chunk_end, float* __restrict__ store) {
    __shared__ PhiloxStep s_step[kStepTable];
    __shared__ float s_x[kLsmChunk];
    const uint32_t chunk = chunk_first + blockIdx.x;
    if (chunk >= chunk_end) return;
    const LsmDev& c = cs[chunk_contract[chunk]];
    const PhiloxKeys k = philox_keys(c.seed);
    const float mu = static_cast<float>(c.drift), sg = static_cast<float>(c.vs), s0 = static_cast<float>(c.spot);
    const uint64_t base = static_cast<uint64_t>(chunk - c.chunk_begin) * kLsmChunk, paths = c.path_count;
    float* S = store + c.s_offset;
    const int n = c.n_steps;
    for (int d0 = 0; d0 < n; d0 += kStepTable) {
        if (d0 > 0) __syncthreads();
        fill_steps(s_step, d0, static_cast<uint32_t>(base >> 32), k);
        __syncthreads();
        const int m = min(kStepTable, n - d0);
        for (int j = 0; j < kLsmChunk; j += 2 * kLsmThreads) {
            const int at = j + threadIdx.x;
            const uint64_t i = base + at;
            if (i >= paths) break;
            float x[2] = {0.0f, 0.0f};
            if (d0 > 0) {
                x[0] = s_x[at];
                x[1] = s_x[at + kLsmThreads];
            }
            forward_pair32(s_step, m, k, static_cast<uint32_t>(i), mu, sg, s0, paths, i + kLsmThreads < paths, x,
                           S + static_cast<uint64_t>(d0) * paths + i);
            if (m < n) {
                s_x[at] = x[0];
                s_x[at + kLsmThreads] = x[1];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// per-date 4x4 algebra (FP64, one thread)
// ---------------------------------------------------------------------------
// Upper-triangular index of (r, c), r <= c, in the packed 10-entry layout.
__device__ __forceinline__ int tri(int r, int col) {
    const int base[4] = {0, 4, 7, 9};
    return base[r] + (col - r);
}

// Cholesky factor of G + shift I = R^T R (R upper); false when a pivot is
// not positive.
__device__ bool chol4(const double G[4][4], double shift, double R[4][4]) {
    for (int a = 0; a < 4; ++a)
        for (int b2 = 0; b2 < 4; ++b2) R[a][b2] = 0.0;
    for (int j = 0; j < 4; ++j) {
        double d = G[j][j] + shift;
        for (int p = 0; p < j; ++p) d -= R[p][j] * R[p][j];
        if (!(d > 0.0)) return false;
        R[j][j] = sqrt(d);
        for (int l = j + 1; l < 4; ++l) {
            double x = G[j][l];
            for (int p = 0; p < j; ++p) x -= R[p][j] * R[p][l];
            R[j][l] = x / R[j][j];
        }
    }
    return true;
}

// The same factorisation without divisions (FP64 division and square root
// are long software sequences on this GPU's FP64 pipe): one reciprocal square
// root per pivot, rinv[j] = 1 / R[j][j].
__device__ bool chol4_rsqrt(const double G[4][4], double R[4][4], double rinv[4]) {
    for (int a = 0; a < 4; ++a)
        for (int b2 = 0; b2 < 4; ++b2) R[a][b2] = 0.0;
    for (int j = 0; j < 4; ++j) {
        double d = G[j][j];
        for (int p = 0; p < j; ++p) d -= R[p][j] * R[p][j];
        if (!(d > 0.0)) return false;
        const double r = rsqrt(d);
        rinv[j] = r;
        R[j][j] = d * r;
        for (int l = j + 1; l < 4; ++l) {
            double x = G[j][l];
            for (int p = 0; p < j; ++p) x -= R[p][j] * R[p][l];
            R[j][l] = x * r;
        }
    }
    return true;
}

// T = R^{-1} from the pivots' reciprocals.
__device__ void inv_upper4_rinv(const double R[4][4], const double rinv[4], double T[4][4]) {
    for (int a = 0; a < 4; ++a)
        for (int b2 = 0; b2 < 4; ++b2) T[a][b2] = 0.0;
    for (int j = 3; j >= 0; --j) {
        T[j][j] = rinv[j];
        for (int l = j + 1; l < 4; ++l) {
            double x = 0.0;
            for (int p = j; p < l; ++p) x += T[j][p] * R[p][l];
            T[j][l] = -x * rinv[l];
        }
    }
}

// T = R^{-1} for upper-triangular R.
__device__ void inv_upper4(const double R[4][4], double T[4][4]) {
    for (int a = 0; a < 4; ++a)
        for (int b2 = 0; b2 < 4; ++b2) T[a][b2] = 0.0;
    for (int j = 3; j >= 0; --j) {
        T[j][j] = 1.0 / R[j][j];
        for (int l = j + 1; l < 4; ++l) {
            double x = 0.0;
            for (int p = j; p < l; ++p) x += T[j][p] * R[p][l];
            T[j][l] = -x / R[l][l];
        }
    }
}

// 4x4 Householder least squares (the reference's algorithm, src/core/linalg.cpp:7-71,
// on a square system): A is overwritten, y too.
__device__ void householder4(double A[4][4], double y[4], double beta[4]) {
    for (int kk = 0; kk < 4; ++kk) {
        double norm_sq = 0.0;
        for (int i = kk; i < 4; ++i) norm_sq += A[i][kk] * A[i][kk];
        const double norm = sqrt(norm_sq);
        if (norm == 0.0) continue;
        const double akk = A[kk][kk];
        const double alpha = akk >= 0.0 ? -norm : norm;
        double v[4] = {0, 0, 0, 0};
        v[kk] = akk - alpha;
        for (int i = kk + 1; i < 4; ++i) v[i] = A[i][kk];
        double vn = 0.0;
        for (int i = kk; i < 4; ++i) vn += v[i] * v[i];
        if (vn == 0.0) continue;
        for (int jj = kk; jj < 4; ++jj) {
            double dot = 0.0;
            for (int i = kk; i < 4; ++i) dot += v[i] * A[i][jj];
            const double f = 2.0 * dot / vn;
            for (int i = kk; i < 4; ++i) A[i][jj] -= f * v[i];
        }
        double dy = 0.0;
        for (int i = kk; i < 4; ++i) dy += v[i] * y[i];
        const double fy = 2.0 * dy / vn;
        for (int i = kk; i < 4; ++i) y[i] -= fy * v[i];
    }
    for (int i = 3; i >= 0; --i) {
        double sum = y[i];
        for (int jj = i + 1; jj < 4; ++jj) sum -= A[i][jj] * beta[jj];
        const double diag = A[i][i];
        beta[i] = diag != 0.0 ? sum / diag : 0.0;
    }
}

__device__ __forceinline__ void unpack_upper(const double* packed, double T[4][4]) {
    for (int a = 0; a < 4; ++a)
        for (int b2 = 0; b2 < 4; ++b2) T[a][b2] = b2 >= a ? packed[tri(a, b2)] : 0.0;
}

__device__ __forceinline__ void store_T(LsmReg& r, const double T[4][4]) {
    for (int a = 0; a < 4; ++a)
        for (int b2 = a; b2 < 4; ++b2) {
            r.T[tri(a, b2)] = T[a][b2];
            r.T_f[tri(a, b2)] = static_cast<float>(T[a][b2]);
        }
}

// Least squares on the preconditioned normal equations: s = (count, 10
// packed entries of G = P^T X^T X P, 4 entries of h = P^T X^T y) for the
// basis X P of preconditioner P (upper triangular).  Solves G beta = h by
// the 4x4 Householder QR and returns gamma = P beta, the coefficients in the
// Laguerre basis (the reference's policy layout).
__device__ void solve_preconditioned(const double* s, const double P[4][4], double gamma[4]) {
    double G[4][4], y[4], beta[4] = {0, 0, 0, 0};
    for (int a = 0; a < 4; ++a)
        for (int b2 = a; b2 < 4; ++b2) G[a][b2] = G[b2][a] = s[1 + tri(a, b2)];
    for (int a = 0; a < 4; ++a) y[a] = s[11 + a];
    householder4(G, y, beta);
    for (int a = 0; a < 4; ++a) {
        double x = 0.0;
        for (int b2 = a; b2 < 4; ++b2) x += P[a][b2] * beta[b2];
        gamma[a] = x;
    }
}

// The regression of one date from its sums in the basis of the lagged
// preconditioner L (the next later date's T).  Cholesky of G' = R^T R gives
// this date's preconditioner T = L R^{-1} (so that T^T X^T X T = I).  When G'
// is well conditioned (cond bound ||R||_F^2 ||R^-1||_F^2 <= kappa_max) the
// date is solved here from the same factor, beta = R^{-1} R^{-T} h and
// gamma = L beta: has = 1.  Otherwise T is stored and the date is marked for
// a second pass in the basis X T (has = 2): that pass and its Householder
// solve are Cholesky-QR2.  The first regression date (L = I, the raw Laguerre
// Gram matrix, condition up to ~1e13) always takes it; where that raw matrix
// is not numerically positive definite (its FP32-path sums carry ~44 bits) the
// factorisation is retried with a diagonal shift of 1e-10 of the trace --
// shifted Cholesky QR (Fukaya, Kannan, Nakatsukasa, Zhang and Yamamoto, SIAM
// J. Sci. Comput. 42 (2020)) -- and the second pass fits the unshifted problem.
__device__ void solve_lagged(const double* s, const double L[4][4], double kappa_max, LsmReg& r,
                             uint32_t* need_second_pass) {
    if (s[0] < 4.0) {  // too few in-the-money paths (src/pricers/lsm.cpp:102-104)
        r.has = -1;
        r.degenerate = 0;
        store_T(r, L);  // the lag passes through to the next earlier date
        return;
    }
    double G[4][4];
    for (int a = 0; a < 4; ++a)
        for (int b2 = a; b2 < 4; ++b2) G[a][b2] = G[b2][a] = s[1 + tri(a, b2)];
    double R[4][4], Ri[4][4], T[4][4], rinv[4];
    bool ok = chol4_rsqrt(G, R, rinv);
    double kappa = 1e300;
    if (ok) {
        inv_upper4_rinv(R, rinv, Ri);
        double fr = 0.0, fi = 0.0;
        for (int a = 0; a < 4; ++a)
            for (int b2 = a; b2 < 4; ++b2) {
                fr += R[a][b2] * R[a][b2];
                fi += Ri[a][b2] * Ri[a][b2];
            }
        kappa = fr * fi;
    }
    r.degenerate = 0;
    if (!ok) {
        const double shift = 1e-10 * (G[0][0] + G[1][1] + G[2][2] + G[3][3]);
        ok = chol4(G, shift, R);
        if (ok) inv_upper4(R, Ri);
        r.degenerate = ok ? 2 : 1;
    }
    if (ok) {
        for (int a = 0; a < 4; ++a)
            for (int b2 = 0; b2 < 4; ++b2) {
                double x = 0.0;
                for (int p = a; p <= b2; ++p) x += L[a][p] * Ri[p][b2];
                T[a][b2] = b2 >= a ? x : 0.0;
            }
    } else {
        for (int a = 0; a < 4; ++a)
            for (int b2 = 0; b2 < 4; ++b2) T[a][b2] = L[a][b2];
    }
    store_T(r, T);
    if (r.degenerate == 0 && kappa <= kappa_max) {
        double w[4], beta[4];
        for (int l = 0; l < 4; ++l) {  // w = R^{-T} h
            double x = 0.0;
            for (int p = 0; p <= l; ++p) x += Ri[p][l] * s[11 + p];
            w[l] = x;
        }
        for (int a = 0; a < 4; ++a) {  // beta = R^{-1} w
            double x = 0.0;
            for (int b2 = a; b2 < 4; ++b2) x += Ri[a][b2] * w[b2];
            beta[a] = x;
        }
        for (int a = 0; a < 4; ++a) {  // gamma = L beta
            double x = 0.0;
            for (int b2 = a; b2 < 4; ++b2) x += L[a][b2] * beta[b2];
            r.gamma[a] = x;
            r.gamma_f[a] = static_cast<float>(x);
        }
        laguerre_poly(r.gamma, r.poly, r.poly_f);
        r.has = 1;
    } else {
        r.has = 2;
        atomicAdd(need_second_pass, 1u);
    }
}

// 1 / sqrt(d), d > 0: an FP32 seed and one cubic iteration (fp64_fast.cuh), five
// FP64 operations in a row where the library's routine takes 427 cycles.
__device__ __forceinline__ double pivot_rsqrt(double d) {
    if (!seed_range(d)) return rsqrt(d);
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(seed_of(d)));
    const double y = seed_wide(r);
    const double e = fma(-d * y, y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// solve_lagged by one warp with one matrix element per lane: lane 4a + b of
// each half-warp holds element (a, b).  An FP64 operation holds the scheduler
// for 64 cycles with one lane active or with 32, and the serial form is a chain
// of about 300 of them.  PREC 1: the serial form's operations on the same
// operands, about 105; on FP32 paths a continuation value one bit off moves
// exercise decisions (those of paths within FP32 rounding of the boundary) and
// with them the price by 1e-5.  PREC 0: 65 (fused products, the pivots' own
// rsqrt, gamma = T R^{-T} h), 12,400 -> 9,000 cycles from the sums to the
// coefficients; decisions there would have to tie to 1e-16.  Only the form
// without a diagonal shift: a matrix that is not positive definite goes to the
// serial routine.
template <int PREC>
__device__ void solve_lagged_warp(const double* s /* shared, 15 */, const double* lag /* packed T, or null */,
                                  double kappa_max, LsmReg& r, uint32_t* need_second_pass) {
    auto madd = [](double x, double y, double z) { return PREC == 0 ? fma(x, y, z) : z + x * y; };
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, a = (lane >> 2) & 3, b = lane & 3;
    const bool writer = lane < 16 && a <= b;  // the upper triangle, first half-warp
    double l[4];                              // row a of the lag
#pragma unroll
    for (int p = 0; p < 4; ++p) l[p] = lag ? (p >= a ? lag[tri(a, p)] : 0.0) : (p == a ? 1.0 : 0.0);
    if (s[0] < 4.0) {  // too few in-the-money paths: the lag passes through
        if (lane == 0) {
            r.has = -1;
            r.degenerate = 0;
        }
        if (writer) {
            const double x = b == 0 ? l[0] : b == 1 ? l[1] : b == 2 ? l[2] : l[3];
            r.T[tri(a, b)] = x;
            r.T_f[tri(a, b)] = static_cast<float>(x);
        }
        return;
    }
    // Cholesky G = R^T R, one row per step
    double x = s[1 + (a <= b ? tri(a, b) : tri(b, a))], R = 0.0, rinv[4];
    bool ok = true;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const double d = __shfl_sync(kAll, x, 5 * p);
        ok = ok && d > 0.0;
        rinv[p] = PREC == 0 ? pivot_rsqrt(d) : rsqrt(d);
        if (a == p) R = x * rinv[p];
        if (p < 3) {
            const double ra = __shfl_sync(kAll, R, 4 * p + a), rb = __shfl_sync(kAll, R, 4 * p + b);
            if (a > p && b >= a) x = madd(-ra, rb, x);
        }
    }
    if (!ok) {
        if (lane == 0) {
            double L[4][4];
            for (int i = 0; i < 4; ++i)
                for (int j = 0; j < 4; ++j) L[i][j] = lag ? (j >= i ? lag[tri(i, j)] : 0.0) : (i == j ? 1.0 : 0.0);
            solve_lagged(s, L, kappa_max, r, need_second_pass);
        }
        return;
    }
    if (b < a) R = 0.0;
    // row a of R^{-1} (zero left of the diagonal)
    double t[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) t[q] = q == a ? rinv[q] : 0.0;
#pragma unroll
    for (int q = 1; q < 4; ++q) {
        double y = 0.0;
#pragma unroll
        for (int p = 0; p < q; ++p) y = madd(t[p], __shfl_sync(kAll, R, 4 * p + q), y);
        if (q > a) t[q] = -y * rinv[q];
    }
    const double ri = b == 0 ? t[0] : b == 1 ? t[1] : b == 2 ? t[2] : t[3];
    // ||R||^2 in the first half-warp, ||R^{-1}||^2 in the second
    const double el = lane < 16 ? R : ri;
    double norm = el * el;
#pragma unroll
    for (int off = 8; off >= 1; off >>= 1) norm += __shfl_xor_sync(kAll, norm, off);
    const double kappa = norm * __shfl_xor_sync(kAll, norm, 16);
    // T = L R^{-1}, and R^{-T} h by column b
    double tab = 0.0, w = 0.0;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const double rpb = __shfl_sync(kAll, ri, 4 * p + b);
        tab = madd(l[p], rpb, tab);
        w = madd(rpb, s[11 + p], w);
    }
    if (writer) {
        r.T[tri(a, b)] = tab;
        r.T_f[tri(a, b)] = static_cast<float>(tab);
    }
    if (lane == 0) r.degenerate = 0;
    if (!(kappa <= kappa_max)) {
        if (lane == 0) {
            r.has = 2;
            atomicAdd(need_second_pass, 1u);
        }
        return;
    }
    double gamma = 0.0;  // by row a
    if constexpr (PREC == 0) {
        gamma = tab * w;  // T R^{-T} h
        gamma += __shfl_xor_sync(kAll, gamma, 1);
        gamma += __shfl_xor_sync(kAll, gamma, 2);
    } else {
        double beta = 0.0;  // R^{-1} w, then L beta
#pragma unroll
        for (int q = 0; q < 4; ++q) beta = madd(t[q], __shfl_sync(kAll, w, q), beta);
#pragma unroll
        for (int q = 0; q < 4; ++q) gamma = madd(l[q], __shfl_sync(kAll, beta, 4 * q), gamma);
    }
    // laguerre_poly, coefficient a in row a (the products of +-1, -2 and 1/2 are exact)
    const double g[4] = {__shfl_sync(kAll, gamma, 0), __shfl_sync(kAll, gamma, 4), __shfl_sync(kAll, gamma, 8),
                         __shfl_sync(kAll, gamma, 12)};
    const double m1 = a == 0 ? 1.0 : a == 1 ? -1.0 : 0.0, m2 = a == 0 ? 1.0 : a == 1 ? -2.0 : 0.5;
    const double m3 = a == 0 ? 1.0 : a == 1 ? -3.0 : 1.5;
    double poly = fma(m2, g[2], fma(m1, g[1], a == 0 ? g[0] : 0.0)) + m3 * g[3];
    const double q0 = -g[3] * (1.0 / 6.0);  // -g3 / 6, correctly rounded
    const double sixth = fma(fma(-q0, 6.0, -g[3]), 1.0 / 6.0, q0);
    if (a == 3) poly = sixth;
    if (lane < 16 && b == 0) {
        r.gamma[a] = gamma;
        r.gamma_f[a] = static_cast<float>(gamma);
        r.poly[a] = poly;
        r.poly_f[a] = static_cast<float>(poly);
    }
    if (lane == 0) r.has = 1;
}

// Fixed-order fold of a contract's chunk partials by the whole CTA: thread t
// takes rows t, t + blockDim, ... in order, then the fixed block tree; the result is
// in res (shared) for every thread.
__device__ __forceinline__ void fold_partials(const LsmPartial* __restrict__ part, uint32_t begin, uint32_t count,
                                              double (*smem)[15], double* res) {
    double v[15];
#pragma unroll
    for (int q = 0; q < 15; ++q) v[q] = 0.0;
    for (uint32_t ch = threadIdx.x; ch < count; ch += blockDim.x) {
        const double2* p = reinterpret_cast<const double2*>(part[begin + ch].v);
        double row[16];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const double2 x = __ldcg(p + q);
            row[2 * q] = x.x;
            row[2 * q + 1] = x.y;
        }
#pragma unroll
        for (int q = 0; q < 15; ++q) v[q] = ch == threadIdx.x ? row[q] : v[q] + row[q];
    }
    block_sum15(v, static_cast<int>(min((count + 31u) / 32u, blockDim.x / 32u)), smem, res);
}

// One arrival at a completion counter; true in the CTA that arrives last.
// The arriving CTA's writes (thread 0's) are fenced before the counter is
// bumped, the last arrival fences again before it reads the others', and
// resets the counter for the next launch.  No CTA waits on another.
__device__ __forceinline__ bool last_arrival(uint32_t* counter, uint32_t expected, int* s_flag) {
    if (threadIdx.x == 0) {
        __threadfence();
        const uint32_t prev = atomicAdd(counter, 1u);
        const bool last = prev == expected - 1;
        if (last) *counter = 0u;
        *s_flag = last ? 1 : 0;
    }
    __syncthreads();
    const bool last = *s_flag != 0;
    if (last) __threadfence();
    return last;
}

// FP64: group sums of a contract up to this many are added in order, one sum per
// lane (15 FP64 additions at most, against 16 and 32 shuffles of the warp's tree).
constexpr uint32_t kSerialFolds = 16;

// Publishes this CTA's chunk partial (in res; thread q < 15 writes entry q) and
// climbs the two-level tree of the contract's sums: the last chunk of a group
// of LsmDev::fold_chunks chunks folds the group's partials in chunk order into
// the group partial, the last group of the contract folds the group partials
// in group order.  Every fold is short (a few dozen to a few hundred rows over
// the whole CTA), so the contract's totals are ready soon after its last
// chunk.  Returns true in the CTA holding the totals, then in res.
// counters: the group counter of group g at group_counters[2 g], the
// contract's at *contract_counter.
template <int PREC>
__device__ bool publish_and_fold(uint32_t chunk, const LsmDev& c, LsmPartial* __restrict__ part,
                                 LsmPartial* __restrict__ gpart, uint32_t* group_counters,
                                 uint32_t* contract_counter, double (*smem)[15], double* res, int* s_flag) {
    const uint32_t local = chunk - c.chunk_begin;
    const uint32_t g = local / c.fold_chunks;
    const uint32_t first = g * c.fold_chunks;
    const uint32_t count = min(c.fold_chunks, c.n_chunks - first);
    if (threadIdx.x < 15) part[chunk].v[threadIdx.x] = res[threadIdx.x];
    __syncthreads();
    if (!last_arrival(&group_counters[2 * (c.fold_begin + g)], count, s_flag)) return false;
    fold_partials(part, c.chunk_begin + first, count, smem, res);
    if (threadIdx.x < 15) gpart[c.fold_begin + g].v[threadIdx.x] = res[threadIdx.x];
    __syncthreads();
    if (!last_arrival(contract_counter, c.n_folds, s_flag)) return false;
    if (PREC == 0 && c.n_folds <= kSerialFolds) {
        if (threadIdx.x < 15) {
            double x = __ldcg(&gpart[c.fold_begin].v[threadIdx.x]);
            for (uint32_t i = 1; i < c.n_folds; ++i) x += __ldcg(&gpart[c.fold_begin + i].v[threadIdx.x]);
            res[threadIdx.x] = x;
        }
        __syncthreads();
    } else {
        fold_partials(gpart, c.fold_begin, c.n_folds, smem, res);
    }
    return true;
}

// ---------------------------------------------------------------------------
// iteration k: exercise at date e, discount, and the regression sums of date
// e-1 in the lagged basis -- or, when e = 1, the final Welford partial.  The
// contract's last CTA folds the sums and solves date e-1.
// ---------------------------------------------------------------------------
// One in-the-money path's share of the regression sums in the basis b T
// (b'_l = sum_{j <= l} b_j T[j][l]), FP64; entry 0, the count, is the caller's.
__device__ __forceinline__ void add_products64(const double (&b)[4], const double (&T)[10], double v,
                                               double (&acc)[15]) {
    const double q0 = b[0] * T[0];
    const double q1 = fma(b[1], T[4], b[0] * T[1]);
    const double q2 = fma(b[2], T[7], fma(b[1], T[5], b[0] * T[2]));
    const double q3 = fma(b[3], T[9], fma(b[2], T[8], fma(b[1], T[6], b[0] * T[3])));
    acc[1] = fma(q0, q0, acc[1]);
    acc[2] = fma(q0, q1, acc[2]);
    acc[3] = fma(q0, q2, acc[3]);
    acc[4] = fma(q0, q3, acc[4]);
    acc[5] = fma(q1, q1, acc[5]);
    acc[6] = fma(q1, q2, acc[6]);
    acc[7] = fma(q1, q3, acc[7]);
    acc[8] = fma(q2, q2, acc[8]);
    acc[9] = fma(q2, q3, acc[9]);
    acc[10] = fma(q3, q3, acc[10]);
    acc[11] = fma(q0, v, acc[11]);
    acc[12] = fma(q1, v, acc[12]);
    acc[13] = fma(q2, v, acc[13]);
    acc[14] = fma(q3, v, acc[14]);
}

// FP64: a warp's in-the-money paths, packed.  The products of a path take 24
// FP64 operations, each of which holds a scheduler for 64 cycles however many
// lanes need it, so the warp's 128 paths are packed before them: near the money
// two or three rounds of 32 instead of four.
constexpr int kWarpPaths = kLsmChunk / (kLsmThreads64 / 32);  // 128
constexpr int kPer64 = kLsmChunk / kLsmThreads64;             // paths per thread
struct MoneyRank {
    uint32_t at[kPer64];  // a path's position among the packed, or kWarpPaths
    uint32_t count;
};
__device__ __forceinline__ MoneyRank rank_money(const double (&s)[kPer64], double strike, int type) {
    MoneyRank r;
    r.count = 0;
    const uint32_t below = (1u << (threadIdx.x & 31)) - 1u;
#pragma unroll
    for (int j = 0; j < kPer64; ++j) {
        const bool in = in_the_money64(s[j], strike, type);
        const uint32_t mask = __ballot_sync(0xffffffffu, in);
        r.at[j] = in ? r.count + __popc(mask & below) : kWarpPaths;
        r.count += __popc(mask);
    }
    return r;
}
struct PackedPaths {
    double s[kWarpPaths], v[kWarpPaths];
};
// The sums of a warp's packed paths (entry 0, their number, in lane 0).
__device__ __forceinline__ void packed_sums64(const PackedPaths& p, uint32_t count, double inv_strike,
                                              const double (&T)[10], const GlobalTables& tables, double (&acc)[15]) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 15; ++q) acc[q] = 0.0;
    if (lane == 0) acc[0] = static_cast<double>(count);
    for (uint32_t at = lane; at < count; at += 32) {
        double b[4];
        basis64(p.s[at], inv_strike, tables, b);
        add_products64(b, T, p.v[at], acc);
    }
}

// COMP (FP32 path): the sums are compensated FP32 per thread and chunk (the
// first iteration, whose basis is the raw Laguerre one); otherwise plain FP32
// per thread and chunk -- the lagged basis is close to orthonormal, where
// FP32 sums lose nothing the FP32 path data does not already carry.
template <int PREC, bool COMP>
__global__ void __launch_bounds__(kChunkThreads<PREC>, PREC == 0 ? 1 : 8)
    lsm_step(int k, const LsmDev* __restrict__ cs, const uint32_t* __restrict__ chunk_contract,
             uint32_t chunk_first, uint32_t chunk_end, const void* __restrict__ store, double* __restrict__ cf,
             LsmReg* __restrict__ reg, LsmPartial* __restrict__ part, LsmPartial* __restrict__ gpart,
             Welford* __restrict__ final_part, uint32_t* __restrict__ counters,
             uint32_t* __restrict__ group_counters, uint32_t* __restrict__ need_second_pass, double kappa_max,
             const FixedTables* __restrict__ fixed) {
    __shared__ double smem[kChunkThreads<PREC> / 32][15];
    __shared__ float2 scratch[COMP ? 15 : 1][kLsmThreads];  // compensated sums' per-thread pairs
    __shared__ float pscratch[COMP ? 1 : 15][kLsmThreads];  // plain sums' per-thread values
    __shared__ double sres[15];
    __shared__ Welford swf[kChunkThreads<PREC> / 32];
    __shared__ Sum64 s64[kLsmThreads / 32];
    __shared__ PackedPaths s_packed[PREC == 0 ? kLsmThreads64 / 32 : 1];
    __shared__ int s_last;
    const uint32_t chunk = chunk_first + blockIdx.x;
    if (chunk >= chunk_end) return;
    const uint32_t ci = chunk_contract[chunk];
    const LsmDev c = cs[ci];
    const int n = c.n_steps;
    const int e = n - k;
    if (e < 1) return;  // this contract has finished (uniform per CTA)
    const bool init = (k == 0);
    const bool last = (e == 1);
    const bool gram = !last;
    const LsmReg* re = (!init && e <= n - 1) ? &reg[c.reg_offset + e] : nullptr;
    const bool exercise = re != nullptr && re->has == 1;
    const uint32_t local = chunk - c.chunk_begin;
    Welford w{0ull, 0.0, 0.0};
    if constexpr (PREC == 0) {
        const GlobalTables tables{fixed};
        double poly[4] = {0.0, 0.0, 0.0, 0.0};
        if (exercise) {
#pragma unroll
            for (int q = 0; q < 4; ++q) poly[q] = re->poly[q];
        }
        // lagged preconditioner: date e's T (identity before the first regression)
        double T[10];
#pragma unroll
        for (int q = 0; q < 10; ++q) T[q] = init ? ((q == 0 || q == 4 || q == 7 || q == 9) ? 1.0 : 0.0) : re->T[q];
        const double* S = static_cast<const double*>(store) + c.s_offset;
        const double* col_e = S + static_cast<uint64_t>(init ? n - 1 : e - 1) * c.path_count;
        const double* col_d = S + static_cast<uint64_t>(gram ? e - 2 : 0) * c.path_count;
        double* cash = cf + c.cf_offset;
        // all loads of this thread's paths first (independent, in flight together)
        const uint64_t i0 = static_cast<uint64_t>(local) * kLsmChunk + threadIdx.x;
        double vv[kPer64], se[kPer64], sd[kPer64];
#pragma unroll
        for (int j = 0; j < kPer64; ++j) {
            const uint64_t i = i0 + j * kLsmThreads64;
            const bool live = i < c.path_count;
            vv[j] = live && !init ? cash[i] : 0.0;
            se[j] = live && (init || exercise) ? col_e[i] : c.strike;
            sd[j] = live && gram ? col_d[i] : c.strike;
        }
        const MoneyRank rank = rank_money(sd, c.strike, c.type);
        PackedPaths& packed = s_packed[threadIdx.x >> 5];
#pragma unroll
        for (int j = 0; j < kPer64; ++j) {
            const uint64_t i = i0 + j * kLsmThreads64;
            if (i >= c.path_count) continue;
            double v = vv[j];
            if (in_the_money64(se[j], c.strike, c.type)) {
                const double ex = put_sign(se[j] - c.strike, c.type);
                if (init || ex > continuation64(se[j], c.inv_strike, poly, tables)) v = ex;
            }
            v *= c.disc;
            if (last) {
                welford_add(w, v);
            } else {
                cash[i] = v;
                if (rank.at[j] < kWarpPaths) {
                    packed.s[rank.at[j]] = sd[j];
                    packed.v[rank.at[j]] = v;
                }
            }
        }
        if (gram) {
            __syncwarp();
            double acc[15];
            packed_sums64(packed, rank.count, c.inv_strike, T, tables, acc);
            block_sum15(acc, kLsmThreads64 / 32, smem, sres);
        }
    } else {
        // FP32 paths: FP32 cash flows (stored in the FP64 buffer's space),
        // basis, continuation value, exercise tests and products; the sums
        // and the final payoff sums up to the warp are compensated FP32,
        // everything above FP64.
        const float phi = c.phi_f, strike = c.strike_f, inv_kf = c.inv_strike_f, disc = c.disc_f;
        float poly[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (exercise) {
#pragma unroll
            for (int q = 0; q < 4; ++q) poly[q] = re->poly_f[q];
        }
        float T[10];
#pragma unroll
        for (int q = 0; q < 10; ++q) T[q] = init ? ((q == 0 || q == 4 || q == 7 || q == 9) ? 1.0f : 0.0f) : re->T_f[q];
        const float* S = static_cast<const float*>(store) + c.s_offset;
        float* cff = reinterpret_cast<float*>(cf) + c.cf_offset;
        float hi[15], lo[15];
#pragma unroll
        for (int q = 0; q < 15; ++q) hi[q] = lo[q] = 0.0f;
        Sum32 fin{0u, 0.0f, 0.0f, 0.0f, 0.0f};  // final payoffs (last date)
        constexpr int kPer = kLsmChunk / kLsmThreads;
        // all loads of this thread's paths first (independent, in flight together);
        // the columns' thread bases once, 32-bit offsets within the chunk
        const uint64_t cb = static_cast<uint64_t>(local) * kLsmChunk;  // first path of the chunk
        const uint64_t i0 = cb + threadIdx.x;
        const uint32_t in_chunk = static_cast<uint32_t>(
            c.path_count - cb < static_cast<uint64_t>(kLsmChunk) ? c.path_count - cb : static_cast<uint64_t>(kLsmChunk));
        float* cf_t = cff + i0;
        const float* col_v = init ? S + static_cast<uint64_t>(n - 1) * c.path_count + i0 : cf_t;
        const float* col_e = S + static_cast<uint64_t>(exercise ? e - 1 : 0) * c.path_count + i0;
        const float* col_d = S + static_cast<uint64_t>(gram ? e - 2 : 0) * c.path_count + i0;
        float vv[kPer], se[kPer], sd[kPer];
        bool live[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const uint32_t o = static_cast<uint32_t>(j * kLsmThreads);
            live[j] = o + threadIdx.x < in_chunk;
            vv[j] = 0.0f;
            se[j] = 0.0f;
            sd[j] = 0.0f;
            if (live[j]) {
                vv[j] = col_v[o];
                if (exercise) se[j] = col_e[o];
                if (gram) sd[j] = col_d[o];
            }
        }
        if constexpr (!COMP) {
            // Branch-free, so that the paths of a thread interleave: a path that
            // is not in the money enters with e = 0, x = 1 and no cash flow, and
            // adds zeros (the sums keep their bits).  Nearly every warp holds
            // in-the-money lanes, so a branch would skip nothing.
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const float ex = phi * (se[j] - strike);
                float v = exercise && ex > 0.0f && ex > continuation_poly32(se[j], inv_kf, poly) ? ex : vv[j];
                v *= disc;
                if (last) {
                    if (live[j]) sum32_add(fin, v);
                    continue;
                }
                if (live[j]) cf_t[j * kLsmThreads] = v;
                const bool itm = live[j] && phi * (sd[j] - strike) > 0.0f;
                float b[4];
                basis32(itm ? sd[j] : strike, inv_kf, itm, b);
                v = itm ? v : 0.0f;
                const float q0 = b[0] * T[0];
                const float q1 = __fmaf_rn(b[1], T[4], b[0] * T[1]);
                const float q2 = __fmaf_rn(b[2], T[7], __fmaf_rn(b[1], T[5], b[0] * T[2]));
                const float q3 = __fmaf_rn(b[3], T[9], __fmaf_rn(b[2], T[8], __fmaf_rn(b[1], T[6], b[0] * T[3])));
                hi[0] += itm ? 1.0f : 0.0f;  // exact: a chunk holds fewer than 2^24 paths
                hi[1] = __fmaf_rn(q0, q0, hi[1]);
                hi[2] = __fmaf_rn(q0, q1, hi[2]);
                hi[3] = __fmaf_rn(q0, q2, hi[3]);
                hi[4] = __fmaf_rn(q0, q3, hi[4]);
                hi[5] = __fmaf_rn(q1, q1, hi[5]);
                hi[6] = __fmaf_rn(q1, q2, hi[6]);
                hi[7] = __fmaf_rn(q1, q3, hi[7]);
                hi[8] = __fmaf_rn(q2, q2, hi[8]);
                hi[9] = __fmaf_rn(q2, q3, hi[9]);
                hi[10] = __fmaf_rn(q3, q3, hi[10]);
                hi[11] = __fmaf_rn(q0, v, hi[11]);
                hi[12] = __fmaf_rn(q1, v, hi[12]);
                hi[13] = __fmaf_rn(q2, v, hi[13]);
                hi[14] = __fmaf_rn(q3, v, hi[14]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                if (!live[j]) continue;
                float v = init ? fmaxf(phi * (vv[j] - strike), 0.0f) : vv[j];
                if (exercise) {
                    const float ex = phi * (se[j] - strike);
                    if (ex > 0.0f && ex > continuation_poly32(se[j], inv_kf, poly)) v = ex;
                }
                v *= disc;
                if (last) {
                    sum32_add(fin, v);
                } else {
                    cf_t[j * kLsmThreads] = v;
                    if (phi * (sd[j] - strike) > 0.0f) {
                        float b[4];
                        basis32(sd[j], inv_kf, true, b);
                        const float q0 = b[0] * T[0];
                        const float q1 = __fmaf_rn(b[1], T[4], b[0] * T[1]);
                        const float q2 = __fmaf_rn(b[2], T[7], __fmaf_rn(b[1], T[5], b[0] * T[2]));
                        const float q3 = __fmaf_rn(b[3], T[9], __fmaf_rn(b[2], T[8], __fmaf_rn(b[1], T[6], b[0] * T[3])));
                        df_add(hi[0], lo[0], 1.0f);
                        df_add(hi[1], lo[1], q0 * q0);
                        df_add(hi[2], lo[2], q0 * q1);
                        df_add(hi[3], lo[3], q0 * q2);
                        df_add(hi[4], lo[4], q0 * q3);
                        df_add(hi[5], lo[5], q1 * q1);
                        df_add(hi[6], lo[6], q1 * q2);
                        df_add(hi[7], lo[7], q1 * q3);
                        df_add(hi[8], lo[8], q2 * q2);
                        df_add(hi[9], lo[9], q2 * q3);
                        df_add(hi[10], lo[10], q3 * q3);
                        df_add(hi[11], lo[11], q0 * v);
                        df_add(hi[12], lo[12], q1 * v);
                        df_add(hi[13], lo[13], q2 * v);
                        df_add(hi[14], lo[14], q3 * v);
                    }
                }
            }
        }
        if (last) {
            const Sum32 r = sum32_warp_reduce(fin);
            if ((threadIdx.x & 31) == 0) s64[threadIdx.x >> 5] = sum32_wide(r);
        }
        if (gram) {
            if constexpr (COMP) {
                block_sum_df<15>(hi, lo, scratch, sres);
            } else {
                block_sum_f32<15>(hi, pscratch, sres);
            }
        }
    }
    if (last) {
        if constexpr (PREC == 0) {
            w = welford_warp_reduce(w);
            if ((threadIdx.x & 31) == 0) swf[threadIdx.x >> 5] = w;
            __syncthreads();
            if (threadIdx.x == 0) {
                Welford m = swf[0];
                for (int q = 1; q < kLsmThreads64 / 32; ++q) m = welford_merge(m, swf[q]);
                final_part[chunk] = m;
            }
        } else {
            __syncthreads();
            if (threadIdx.x == 0) final_part[chunk] = sum64_fold<kLsmThreads / 32>(s64);
        }
        return;
    }
    if (!publish_and_fold<PREC>(chunk, c, part, gpart, group_counters, &counters[2 * ci], smem, sres, &s_last)) return;
    if (threadIdx.x < 32)
        solve_lagged_warp<PREC>(sres, init ? nullptr : re->T, kappa_max, reg[c.reg_offset + e - 1], need_second_pass + k);
}

// Second pass for the dates solve_lagged marked (has = 2): the sums in the
// basis of that date's own preconditioner T (compensated FP32 on the FP32
// path), then the contract's last chunk solves (has = 1).  A small
// persistent grid walks the chunks and skips those of other contracts.
template <int PREC>
__global__ void __launch_bounds__(kChunkThreads<PREC>, PREC == 0 ? 1 : 4)
    lsm_refine(int k, const LsmDev* __restrict__ cs, const uint32_t* __restrict__ chunk_contract,
               uint32_t chunk_first, uint32_t chunk_end, const void* __restrict__ store, const double* __restrict__ cf,
               LsmReg* __restrict__ reg, LsmPartial* __restrict__ part, LsmPartial* __restrict__ gpart,
               uint32_t* __restrict__ counters, uint32_t* __restrict__ group_counters,
               const uint32_t* __restrict__ need_second_pass, const FixedTables* __restrict__ fixed) {
    __shared__ double smem[kChunkThreads<PREC> / 32][15];
    __shared__ float2 scratch[15][kLsmThreads];  // FP32 path: the sums' per-thread pairs
    __shared__ double sres[15];
    __shared__ PackedPaths s_packed[PREC == 0 ? kLsmThreads64 / 32 : 1];
    __shared__ int s_last;
    if (__ldcg(need_second_pass + k) == 0) return;  // no date of this iteration needs it
    for (uint32_t chunk = chunk_first + blockIdx.x; chunk < chunk_end; chunk += gridDim.x) {
    const uint32_t ci = chunk_contract[chunk];
    const LsmDev c = cs[ci];
    const int date = c.n_steps - k - 1;
    if (date < 1) continue;
    LsmReg& r = reg[c.reg_offset + date];
    if (r.has != 2) continue;  // solved by the first pass, or no regression at this date
    const uint32_t local = chunk - c.chunk_begin;
    if constexpr (PREC == 0) {
        const GlobalTables tables{fixed};
        double T[10];
#pragma unroll
        for (int q = 0; q < 10; ++q) T[q] = r.T[q];
        const double* S = static_cast<const double*>(store) + c.s_offset + static_cast<uint64_t>(date - 1) * c.path_count;
        const uint64_t i0 = static_cast<uint64_t>(local) * kLsmChunk + threadIdx.x;
        double s[kPer64], v[kPer64];
#pragma unroll
        for (int j = 0; j < kPer64; ++j) {
            const uint64_t i = i0 + j * kLsmThreads64;
            s[j] = i < c.path_count ? S[i] : c.strike;
            v[j] = i < c.path_count ? cf[c.cf_offset + i] : 0.0;
        }
        const MoneyRank rank = rank_money(s, c.strike, c.type);
        PackedPaths& packed = s_packed[threadIdx.x >> 5];
#pragma unroll
        for (int j = 0; j < kPer64; ++j)
            if (rank.at[j] < kWarpPaths) {
                packed.s[rank.at[j]] = s[j];
                packed.v[rank.at[j]] = v[j];
            }
        __syncwarp();
        double acc[15];
        packed_sums64(packed, rank.count, c.inv_strike, T, tables, acc);
        block_sum15(acc, kLsmThreads64 / 32, smem, sres);
    } else {
        float T[10];
#pragma unroll
        for (int q = 0; q < 10; ++q) T[q] = r.T_f[q];
        const float phi = c.phi_f, strike = c.strike_f, inv_kf = c.inv_strike_f;
        const float* S = static_cast<const float*>(store) + c.s_offset;
        float hi[15], lo[15];
#pragma unroll
        for (int q = 0; q < 15; ++q) hi[q] = lo[q] = 0.0f;
        constexpr int kPer = kLsmChunk / kLsmThreads;
        float sv[kPer], yv[kPer];
        bool live[kPer];
        const float* cff = reinterpret_cast<const float*>(cf) + c.cf_offset;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const uint64_t i = static_cast<uint64_t>(local) * kLsmChunk + j * kLsmThreads + threadIdx.x;
            live[j] = i < c.path_count;
            sv[j] = live[j] ? S[static_cast<uint64_t>(date - 1) * c.path_count + i] : 0.0f;
            yv[j] = live[j] ? cff[i] : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            if (!live[j] || !(phi * (sv[j] - strike) > 0.0f)) continue;
            float b[4];
            basis32(sv[j], inv_kf, true, b);
            const float q0 = b[0] * T[0];
            const float q1 = __fmaf_rn(b[1], T[4], b[0] * T[1]);
            const float q2 = __fmaf_rn(b[2], T[7], __fmaf_rn(b[1], T[5], b[0] * T[2]));
            const float q3 = __fmaf_rn(b[3], T[9], __fmaf_rn(b[2], T[8], __fmaf_rn(b[1], T[6], b[0] * T[3])));
            const float y = yv[j];
            df_add(hi[0], lo[0], 1.0f);
            df_add(hi[1], lo[1], q0 * q0);
            df_add(hi[2], lo[2], q0 * q1);
            df_add(hi[3], lo[3], q0 * q2);
            df_add(hi[4], lo[4], q0 * q3);
            df_add(hi[5], lo[5], q1 * q1);
            df_add(hi[6], lo[6], q1 * q2);
            df_add(hi[7], lo[7], q1 * q3);
            df_add(hi[8], lo[8], q2 * q2);
            df_add(hi[9], lo[9], q2 * q3);
            df_add(hi[10], lo[10], q3 * q3);
            df_add(hi[11], lo[11], q0 * y);
            df_add(hi[12], lo[12], q1 * y);
            df_add(hi[13], lo[13], q2 * y);
            df_add(hi[14], lo[14], q3 * y);
        }
        block_sum_df<15>(hi, lo, scratch, sres);
    }
    if (publish_and_fold<PREC>(chunk, c, part, gpart, group_counters + 1, &counters[2 * ci + 1], smem, sres, &s_last)) {
        if (threadIdx.x == 0) {
            double T[4][4], gamma[4];
            unpack_upper(r.T, T);
            solve_preconditioned(sres, T, gamma);
            for (int a = 0; a < 4; ++a) {
                r.gamma[a] = gamma[a];
                r.gamma_f[a] = static_cast<float>(gamma[a]);
            }
            laguerre_poly(r.gamma, r.poly, r.poly_f);
            r.has = 1;
        }
    }
    __syncthreads();  // shared memory is reused by the next chunk
    }
}

// ---------------------------------------------------------------------------
// FP64 batches whose chunks all fit on the GPU at once: every date in one
// cooperative launch, one CTA per chunk.
// ---------------------------------------------------------------------------
// The lockstep form spends a date of a single contract mostly on latencies: two
// launches, the contract's and the date's records, two columns and the cash
// flows read again.  Here a CTA keeps its chunk's cash flows and the basis
// values of its in-the-money paths in shared memory.  The contract's last CTA
// folds and solves a date and publishes its number; meanwhile the others pack
// the next date's column and evaluate its basis.  Every operation on a path and
// every sum is the lockstep form's (the basis is evaluated once for both uses),
// so prices and policies have its bits.  A CTA waits for its own contract's
// CTAs only, all of them resident; a wait that runs out (kLsmChainPolls) is
// recorded and ends the CTA.
//
// Bound: a date is a serial chain of products (about 8,000 cycles, the FP64
// pipe), the CTA's and the contract's folds (9,000), the solve (9,000), two
// trips through L2 and the exercise tests (5,000).  A put of 131,072 paths and
// 50 dates: 37 -> 17 us a date, the call 1.92 -> 1.0 ms.  Two CTAs fit an SM, so
// batches of up to 304 chunks come here.  Puts of 50 dates, one launch against a
// launch per date, ms: one of 5,000 paths 1.10 and 1.53, of 131,072 1.13 and
// 1.69, of 311,296 1.81 and 2.36; five of 51,200 1.65 and 2.10; a hundred of
// 3,072 1.65 and 2.22; 300 of 1,000 1.60 and 2.27.
constexpr int kChainSlots = 5;  // s and the four basis values of a packed path
struct ChainWarp {
    double f[2][kChainSlots][kWarpPaths];  // packed paths of this date and of the next
    uint8_t path[2][kWarpPaths];           // their place in the warp's 128
    double cash[kWarpPaths];
};
struct ChainShared {
    ChainWarp warp[kLsmThreads64 / 32];
    double T[10], poly[4];
    int has;
};

__device__ __forceinline__ uint32_t load_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void store_release(uint32_t* p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Packs a column's in-the-money paths and evaluates their basis; returns their number.
__device__ __forceinline__ uint32_t pack_date(ChainWarp& w, int side, const double* __restrict__ col, uint64_t i0,
                                              const LsmDev& c, const GlobalTables& tables) {
    const uint32_t lane = threadIdx.x & 31;
    double s[kPer64];
#pragma unroll
    for (int j = 0; j < kPer64; ++j) {
        const uint64_t i = i0 + j * kLsmThreads64;
        s[j] = i < c.path_count ? __ldg(col + i) : c.strike;
    }
    const MoneyRank rank = rank_money(s, c.strike, c.type);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kPer64; ++j)
        if (rank.at[j] < kWarpPaths) {
            w.f[side][0][rank.at[j]] = s[j];
            w.path[side][rank.at[j]] = static_cast<uint8_t>(j * 32 + lane);
        }
    __syncwarp();
    for (uint32_t at = lane; at < rank.count; at += 32) {
        double b[4];
        basis64(w.f[side][0][at], c.inv_strike, tables, b);
#pragma unroll
        for (int q = 0; q < 4; ++q) w.f[side][1 + q][at] = b[q];
    }
    return rank.count;
}

// A chunk's sums over its packed paths, published; in the contract's last CTA
// the totals are in sres.  The two-level tree of publish_and_fold, a group of
// chunks per warp.
__device__ bool chain_sums(const ChainWarp& w, int side, uint32_t count, const double* T_shared, uint32_t chunk,
                           const LsmDev& c, LsmPartial* __restrict__ part, uint32_t* counter, double (*smem)[15],
                           double (*group)[15], double* sres, int* s_flag) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double T[10], acc[15];
#pragma unroll
    for (int q = 0; q < 10; ++q) T[q] = T_shared[q];
#pragma unroll
    for (int q = 0; q < 15; ++q) acc[q] = 0.0;
    if (lane == 0) acc[0] = static_cast<double>(count);
    for (uint32_t at = lane; at < count; at += 32) {
        double b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) b[q] = w.f[side][1 + q][at];
        add_products64(b, T, w.cash[w.path[side][at]], acc);
    }
    block_sum15(acc, kLsmThreads64 / 32, smem, sres);
    if (threadIdx.x < 15) part[chunk].v[threadIdx.x] = sres[threadIdx.x];
    __syncthreads();
    if (!last_arrival(counter, c.n_chunks, s_flag)) return false;
    for (uint32_t g = warp; g < c.n_folds; g += kLsmThreads64 / 32) {
        const uint32_t at = g * c.fold_chunks + lane;
        double v[16] = {};
        if (at < c.n_chunks) {
            const double2* p = reinterpret_cast<const double2*>(part[c.chunk_begin + at].v);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const double2 x = __ldcg(p + q);
                v[2 * q] = x.x;
                v[2 * q + 1] = x.y;
            }
        }
        double u[15];
#pragma unroll
        for (int q = 0; q < 15; ++q) u[q] = v[q];
        const double x = warp_sums15(u);
        if ((lane & 1) == 0 && lane < 30) group[g][lane >> 1] = x;
    }
    __syncthreads();
    if (threadIdx.x < 15) {
        double x = group[0][threadIdx.x];
        for (uint32_t i = 1; i < c.n_folds; ++i) x += group[i][threadIdx.x];
        sres[threadIdx.x] = x;
    }
    __syncwarp();
    return true;
}

__global__ void __launch_bounds__(kLsmThreads64, 2)
    lsm_chain64(const LsmDev* __restrict__ cs, const uint32_t* __restrict__ chunk_contract,
                const double* __restrict__ store, LsmReg* __restrict__ reg, LsmPartial* __restrict__ part,
                Welford* __restrict__ final_part, uint32_t* __restrict__ counters /* arrivals, epoch */,
                uint32_t* __restrict__ need, double kappa_max, double* __restrict__ error, uint32_t max_polls,
                const FixedTables* __restrict__ fixed) {
    extern __shared__ __align__(16) unsigned char chain_smem[];
    ChainShared& sh = *reinterpret_cast<ChainShared*>(chain_smem);
    __shared__ double smem[kLsmThreads64 / 32][15];
    __shared__ double group[kSerialFolds][15];
    __shared__ double sres[15];
    __shared__ Welford swf[kLsmThreads64 / 32];
    __shared__ int s_flag, s_waited;
    const uint32_t chunk = blockIdx.x, ci = chunk_contract[chunk];
    const LsmDev c = cs[ci];
    const GlobalTables tables{fixed};
    const uint32_t lane = threadIdx.x & 31;
    ChainWarp& w = sh.warp[threadIdx.x >> 5];
    uint32_t* arrivals = &counters[2 * ci];
    uint32_t* epoch = &counters[2 * ci + 1];
    uint32_t seen = 0;
    const uint64_t i0 = static_cast<uint64_t>(chunk - c.chunk_begin) * kLsmChunk + threadIdx.x;
    const double* S = store + c.s_offset;
    auto column = [&](int date) { return S + static_cast<uint64_t>(date - 1) * c.path_count; };
    auto publish = [&] {  // warp 0 of the contract's last CTA
        __syncwarp();
        if (lane == 0) {
            __threadfence();
            store_release(epoch, seen + 1);
        }
    };
    // Waits for the next epoch and takes the date's record; false: gave up.
    auto await = [&](int date) {
        ++seen;
        if (threadIdx.x == 0) {
            uint32_t polls = 0;
            while (load_acquire(epoch) < seen && ++polls < max_polls) {}
            s_waited = polls < max_polls;
        }
        __syncthreads();
        const bool ok = s_waited != 0;
        const LsmReg& r = reg[c.reg_offset + date];
        if (threadIdx.x < 10) sh.T[threadIdx.x] = __ldcg(&r.T[threadIdx.x]);
        else if (threadIdx.x < 14) sh.poly[threadIdx.x - 10] = __ldcg(&r.poly[threadIdx.x - 10]);
        else if (threadIdx.x == 14) sh.has = __ldcg(&r.has);
        __syncthreads();
        if (!ok && threadIdx.x == 0) *error = 1.0;
        return ok;
    };
    // the terminal date
    const int n = c.n_steps;
#pragma unroll
    for (int j = 0; j < kPer64; ++j) {
        const uint64_t i = i0 + j * kLsmThreads64;
        const double s = i < c.path_count ? column(n)[i] : c.strike;
        const double v = in_the_money64(s, c.strike, c.type) ? put_sign(s - c.strike, c.type) : 0.0;
        w.cash[j * 32 + lane] = v * c.disc;
    }
    if (threadIdx.x < 10) {
        const int q = threadIdx.x;
        sh.T[q] = q == 0 || q == 4 || q == 7 || q == 9 ? 1.0 : 0.0;
    }
    __syncthreads();
    int side = 0;
    uint32_t count = n > 1 ? pack_date(w, side, column(n - 1), i0, c, tables) : 0u;
    __syncwarp();
    for (int e = n; e > 1; --e) {
        // the sums of date e - 1 in the basis of date e, whose T is in sh
        if (chain_sums(w, side, count, sh.T, chunk, c, part, arrivals, smem, group, sres, &s_flag) && threadIdx.x < 32) {
            solve_lagged_warp<0>(sres, e == n ? nullptr : sh.T, kappa_max, reg[c.reg_offset + e - 1], need);
            publish();
        }
        // meanwhile the date before it
        uint32_t next = 0;
        if (e > 2) next = pack_date(w, side ^ 1, column(e - 2), i0, c, tables);
        if (!await(e - 1)) return;
        if (sh.has == 2) {  // second pass in the basis of the date's own T (lsm_refine)
            if (chain_sums(w, side, count, sh.T, chunk, c, part, arrivals, smem, group, sres, &s_flag) &&
                threadIdx.x < 32) {
                if (lane == 0) {
                    LsmReg& r = reg[c.reg_offset + e - 1];
                    double T[4][4], gamma[4];
                    unpack_upper(sh.T, T);
                    solve_preconditioned(sres, T, gamma);
                    for (int a = 0; a < 4; ++a) {
                        r.gamma[a] = gamma[a];
                        r.gamma_f[a] = static_cast<float>(gamma[a]);
                    }
                    laguerre_poly(r.gamma, r.poly, r.poly_f);
                    r.has = 1;
                }
                publish();
            }
            if (!await(e - 1)) return;
        }
        // exercise at date e - 1, discount
        if (sh.has == 1) {
#pragma unroll
            for (int j = 0; j < kPer64; ++j) {
                const uint32_t at = j * 32 + lane;
                if (at >= count) break;
                const double s = w.f[side][0][at], x = s * c.inv_strike;
                const double ex = put_sign(s - c.strike, c.type);
                const double go = w.f[side][1][at] * fma(fma(fma(sh.poly[3], x, sh.poly[2]), x, sh.poly[1]), x, sh.poly[0]);
                if (ex > go) w.cash[w.path[side][at]] = ex;
            }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < kPer64; ++j) w.cash[j * 32 + lane] *= c.disc;
        __syncwarp();
        side ^= 1;
        count = next;
    }
    Welford f{0ull, 0.0, 0.0};
#pragma unroll
    for (int j = 0; j < kPer64; ++j)
        if (i0 + j * kLsmThreads64 < c.path_count) welford_add(f, w.cash[j * 32 + lane]);
    f = welford_warp_reduce(f);
    if (lane == 0) swf[threadIdx.x >> 5] = f;
    __syncthreads();
    if (threadIdx.x == 0) {
        Welford m = swf[0];
        for (int q = 1; q < kLsmThreads64 / 32; ++q) m = welford_merge(m, swf[q]);
        final_part[chunk] = m;
    }
}

// One CTA per contract.
__global__ void __launch_bounds__(kMergeThreads)
    lsm_finish(const LsmDev* __restrict__ cs, const Welford* __restrict__ final_part, double* __restrict__ out) {
    const int ci = blockIdx.x;
    const LsmDev& c = cs[ci];
    const MergedResult w = merge_items(final_part + c.chunk_begin, c.n_chunks, 1);
    if (threadIdx.x != 0) return;
    const double se = w.standard_error;
    // inception decision (src/pricers/lsm.cpp:141-148)
    const bool ex0 = c.inception > w.mean;
    out[6 * ci + 0] = ex0 ? c.inception : w.mean;
    out[6 * ci + 1] = ex0 ? 0.0 : se;
    out[6 * ci + 2] = static_cast<double>(w.count);
    out[6 * ci + 3] = ex0 ? 1.0 : 0.0;
    out[6 * ci + 4] = w.mean;  // path average before the inception test
    out[6 * ci + 5] = se;
}

}  // namespace

cudaError_t launch_lsm_forward(int precision, int sm_count, const LsmDev* c, const uint32_t* chunk_contract,
                               uint32_t chunk_first, uint32_t chunk_count, void* s_store, const FixedTables* tables,
                               cudaStream_t stream) {
    cudaGetLastError();
    if (chunk_count == 0) return cudaSuccess;
    const uint32_t end = chunk_first + chunk_count;
    if (precision == 0) {
        constexpr int bytes = static_cast<int>(sizeof(ForwardShared));
        cudaError_t e = cudaFuncSetAttribute(lsm_forward64, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
        lsm_forward64<<<sm_count, 1024, bytes, stream>>>(c, chunk_contract, chunk_first, end,
                                                         static_cast<double*>(s_store), tables);
    } else {
        lsm_forward32<<<chunk_count, kLsmThreads, 0, stream>>>(c, chunk_contract, chunk_first, end,
                                                               static_cast<float*>(s_store));
    }
    return cudaGetLastError();
}

cudaError_t launch_lsm_iteration(int precision, int k, const LsmDev* c, int n_contracts,
                                 const uint32_t* chunk_contract, uint32_t chunk_first, uint32_t chunk_count,
                                 uint32_t total_folds, const void* s_store, double* cf, LsmReg* reg,
                                 LsmPartial* part, LsmPartial* gpart, Welford* final_part, uint32_t* counters,
                                 const FixedTables* tables, cudaStream_t stream) {
    cudaGetLastError();
    if (chunk_count == 0) return cudaSuccess;
    const uint32_t end = chunk_first + chunk_count;
    // counters: 2 per contract (first pass, second pass), 2 per fold group, then
    // one word per iteration counting the dates marked for the second pass
    // (shared by concurrent chains: a chain's second pass reads it after its
    // own first pass, and only adds are made to it).
    uint32_t* group_counters = counters + 2 * static_cast<size_t>(n_contracts);
    uint32_t* need = group_counters + 2 * static_cast<size_t>(total_folds);
    // The second pass always runs after the first iteration (its lag is the
    // identity), on a CTA per chunk; later it is rare and runs on a small
    // persistent grid whose CTAs walk the chunks and skip those of contracts
    // whose date needs no second pass (all of them return at once when no
    // date does).
    const unsigned refine_grid = (k == 0 || chunk_count < kRefineGrid) ? chunk_count : kRefineGrid;
    // Condition bound below which a date is solved from its lagged sums: FP64
    // sums are good to ~1e-15, so 1e2 keeps the solve near FP64 accuracy; the
    // FP32 path's plain chunk sums are good to ~1e-8 relative once summed
    // over the chunks, and 1e3 keeps its coefficients inside the rounding the
    // FP32 basis values carry anyway.
    if (precision == 0) {
        if (k == 0)
            lsm_step<0, true><<<chunk_count, kLsmThreads64, 0, stream>>>(
                k, c, chunk_contract, chunk_first, end, s_store, cf, reg, part, gpart, final_part, counters,
                group_counters, need, 1e2, tables);
        else
            lsm_step<0, false><<<chunk_count, kLsmThreads64, 0, stream>>>(
                k, c, chunk_contract, chunk_first, end, s_store, cf, reg, part, gpart, final_part, counters,
                group_counters, need, 1e2, tables);
        lsm_refine<0><<<refine_grid, kLsmThreads64, 0, stream>>>(k, c, chunk_contract, chunk_first, end, s_store, cf,
                                                               reg, part, gpart, counters, group_counters, need,
                                                               tables);
    } else {
        if (k == 0)
            lsm_step<1, true><<<chunk_count, kLsmThreads, 0, stream>>>(
                k, c, chunk_contract, chunk_first, end, s_store, cf, reg, part, gpart, final_part, counters,
                group_counters, need, 1e3, tables);
        else
            lsm_step<1, false><<<chunk_count, kLsmThreads, 0, stream>>>(
                k, c, chunk_contract, chunk_first, end, s_store, cf, reg, part, gpart, final_part, counters,
                group_counters, need, 1e3, tables);
        lsm_refine<1><<<refine_grid, kLsmThreads, 0, stream>>>(k, c, chunk_contract, chunk_first, end, s_store, cf,
                                                               reg, part, gpart, counters, group_counters, need,
                                                               tables);
    }
    return cudaGetLastError();
}

cudaError_t lsm_chain64_capacity(int sm_count, uint32_t* chunks) {
    constexpr int bytes = static_cast<int>(sizeof(ChainShared));
    cudaError_t e = cudaFuncSetAttribute(lsm_chain64, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    int blocks = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, lsm_chain64, kLsmThreads64, bytes);
    *chunks = e == cudaSuccess ? static_cast<uint32_t>(blocks) * static_cast<uint32_t>(sm_count) : 0u;
    return e;
}

cudaError_t launch_lsm_chain64(const LsmDev* c, int n_contracts, const uint32_t* chunk_contract, uint32_t chunk_count,
                               uint32_t total_folds, const double* s_store, LsmReg* reg, LsmPartial* part,
                               Welford* final_part, uint32_t* counters, double* error, uint32_t polls, size_t shared,
                               const FixedTables* tables, cudaStream_t stream) {
    cudaGetLastError();
    if (chunk_count == 0) return cudaSuccess;
    uint32_t* need = counters + 2 * static_cast<size_t>(n_contracts) + 2 * static_cast<size_t>(total_folds);
    double kappa_max = 1e2;  // as launch_lsm_iteration
    void* args[] = {&c, &chunk_contract, &s_store, &reg, &part, &final_part, &counters, &need, &kappa_max, &error, &polls, &tables};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(lsm_chain64), dim3(chunk_count),
                                       dim3(kLsmThreads64), args, shared ? shared : sizeof(ChainShared), stream);
}

cudaError_t launch_lsm_finish(const LsmDev* c, int n_contracts, const Welford* final_part,
                              double* out, cudaStream_t stream) {
    cudaGetLastError();
    if (n_contracts > 0) lsm_finish<<<n_contracts, kMergeThreads, 0, stream>>>(c, final_part, out);
    return cudaGetLastError();
}

}  // namespace mcdg
