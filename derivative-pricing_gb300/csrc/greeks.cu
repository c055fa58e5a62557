// greeks.cu -- Monte Carlo sensitivities of a batch of GBM contracts in one
// persistent launch: common-random-number finite differences (spot and vol
// bumps), pathwise and likelihood-ratio estimators, all from one pass over
// each path's draws.
//
// The work items, slab layout, reduction trees and merge are those of the
// path engine (gbm_paths.cu), so the price output of this kernel is bitwise
// the price of mcd_price_batch for the same contract and precision.
//
// Reference semantics:
//   finite differences  src/greeks/finite_difference.cpp:40-65 (central
//                       differences of CRN re-prices; here per path, so the
//                       estimate comes with its standard error)
//   likelihood ratio    src/greeks/likelihood_ratio.cpp:33-73 (terminal) and
//                       :105-154 (barrier: first-step score for delta and
//                       gamma, per-step sums for vega and rho); the same
//                       first-step score is applied to Asian and lookback
//                       payoffs, which the reference does not cover
//   pathwise            src/greeks/pathwise.cpp:28-55 (European), :64-147
//                       (Asian)
//
// This file holds the FP32 kernel; the FP64 one, which evaluates every bumped
// state literally (five separate re-prices on one path's draws), is
// greeks64.cu.  FP32 shares one log-path between the spot states (only the
// FP64 payoff is rescaled) and carries the vol-bumped states as differentials: with D_i = dx_i/dvol = sqrt(dt) W_i - vol i dt, the bumped
// log-spot is x_i +/- h D_i - h^2 i dt / 2 exactly, and its effect on a sum
// of spots is sum S_i expm1(+/- h D_i - h^2 i dt / 2), which FP32 resolves to
// full relative precision even for bumps of 1e-4 (a plain FP32 re-price
// would lose the difference in rounding noise).
//
// Measured (1024 Asians and barriers, 252 dates, 2^18 paths): 279 ms at the
// former default of 128 registers, 239 ms at its best launch shape (64
// registers, 8 CTAs per SM), 221 ms with the Philox products of the draw and of
// the path taken out of the step, transposed warp sums instead of twelve
// Welford trees, and 8 CTAs per SM as the default, 211 ms with the logarithm and
// the exponentials of fp32_fast.cuh.
//
// nvcc-flags: --fmad=false
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "engine.hpp"
#include "greeks.hpp"
#include "merge.cuh"
#include "unit_sums.cuh"

namespace mcdg {

namespace {

__device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; }

// expm1 for the vol-bump exponents: a short Taylor series where |a| < 1/64
// (relative error below 2e-12 there; bumps of 1e-4 give |a| ~ 1e-4), else
// fast_exp(a) - 1 (relative error ~1e-7 / |a|, used for bumps above ~1 %).
__device__ __forceinline__ float expm1_small(float a) {
    if (fabsf(a) < 0.015625f) {
        const float p = __fmaf_rn(__fmaf_rn(__fmaf_rn(a, 1.0f / 120.0f, 1.0f / 24.0f), a, 1.0f / 6.0f), a, 0.5f);
        return __fmaf_rn(p * a, a, a);
    }
    return fast_exp(a) - 1.0f;
}

// expm1 by its cubic Taylor polynomial, for exponents the host bounds by
// 1e-2 (DevGreeks::vol_series): the first omitted term is below a^3 / 24 <
// 5e-8 of the result, under an FP32 rounding, in three instructions and
// without the range test of expm1_small.
__device__ __forceinline__ float expm1_series(float a) {
    return __fmaf_rn(__fmaf_rn(a, 1.0f / 6.0f, 0.5f) * a, a, a);
}

// ===========================================================================
// FP32: one log-path, differential vol states, FP64 payoffs of the states
// ===========================================================================
template <int KIND, bool SER>
__device__ void greeks32(const DevContract& c, const DevGreeks& g, const PhiloxKeys& k, PhiloxStep* table,
                         uint64_t path, bool refill, double (&o)[kNumGreeks]) {
#pragma unroll
    for (int i = 0; i < kNumGreeks; ++i) o[i] = 0.0;
    const float phi = c.type == 0 ? 1.0f : -1.0f;
    const double phid = c.type == 0 ? 1.0 : -1.0;
    const float mu = static_cast<float>(c.drift);
    const float sg = static_cast<float>(c.vs);
    const float s0 = static_cast<float>(c.spot);
    const float strike = static_cast<float>(c.strike);
    const double S0 = c.spot, K = c.strike, disc = c.discount, hs = g.h_spot, hv = g.h_vol;
    const float hvf = static_cast<float>(hv);
    const float cq = static_cast<float>(0.5 * hv * hv * g.dt);
    const uint32_t path_hi = static_cast<uint32_t>(path >> 32);
    const PhiloxRow row = philox_row(static_cast<uint32_t>(path), 0u, k);
    double v[5];
    if constexpr (KIND == kEuropean || KIND == kDigital) {
        const float z = normal_from_bits_f32(philox_word0(row, philox_step(0u, path_hi, k), k));
        const float ef = __expf(__fmaf_rn(sg, z, mu));  // (subnormal too: a bumped state multiplies it by up to 1e38)
        const float s = s0 * ef;  // as the path engine
        float payoff;
        if constexpr (KIND == kEuropean) {
            payoff = fmaxf(phi * (s - strike), 0.0f);
        } else {
            const bool itm = phi * (s - strike) > 0.0f;
            payoff = itm ? (c.asset ? s : static_cast<float>(c.cash)) : 0.0f;
        }
        o[kGPrice] = c.discount * static_cast<double>(payoff);
        const float D = __fmaf_rn(static_cast<float>(g.sqrt_dt), z, -static_cast<float>(g.vol * g.time));
        const double em_up = static_cast<double>(expm1_small(__fmaf_rn(hvf, D, -cq)));
        const double em_dn = static_cast<double>(expm1_small(__fmaf_rn(-hvf, D, -cq)));
        const double st0 = S0 * static_cast<double>(ef);
        const double st[5] = {st0, (S0 + hs) * static_cast<double>(ef), (S0 - hs) * static_cast<double>(ef),
                              st0 + st0 * em_up, st0 + st0 * em_dn};
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            if constexpr (KIND == kEuropean) {
                v[j] = disc * dmax(phid * (st[j] - K), 0.0);
            } else {
                const bool itm = phid * (st[j] - K) > 0.0;
                v[j] = disc * (itm ? (c.asset ? st[j] : c.cash) : 0.0);
            }
        }
        const double h = v[0];
        const double zd = static_cast<double>(z);
        const double sqrt_t = g.sqrt_dt;
        o[kGLrDelta] = h * (zd * g.lr_delta_scale);
        o[kGLrGamma] = h * ((zd * zd - g.vol * sqrt_t * zd - 1.0) * g.lr_gamma_scale);
        o[kGLrVega] = h * ((zd * zd - 1.0) * g.inv_vol - sqrt_t * zd);
        o[kGLrRho] = h * (g.sqrt_dt_over_vol * zd - g.time);
        o[kGLrTheta] = h * (g.rate - ((zd * zd - 1.0) * g.inv_2t + g.mu_over_vol_sqrt_t * zd));
        if constexpr (KIND == kEuropean) {
            const bool itm = phid * (st0 - K) > 0.0;
            const double slope = itm ? phid : 0.0;
            o[kGPwDelta] = disc * slope * static_cast<double>(ef);
            o[kGPwVega] = disc * slope * st0 * static_cast<double>(D);
            o[kGPwRho] = disc * slope * st0 * g.time - g.time * h;
        }
    } else {
        const float lnh = static_cast<float>(c.log_h_rel);
        const float lnh_su = static_cast<float>(g.log_h_rel_up);
        const float lnh_sd = static_cast<float>(g.log_h_rel_dn);
        const float sqdt = static_cast<float>(g.sqrt_dt);
        const float vdt = static_cast<float>(g.vol * g.dt);
        const float inv_vol = static_cast<float>(1.0 / g.vol);
        // Per step: the log-spot x (as the path engine), the running sums of
        // the draws and of their squares (the likelihood-ratio vega and rho
        // scores follow from them), D = dx/dvol = sqrt(dt) sum z - vol i dt,
        // and the vol-bump exponents +/- h D - h^2 i dt / 2.  A barrier or
        // lookback state needs only the running extremes of x, x + e_up and
        // x + e_dn: a barrier is touched on some date exactly when the extreme
        // over the dates reaches it.
        float x = 0.0f, D = 0.0f, z1 = 0.0f, zsum = 0.0f, zsq = 0.0f, fi = 0.0f;
        float acc = 0.0f, acc2 = 0.0f, xmax = 0.0f, xmin = 0.0f;  // as the path engine
        float a_d = 0.0f, a_r = 0.0f, a_up = 0.0f, a_dn = 0.0f, sd = 0.0f;
        float xmax_up = 0.0f, xmin_up = 0.0f, xmax_dn = 0.0f, xmin_dn = 0.0f;
        float e_up = 0.0f, e_dn = 0.0f;  // bump exponents of the last step
        if constexpr (KIND == kBarrier) {  // extremes over the monitoring dates only
            const float start = c.up ? -3.0e38f : 3.0e38f;
            xmax = xmin = xmax_up = xmin_up = xmax_dn = xmin_dn = start;
        }
        for (int d0 = 0; d0 < c.n_steps; d0 += 32) {
          if (refill || c.n_steps > 32) {  // the Philox words of the warp's next 32 steps
            __syncwarp();
            table[threadIdx.x & 31] = philox_step(static_cast<uint32_t>(d0 + (threadIdx.x & 31)), path_hi, k);
            __syncwarp();
          }
          const int count = min(32, c.n_steps - d0);
          for (int step = 0; step < count; ++step) {
            const float z = normal_from_bits_f32(philox_word0(row, table[step], k));
            if (d0 + step == 0) z1 = z;
            x = __fmaf_rn(sg, z, x + mu);
            zsum += z;
            zsq = __fmaf_rn(z, z, zsq);
            fi += 1.0f;
            D = __fmaf_rn(sqdt, zsum, -vdt * fi);
            const float q = cq * fi;
            e_up = __fmaf_rn(hvf, D, -q);
            e_dn = __fmaf_rn(-hvf, D, -q);
            if constexpr (KIND == kAsianArith) {
                // with bumps beyond the series a growth factor may be as large as e is small
                const float e = SER ? fast_exp(x) : __expf(x);
                acc += e;
                a_d = __fmaf_rn(e, D, a_d);
                a_r = __fmaf_rn(e, fi, a_r);
                a_up = __fmaf_rn(e, SER ? expm1_series(e_up) : expm1_small(e_up), a_up);
                a_dn = __fmaf_rn(e, SER ? expm1_series(e_dn) : expm1_small(e_dn), a_dn);
            } else if constexpr (KIND == kAsianGeo) {
                acc2 += x;
                sd += D;
            } else if constexpr (KIND == kBarrier) {
                if (c.up) {
                    xmax = fmaxf(xmax, x);
                    xmax_up = fmaxf(xmax_up, x + e_up);
                    xmax_dn = fmaxf(xmax_dn, x + e_dn);
                } else {
                    xmin = fminf(xmin, x);
                    xmin_up = fminf(xmin_up, x + e_up);
                    xmin_dn = fminf(xmin_dn, x + e_dn);
                }
            } else {
                xmax = fmaxf(xmax, x);
                xmin = fminf(xmin, x);
                xmax_up = fmaxf(xmax_up, x + e_up);
                xmin_up = fminf(xmin_up, x + e_up);
                xmax_dn = fmaxf(xmax_dn, x + e_dn);
                xmin_dn = fminf(xmin_dn, x + e_dn);
            }
          }
        }
        // sum over steps of (z^2 - 1) / vol - sqrt(dt) z
        const float lr_vega = __fmaf_rn(zsq - fi, inv_vol, -sqdt * zsum);
        bool br = false, br_su = false, br_sd = false, br_vu = false, br_vd = false;
        if constexpr (KIND == kBarrier) {
            if (c.up) {
                br = xmax >= lnh;
                br_su = xmax >= lnh_su;
                br_sd = xmax >= lnh_sd;
                br_vu = xmax_up >= lnh;
                br_vd = xmax_dn >= lnh;
            } else {
                br = xmin <= lnh;
                br_su = xmin <= lnh_su;
                br_sd = xmin <= lnh_sd;
                br_vu = xmin_up <= lnh;
                br_vd = xmin_dn <= lnh;
            }
        }
        // price: the path engine's FP32 payoff
        const float inv_n = 1.0f / static_cast<float>(c.n_steps);
        const float lastf = s0 * __expf(x);
        if constexpr (KIND == kAsianArith || KIND == kAsianGeo) {
            const float avg = KIND == kAsianArith ? s0 * (acc * inv_n) : s0 * __expf(acc2 * inv_n);
            const float ref = c.floating ? (lastf - avg) : (avg - strike);
            o[kGPrice] = c.discount * static_cast<double>(fmaxf(phi * ref, 0.0f));
        } else if constexpr (KIND == kBarrier) {
            const float vanilla = fmaxf(phi * (lastf - strike), 0.0f);
            const bool pays = c.out ? !br : br;
            o[kGPrice] = c.discount * static_cast<double>(pays ? vanilla : static_cast<float>(c.rebate));
        } else if constexpr (KIND == kLookbackFixed) {
            const float val = c.type == 0 ? fmaxf(s0 * __expf(xmax) - strike, 0.0f)
                                          : fmaxf(strike - s0 * __expf(xmin), 0.0f);
            o[kGPrice] = c.discount * static_cast<double>(val);
        } else {
            const float val = c.type == 0 ? (lastf - s0 * __expf(xmin)) : (s0 * __expf(xmax) - lastf);
            o[kGPrice] = c.discount * static_cast<double>(val);
        }
        // the five states in FP64
        const double n = static_cast<double>(c.n_steps);
        const double le = static_cast<double>(__expf(x));  // S_n / S0
        const double em_up_n = static_cast<double>(expm1_small(e_up));
        const double em_dn_n = static_cast<double>(expm1_small(e_dn));
        const double last0 = S0 * le;
        const double last[5] = {last0, (S0 + hs) * le, (S0 - hs) * le, last0 + last0 * em_up_n,
                                last0 + last0 * em_dn_n};
        double avg0 = 0.0;
        if constexpr (KIND == kAsianArith || KIND == kAsianGeo) {
            double avg[5];
            if constexpr (KIND == kAsianArith) {
                const double a = static_cast<double>(acc) * g.inv_n;
                avg[0] = S0 * a;
                avg[1] = (S0 + hs) * a;
                avg[2] = (S0 - hs) * a;
                avg[3] = avg[0] + S0 * (static_cast<double>(a_up) * g.inv_n);
                avg[4] = avg[0] + S0 * (static_cast<double>(a_dn) * g.inv_n);
            } else {
                const double gm = exp(static_cast<double>(acc2) * g.inv_n);
                const double dbar = static_cast<double>(sd) * g.inv_n;
                const double ibar = 0.5 * (n + 1.0) * g.dt;  // mean of i dt
                avg[0] = S0 * gm;
                avg[1] = (S0 + hs) * gm;
                avg[2] = (S0 - hs) * gm;
                avg[3] = avg[0] + avg[0] * expm1(hv * dbar - 0.5 * hv * hv * ibar);
                avg[4] = avg[0] + avg[0] * expm1(-hv * dbar - 0.5 * hv * hv * ibar);
            }
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                const double ref = c.floating ? (last[j] - avg[j]) : (avg[j] - K);
                v[j] = disc * dmax(phid * ref, 0.0);
            }
            avg0 = avg[0];
        } else if constexpr (KIND == kBarrier) {
            const bool b[5] = {br, br_su, br_sd, br_vu, br_vd};
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                const double vanilla = dmax(phid * (last[j] - K), 0.0);
                const bool pays = c.out ? !b[j] : b[j];
                v[j] = disc * (pays ? vanilla : c.rebate);
            }
        } else {
            const double hi[5] = {S0 * exp(static_cast<double>(xmax)), (S0 + hs) * exp(static_cast<double>(xmax)),
                                  (S0 - hs) * exp(static_cast<double>(xmax)), S0 * exp(static_cast<double>(xmax_up)),
                                  S0 * exp(static_cast<double>(xmax_dn))};
            const double lo[5] = {S0 * exp(static_cast<double>(xmin)), (S0 + hs) * exp(static_cast<double>(xmin)),
                                  (S0 - hs) * exp(static_cast<double>(xmin)), S0 * exp(static_cast<double>(xmin_up)),
                                  S0 * exp(static_cast<double>(xmin_dn))};
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                if constexpr (KIND == kLookbackFixed)
                    v[j] = disc * (c.type == 0 ? dmax(hi[j] - K, 0.0) : dmax(K - lo[j], 0.0));
                else
                    v[j] = disc * (c.type == 0 ? (last[j] - lo[j]) : (hi[j] - last[j]));
            }
        }
        const double h = v[0];
        const double z1d = static_cast<double>(z1);
        o[kGLrDelta] = h * (z1d * g.lr_delta_scale);
        o[kGLrGamma] = h * ((z1d * z1d - g.vol * g.sqrt_dt * z1d - 1.0) * g.lr_gamma_scale);
        o[kGLrVega] = h * static_cast<double>(lr_vega);
        o[kGLrRho] = h * (g.sqrt_dt_over_vol * static_cast<double>(zsum) - g.time);
        if constexpr (KIND == kAsianArith || KIND == kAsianGeo) {
            const bool arith = KIND == kAsianArith;
            const double d_avg_dspot = avg0 * g.inv_spot;
            const double d_avg_dvol =
                arith ? S0 * static_cast<double>(a_d) * g.inv_n : avg0 * (static_cast<double>(sd) * g.inv_n);
            const double d_avg_drate =
                arith ? S0 * static_cast<double>(a_r) * g.dt * g.inv_n : avg0 * (0.5 * (n + 1.0) * g.dt);
            const double ref = c.floating ? (last0 - avg0) : (avg0 - K);
            const double slope = phid * ref > 0.0 ? phid : 0.0;
            double delta_raw, vega_raw, rate_raw;
            if (!c.floating) {
                delta_raw = slope * d_avg_dspot;
                vega_raw = slope * d_avg_dvol;
                rate_raw = slope * d_avg_drate;
            } else {
                delta_raw = slope * (le - d_avg_dspot);
                vega_raw = slope * (last0 * static_cast<double>(D) - d_avg_dvol);
                rate_raw = slope * (last0 * n * g.dt - d_avg_drate);
            }
            o[kGPwDelta] = disc * delta_raw;
            o[kGPwVega] = disc * vega_raw;
            o[kGPwRho] = disc * rate_raw - g.time * h;
        }
    }
    o[kGFdDelta] = (v[1] - v[2]) * g.inv_2hs;
    o[kGFdGamma] = (v[1] - 2.0 * v[0] + v[2]) * g.inv_hs2;
    o[kGFdVega] = (v[3] - v[4]) * g.inv_2hv;
}

// One slab: shifted sums per thread in path order, as the path engine
// (unit_sums.cuh).  The twelve accumulator pairs live in shared memory
// (acc[0][i][t], acc[1][i][t]) rather than registers: they are touched once per
// path, and the registers go to the path state instead.  Every lane runs every
// round (the step table's refills synchronise the warp); a path past the
// contract's last one is not counted.  Leaves each warp's triples in out.
template <int KIND, bool SER = false>
__device__ void slab_greeks(const DevContract& c, const DevGreeks& g, const PhiloxKeys& k, PhiloxStep* table,
                            uint64_t base, double (*acc)[kNumGreeks][kSlabThreads], double* pivot, Welford* out) {
    const int t = threadIdx.x, lane = t & 31;
    const uint64_t left = c.path_count - base;
    const uint64_t size = static_cast<uint64_t>(kSlabThreads) << c.item_log;
    const int rounds = static_cast<int>(((left < size ? left : size) + kSlabThreads - 1) / kSlabThreads);
    unsigned count = 0;
    for (int j = 0; j < rounds; ++j) {
        const uint64_t path = base + static_cast<uint64_t>(j * kSlabThreads) + t;
        double o[kNumGreeks];
        greeks32<KIND, SER>(c, g, k, table, path, j == 0, o);
        const bool live = path < c.path_count;
        count += live ? 1u : 0u;
#pragma unroll
        for (int i = 0; i < kNumGreeks; ++i) {
            if (j == 0) {
                const double first = __shfl_sync(0xffffffffu, o[i], 0);
                if (lane == 0) pivot[i] = first;
                const double d = live ? o[i] - first : 0.0;
                acc[0][i][t] = d;
                acc[1][i][t] = d * d;
            } else if (live) {
                const double d = o[i] - pivot[i];
                acc[0][i][t] += d;
                acc[1][i][t] = fma(d, d, acc[1][i][t]);
            }
        }
        if (j == 0) __syncwarp();  // pivots written
    }
    count = __reduce_add_sync(0xffffffffu, count);
    double s[kNumGreeks];
    int index;
#pragma unroll
    for (int i = 0; i < kNumGreeks; ++i) s[i] = acc[0][i][t];
    const double a = warp_sums(s, lane, index);
#pragma unroll
    for (int i = 0; i < kNumGreeks; ++i) s[i] = acc[1][i][t];
    const double b = warp_sums(s, lane, index);
    if (index < kNumGreeks) out[index] = unit_triple(count, pivot[index], a, b);
}

__device__ void run_greeks_slab(const DevContract& c, const DevGreeks& g, PhiloxStep* table, uint64_t base,
                                double (*acc)[kNumGreeks][kSlabThreads], double* pivot, Welford* out) {
    const PhiloxKeys k = philox_keys(c.seed);
    switch (c.kind) {
        case kEuropean: slab_greeks<kEuropean>(c, g, k, table, base, acc, pivot, out); break;
        case kDigital: slab_greeks<kDigital>(c, g, k, table, base, acc, pivot, out); break;
        case kAsianArith:
            if (g.vol_series) slab_greeks<kAsianArith, true>(c, g, k, table, base, acc, pivot, out);
            else slab_greeks<kAsianArith, false>(c, g, k, table, base, acc, pivot, out);
            break;
        case kAsianGeo: slab_greeks<kAsianGeo>(c, g, k, table, base, acc, pivot, out); break;
        case kBarrier: slab_greeks<kBarrier>(c, g, k, table, base, acc, pivot, out); break;
        case kLookbackFixed: slab_greeks<kLookbackFixed>(c, g, k, table, base, acc, pivot, out); break;
        default: slab_greeks<kLookbackFloating>(c, g, k, table, base, acc, pivot, out); break;
    }
}

template <int MINB>
__global__ void __launch_bounds__(kSlabThreads, MINB)
    greeks_kernel(const DevContract* __restrict__ contracts, const DevGreeks* __restrict__ greeks, int n_contracts,
                  const uint32_t* __restrict__ item_prefix, uint32_t* __restrict__ ticket, Welford* __restrict__ partials,
                  uint32_t* __restrict__ error_flag) {
    __shared__ uint32_t s_item;
    __shared__ DevContract s_contract;
    __shared__ DevGreeks s_greeks;
    __shared__ double s_acc[2][kNumGreeks][kSlabThreads];
    __shared__ double s_pivot[kSlabThreads / 32][kNumGreeks];
    // A warp's step table, and its triples once the slab's paths are done (27.5
    // KB in all: eight CTAs fit an SM's shared memory).
    __shared__ union {
        PhiloxStep step[32];
        Welford triple[kNumGreeks];
    } s_warp[kSlabThreads / 32];
    const int warp = threadIdx.x >> 5;
    static_assert(sizeof(DevContract) % 4 == 0 && sizeof(DevGreeks) % 4 == 0 &&
                      (sizeof(DevContract) + sizeof(DevGreeks)) / 4 <= 2 * kSlabThreads,
                  "contract staging assumes at most two words per thread");
    const uint32_t first = item_prefix[0], total = item_prefix[n_contracts] - first;
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(ticket, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= total) return;
        int lo = 0, hi = n_contracts;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (item_prefix[mid] - first <= item) lo = mid; else hi = mid;
        }
        for (int i = threadIdx.x; i < static_cast<int>(sizeof(DevContract) / 4); i += kSlabThreads)
            reinterpret_cast<uint32_t*>(&s_contract)[i] = reinterpret_cast<const uint32_t*>(&contracts[lo])[i];
        for (int i = threadIdx.x; i < static_cast<int>(sizeof(DevGreeks) / 4); i += kSlabThreads)
            reinterpret_cast<uint32_t*>(&s_greeks)[i] = reinterpret_cast<const uint32_t*>(&greeks[lo])[i];
        __syncthreads();
        const uint32_t slab = item - (item_prefix[lo] - first);
        if (slab >= s_contract.n_items) {
            if (threadIdx.x == 0) atomicOr(error_flag, 1u);
            __syncthreads();
            continue;
        }
        run_greeks_slab(s_contract, s_greeks, s_warp[warp].step,
                        static_cast<uint64_t>(slab) * kSlabThreads << s_contract.item_log, s_acc,
                        s_pivot[warp], s_warp[warp].triple);
        __syncthreads();
        if (threadIdx.x < kNumGreeks) {
            const int i = threadIdx.x;
            partials[static_cast<size_t>(item) * kNumGreeks + i] =
                merge_warps(s_warp[0].triple[i], s_warp[1].triple[i], s_warp[2].triple[i], s_warp[3].triple[i]);
        }
        __syncthreads();
    }
}

// One CTA per (contract, output): the path engine's merge.
__global__ void __launch_bounds__(kMergeThreads)
    greeks_merge_kernel(const DevContract* __restrict__ contracts, const uint32_t* __restrict__ item_prefix,
                        const Welford* __restrict__ partials, double* __restrict__ out) {
    const int ci = blockIdx.x, gi = blockIdx.y;
    const size_t begin = item_prefix[ci] - item_prefix[0];
    const MergedResult m =
        merge_items(partials + begin * kNumGreeks + gi, item_prefix[ci + 1] - item_prefix[ci], kNumGreeks);
    if (threadIdx.x == 0) {
        double* o = out + static_cast<size_t>(contracts[ci].orig_index) * kGreeksOutStride;
        o[2 * gi] = m.mean;
        o[2 * gi + 1] = m.standard_error;
        if (gi == 0) o[2 * kNumGreeks] = static_cast<double>(m.count);
    }
}

template <int MINB>
cudaError_t launch_one(int grid, const DevContract* c, const DevGreeks* g, int n, const uint32_t* prefix,
                       uint32_t* ticket, Welford* partials, uint32_t* err, cudaStream_t stream) {
    cudaGetLastError();
    greeks_kernel<MINB><<<grid, kSlabThreads, 0, stream>>>(c, g, n, prefix, ticket, partials, err);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_greeks_kernel(int precision, int variant, int grid, const DevContract* contracts,
                                 const DevGreeks* greeks, int n_contracts, const uint32_t* item_prefix,
                                 uint32_t* ticket, Welford* partials, uint32_t* error_flag,
                                 const FixedTables* tables, cudaStream_t stream) {
    if (precision == 0)
        return launch_greeks64_kernel(grid, contracts, greeks, n_contracts, item_prefix, ticket, partials, error_flag,
                                      tables, stream);
#define MCD_GREEKS_ARGS grid, contracts, greeks, n_contracts, item_prefix, ticket, partials, error_flag, stream
    switch (variant) {
        case 0: return launch_one<2>(MCD_GREEKS_ARGS);
        case 1: return launch_one<4>(MCD_GREEKS_ARGS);
        case 2: return launch_one<6>(MCD_GREEKS_ARGS);
        default: return launch_one<8>(MCD_GREEKS_ARGS);
    }
#undef MCD_GREEKS_ARGS
}

cudaError_t launch_greeks_merge(const DevContract* contracts, int n_contracts, const uint32_t* item_prefix,
                                const Welford* partials, double* out, cudaStream_t stream) {
    cudaGetLastError();
    if (n_contracts > 0)
        greeks_merge_kernel<<<dim3(static_cast<unsigned>(n_contracts), kNumGreeks), kMergeThreads, 0, stream>>>(
            contracts, item_prefix, partials, out);
    return cudaGetLastError();
}

cudaError_t greeks_kernel_occupancy(int precision, int variant, int* blocks) {
    if (precision == 0) {  // one CTA per SM shares the fixed-point tables
        *blocks = 1;
        return cudaSuccess;
    }
    switch (variant) {
        case 0: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, greeks_kernel<2>, kSlabThreads, 0);
        case 1: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, greeks_kernel<4>, kSlabThreads, 0);
        case 2: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, greeks_kernel<6>, kSlabThreads, 0);
        default: return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, greeks_kernel<8>, kSlabThreads, 0);
    }
}

}  // namespace mcdg
