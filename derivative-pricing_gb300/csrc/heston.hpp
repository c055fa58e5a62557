// heston.hpp -- Heston QE batch: per-set constants shared by host and device.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "engine.hpp"

namespace mcdg {

// One parameter set, with the reference's per-step constants precomputed on
// the host in its operation order (src/pricers/heston.cpp:95-99, :123-132).
struct HestonSet {
    double spot, v0, theta, kappa, xi;
    double e;          // exp(-kappa dt)
    double s2_const;   // theta xi^2 / (2 kappa) (1-e)^2
    double drift;      // (r - q) dt
    double k0, k1, k2, k3, k4;
    double discount;   // exp(-r T)
    double log_s0;     // ln S0
    double s2_lin;     // xi^2 e / kappa (1-e)   (FP32 path: s2 = v s2_lin + s2_const)
    // FP64 path (heston64.cu): psi = r (qe_b - qe_a r) with r = 1 / E[v'], and
    double qe_a, qe_b;  // theta xi^2 (1-e)^2 / (2 kappa), xi^2 (1-e) / kappa
    double reversion;   // theta (1-e): E[v'] = v e + reversion
    // ln(S_T / S_0) = drift_sum + k12 sum(v) + k2 (v_n - v_0) + root_k3 sum(z sqrt(v + v'))
    double drift_sum, k12, root_k3;
    uint64_t seed;
    uint64_t path_count;
    uint32_t n_slabs;
    int32_t n_steps;
};
constexpr int kHestonMaxStrikes = 256;

// FP32 view used inside the FP32 kernel.
struct HestonSet32 {
    float s0, v0, theta, e, s2_lin, s2_const, c0, k1, k2, k3, k4;
};

__host__ __device__ inline HestonSet32 make_set32(const HestonSet& h) {
    HestonSet32 r;
    r.s0 = static_cast<float>(h.spot);
    r.v0 = static_cast<float>(h.v0);
    r.theta = static_cast<float>(h.theta);
    r.e = static_cast<float>(h.e);
    r.s2_lin = static_cast<float>(h.s2_lin);
    r.s2_const = static_cast<float>(h.s2_const);
    r.c0 = static_cast<float>(h.drift + h.k0);
    r.k1 = static_cast<float>(h.k1);
    r.k2 = static_cast<float>(h.k2);
    r.k3 = static_cast<float>(h.k3);
    r.k4 = static_cast<float>(h.k4);
    return r;
}

// Items of a set: slabs of 4096 paths (FP32) or units of 32 << unit_log paths
// (FP64); one Welford triple per (item, strike).  The merge folds them per
// (set, strike) into {price, standard error, count}.
cudaError_t launch_heston32(int grid, const HestonSet* sets, int n_sets, const double* strikes, int n_strikes,
                            int type, uint32_t items_per_set, uint32_t* ticket, Welford* partials,
                            cudaStream_t stream);
cudaError_t launch_heston64(int grid, const HestonSet* sets, int n_sets, const double* strikes, int n_strikes,
                            int type, uint32_t units_per_set, int unit_log, uint32_t* ticket, Welford* partials,
                            const FixedTables* tables, cudaStream_t stream);
cudaError_t launch_heston_merge(int n_sets, int n_strikes, uint32_t items_per_set, const Welford* partials,
                                double* out, cudaStream_t stream);
cudaError_t heston32_occupancy(int* blocks);

}  // namespace mcdg
