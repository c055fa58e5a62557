// fixed_path.cuh -- device side of the FP64 paths in 64-bit fixed point
// (fixed_math.hpp): the tables in shared memory, Philox draws with the parts
// that do not depend on the path computed once per warp and step, and the
// log-spot step.  The kernels that use it run one warp per unit of paths, up
// to 32 warps sharing one copy of the tables.
#pragma once

#include "cp_async.cuh"
#include "device_common.cuh"
#include "fixed_math.hpp"

namespace mcdg {

// Tables of the CTA: the quantile's first kQuantSharedOctaves octaves (160 KB)
// and both exponential tables (16 KB).
struct QuantTables {
    QuantLo lo[kQuantShared];
    QuantHi hi[kQuantShared];
};
struct FixedShared : QuantTables {
    uint64_t exp_a[kExpEntries];
    uint64_t exp_b[kExpEntries];
};

// Starts a table's copy into shared memory (asynchronous 16-byte copies by the
// whole CTA).
__device__ __forceinline__ void copy_table(void* to, const void* from, int bytes) {
    for (int o = threadIdx.x * 16; o < bytes; o += blockDim.x * 16)
        cp_async16(static_cast<char*>(to) + o, static_cast<const char*>(from) + o);
}
__device__ __forceinline__ void copy_quantile(QuantTables& s, const FixedTables* __restrict__ g) {
    copy_table(s.lo, g->lo, sizeof s.lo);
    copy_table(s.hi, g->hi, sizeof s.hi);
}
__device__ __forceinline__ void wait_tables() {
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
}
__device__ __forceinline__ void load_fixed_tables(FixedShared& s, const FixedTables* __restrict__ g) {
    copy_quantile(s, g);
    copy_table(s.exp_a, g->exp_a, sizeof s.exp_a);
    copy_table(s.exp_b, g->exp_b, sizeof s.exp_b);
    wait_tables();
}

// -Phi^-1(w / 2^33) in units of 2^-61, 1 <= w < 2^32.
__device__ __forceinline__ uint64_t quantile_units(uint32_t w, const QuantTables& s,
                                                   const FixedTables* __restrict__ g) {
    const QuantArg a = quant_arg(w);
    const uint32_t i = min(a.entry, static_cast<uint32_t>(kQuantShared - 1));
    QuantLo lo = s.lo[i];
    QuantHi hi = s.hi[i];
    if (a.entry >= static_cast<uint32_t>(kQuantShared)) {  // q < 2^-11: one draw in 1024
        lo.c0 = __ldg(&g->lo[a.entry].c0);
        lo.c1 = __ldg(&g->lo[a.entry].c1);
        hi.c2 = __ldg(&g->hi[a.entry].c2);
        hi.c3 = __ldg(&g->hi[a.entry].c3);
        hi.c4 = __ldg(&g->hi[a.entry].c4);
    }
    return quant_eval(lo, hi, a.s);
}

// The normal of 32 Philox bits, u = (bits + 1/2) / 2^32: magnitude in units of
// 2^-61 and the sign (all ones when negative).
struct FixedNormal {
    uint64_t mag;
    int32_t neg;
};
__device__ __forceinline__ FixedNormal normal_fixed(uint32_t bits, const QuantTables& s,
                                                    const FixedTables* __restrict__ g) {
    const int32_t upper = static_cast<int32_t>(bits) >> 31;
    const uint32_t m = bits ^ static_cast<uint32_t>(upper);
    return FixedNormal{quantile_units(2u * m + 1u, s, g), ~upper};
}

// The same normal rounded to a double.
__device__ __forceinline__ double normal_to_double(const FixedNormal& z) {
    const int lz = __clzll(static_cast<long long>(z.mag | 1u));
    const uint64_t m = z.mag << lz;
    const uint64_t b = double_bits(m, 2 - lz) | (static_cast<uint64_t>(z.neg & 0x80000000) << 32);
    return __longlong_as_double(static_cast<long long>(b));
}

// +/- scale * |z|: scale is (value per unit normal) 2^(F + 3), the result in
// units of 2^-F.
__device__ __forceinline__ int64_t scaled_normal(const FixedNormal& z, uint64_t scale) {
    const uint64_t p = mul_hi64(scale, z.mag);
    const uint64_t m = static_cast<uint64_t>(static_cast<int64_t>(z.neg));
    return static_cast<int64_t>((p ^ m) - m);
}

// 2^y of a log-spot in units of 2^-F (|y| < 2^9), rounded to a double.
__device__ __forceinline__ double exp2_units(int64_t y, int frac, const FixedShared& s) {
    const uint64_t f = static_cast<uint64_t>(y) << (64 - frac);
    const uint64_t m = exp2_frac(f, s.exp_a[exp2_index_a(f)], s.exp_b[exp2_index_b(f)]);
    return __longlong_as_double(static_cast<long long>(double_bits(m, static_cast<int>(y >> frac))));
}

// A drift of hi + lo 2^-32 units per step: what step d adds to d whole steps'
// hi when the running sum of lo is cut to whole units (0 or 1), so that the
// drift's rounding does not add up over the steps.
__device__ __forceinline__ uint32_t drift_carry(uint32_t d, uint32_t lo) {
    return static_cast<uint32_t>((static_cast<uint64_t>(d) * lo & 0xFFFFFFFFull) + lo >> 32);
}

}  // namespace mcdg
