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

// Tables of the CTA: the quantile's first kQuantSharedOctaves octaves and both
// exponential tables (176 KB).
struct FixedShared {
    QuantLo lo[kQuantShared];
    QuantHi hi[kQuantShared];
    uint64_t exp_a[kExpEntries];
    uint64_t exp_b[kExpEntries];
};

// Copies the tables into shared memory (asynchronous 16-byte copies by the
// whole CTA; ends with a barrier).
__device__ __forceinline__ void load_fixed_tables(FixedShared& s, const FixedTables* __restrict__ g) {
    auto copy = [](void* to, const void* from, int bytes) {
        for (int o = threadIdx.x * 16; o < bytes; o += blockDim.x * 16)
            cp_async16(static_cast<char*>(to) + o, static_cast<const char*>(from) + o);
    };
    copy(s.lo, g->lo, sizeof s.lo);
    copy(s.hi, g->hi, sizeof s.hi);
    copy(s.exp_a, g->exp_a, sizeof s.exp_a);
    copy(s.exp_b, g->exp_b, sizeof s.exp_b);
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
}

// -Phi^-1(w / 2^33) in units of 2^-61, 1 <= w < 2^32.
__device__ __forceinline__ uint64_t quantile_units(uint32_t w, const FixedShared& s,
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
__device__ __forceinline__ FixedNormal normal_fixed(uint32_t bits, const FixedShared& s,
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

// Philox4x32-10 word 0 with round 0 and the products of round 1 taken apart:
// of the counter {path_lo, path_hi, draw, stream} round 0 mixes the path and
// the stream into words 2 and 3 and the draw into words 0 and 1, so round 1's
// two products depend on the draw alone (PhiloxStep: one per warp and step,
// path_hi being the same for a unit of paths) and on the path alone
// (PhiloxRow: once per path).  A draw is left with rounds 2 to 9: 13 wide
// products instead of 18.
struct alignas(16) PhiloxStep {
    uint32_t a, b, c;  // lo(M1 draw) ^ k0[1], hi(M0 w0) ^ k1[1], lo(M0 w0) ^ k1[2]
    uint32_t carry;    // this step's carry of the drift's fraction below 2^-F (drift_carry)
};
struct PhiloxRow {
    uint32_t a, b, c;  // hi(M1 w2), lo(M1 w2) ^ k0[2], lo(M0 path_lo)
};

__device__ __forceinline__ PhiloxStep philox_step(uint32_t draw, uint32_t path_hi, const PhiloxKeys& k) {
    const uint64_t p = static_cast<uint64_t>(kPhiloxM1) * draw;
    const uint32_t w0 = static_cast<uint32_t>(p >> 32) ^ path_hi ^ k.k0[0];
    const uint64_t q = static_cast<uint64_t>(kPhiloxM0) * w0;
    return PhiloxStep{static_cast<uint32_t>(p) ^ k.k0[1], static_cast<uint32_t>(q >> 32) ^ k.k1[1],
                      static_cast<uint32_t>(q) ^ k.k1[2], 0u};
}

// A drift of hi + lo 2^-32 units per step: what step d adds to d whole steps'
// hi when the running sum of lo is cut to whole units (0 or 1), so that the
// drift's rounding does not add up over the steps.
__device__ __forceinline__ uint32_t drift_carry(uint32_t d, uint32_t lo) {
    return static_cast<uint32_t>((static_cast<uint64_t>(d) * lo & 0xFFFFFFFFull) + lo >> 32);
}

__device__ __forceinline__ PhiloxRow philox_row(uint32_t path_lo, uint32_t stream, const PhiloxKeys& k) {
    const uint64_t p = static_cast<uint64_t>(kPhiloxM0) * path_lo;
    const uint32_t w2 = static_cast<uint32_t>(p >> 32) ^ stream ^ k.k1[0];
    const uint64_t q = static_cast<uint64_t>(kPhiloxM1) * w2;
    return PhiloxRow{static_cast<uint32_t>(q >> 32), static_cast<uint32_t>(q) ^ k.k0[2], static_cast<uint32_t>(p)};
}

__device__ __forceinline__ uint32_t philox_word0(const PhiloxRow& r, const PhiloxStep& s, const PhiloxKeys& k) {
    uint32_t c0 = r.a ^ s.a, c2 = r.c ^ s.b;
    uint32_t x1 = r.b, x3 = s.c;  // words 1 and 3 with the next round's keys
#pragma unroll
    for (int i = 2; i < 8; ++i) {
        const uint64_t p0 = static_cast<uint64_t>(kPhiloxM0) * c0;
        const uint64_t p1 = static_cast<uint64_t>(kPhiloxM1) * c2;
        c0 = static_cast<uint32_t>(p1 >> 32) ^ x1;
        c2 = static_cast<uint32_t>(p0 >> 32) ^ x3;
        x1 = static_cast<uint32_t>(p1) ^ k.k0[i + 1];
        x3 = static_cast<uint32_t>(p0) ^ k.k1[i + 1];
    }
    const uint32_t w2 = __umulhi(kPhiloxM0, c0) ^ x3;
    return __umulhi(kPhiloxM1, w2) ^ (kPhiloxM1 * c2) ^ k.k0[9];
}

}  // namespace mcdg
