// fixed_math.hpp -- 64-bit fixed-point normal quantile and exponential for the
// FP64 paths (host and device).
//
// Why integers.  An FP64 operation on this GPU issues at 1.7 lanes per clock
// and SM (measured: DFMA, DADD and DMUL alike), a 32x32->64-bit integer
// multiply-add at 25-31 and a 32-bit one at 62.  A 64-bit fixed-point
// multiply is two or three of the former, so the quantile, the log-spot and
// the exponential of a path step cost less in 64-bit integers than a single
// DFMA, and carry 61 to 64 bits instead of 53.
//
// Quantile.  A draw's 32 random bits give q = min(u, 1-u) = w / 2^33 with w an
// odd 32-bit integer (Philox, u = (bits + 1/2) / 2^32) or an even one (Sobol,
// u = x / 2^32).  -Phi^-1(q) is tabulated per interval of w: 32 octaves of 512
// intervals each, a polynomial of degree 4 per interval in s in [0, 1), the
// distance from the interval's right end.  In that variable every coefficient
// is non-negative, so the evaluation is unsigned throughout.  Truncation error
// of the polynomials: below 2^-56 (the FP64 quantile of the reference, Acklam
// and one Halley step, is good to about 3e-16 near the centre and to 1e-16 /
// phi(z) in the upper tail).
//
// Log-spots are kept in base 2 as signed 64-bit integers in units of 2^-F, F
// chosen per contract so that no path can overflow (host, fixed_scale).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define MCD_HD __host__ __device__ __forceinline__
#else
#define MCD_HD inline
#endif

namespace mcdg {

constexpr int kQuantSubBits = 9;                      // intervals per octave: 2^9
constexpr int kQuantSub = 1 << kQuantSubBits;
constexpr int kQuantOctaves = 32;                     // w in [1, 2^32)
constexpr int kQuantEntries = kQuantOctaves * kQuantSub;
// Octaves held in shared memory (5120 entries, 160 KB): q >= 2^-11.  One draw
// in 1024 reads the rest of the table from global memory.
constexpr int kQuantSharedOctaves = 10;
constexpr int kQuantShared = kQuantSharedOctaves * kQuantSub;

// One interval: value = c0 + s (c1 + s (c2 + s (c3 + s c4))), units of 2^-61.
// Two 16-byte halves kept in separate arrays, so that a warp's gathers spread
// over all banks.
struct alignas(16) QuantLo {
    uint64_t c0, c1;
};
struct alignas(16) QuantHi {
    uint64_t c2;
    uint32_t c3, c4;
};

constexpr int kExpBits = 10;  // 2^x by two tables of 2^10 entries and a quadratic
constexpr int kExpEntries = 1 << kExpBits;

constexpr int kLogBits = 10;  // logarithm: intervals of [1, 2) (fixed_root.hpp)
constexpr int kLogEntries = 1 << kLogBits;

struct FixedTables {
    QuantLo lo[kQuantEntries];
    QuantHi hi[kQuantEntries];
    uint64_t exp_a[kExpEntries];  // 2^(i / 2^10), units of 2^-63
    uint64_t exp_b[kExpEntries];  // 2^(i / 2^20) - 1, units of 2^-64
    alignas(16) uint64_t log_l[kLogEntries];  // -ln(c 2^-31), units of 2^-59
    uint32_t log_c[kLogEntries];              // 1 / (1 + i / 2^10) rounded up, units of 2^-31
};

MCD_HD uint32_t mul_hi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return static_cast<uint32_t>((static_cast<uint64_t>(a) * b) >> 32);
#endif
}

MCD_HD int count_lz32(uint32_t x) {  // x != 0
#ifdef __CUDA_ARCH__
    return __clz(static_cast<int>(x));
#else
    return __builtin_clz(x);
#endif
}

// High 64 bits of a 64x64-bit product without the low-by-low term, plus one:
// within 1 unit of the exact value and centred on it (the three truncations
// lose 1.25 units on average).
MCD_HD uint64_t mul_hi64(uint64_t a, uint64_t b) {
    const uint32_t ah = static_cast<uint32_t>(a >> 32), al = static_cast<uint32_t>(a);
    const uint32_t bh = static_cast<uint32_t>(b >> 32), bl = static_cast<uint32_t>(b);
    const uint64_t hh = static_cast<uint64_t>(ah) * bh;
    return hh + mul_hi32(ah, bl) + mul_hi32(al, bh) + 1u;
}

// s (32-bit fraction) times p, p in any unit: s * p, at most 1 unit low.
MCD_HD uint64_t mul_frac(uint32_t s, uint64_t p) {
    return static_cast<uint64_t>(s) * static_cast<uint32_t>(p >> 32) + mul_hi32(s, static_cast<uint32_t>(p));
}

// Where a quantile argument w (1 <= w < 2^32, q = w / 2^33) lies: table entry
// and distance s from the interval's right end.
struct QuantArg {
    uint32_t entry, s;
};
MCD_HD QuantArg quant_arg(uint32_t w) {
    const int lz = count_lz32(w);
    const uint32_t n = w << lz;
    QuantArg a;
    a.entry = static_cast<uint32_t>(lz) * kQuantSub + ((n >> (31 - kQuantSubBits)) & (kQuantSub - 1));
    a.s = ~(n << (kQuantSubBits + 1));
    return a;
}

// -Phi^-1(q) in units of 2^-61.
MCD_HD uint64_t quant_eval(const QuantLo& lo, const QuantHi& hi, uint32_t s) {
    const uint32_t p3 = hi.c3 + mul_hi32(s, hi.c4);
    const uint64_t p2 = hi.c2 + mul_hi32(s, p3);
    const uint64_t p1 = lo.c1 + mul_frac(s, p2);
    return lo.c0 + mul_frac(s, p1);
}

// 2^f for a 64-bit fraction f: the significand in [1, 2), units of 2^-63.
// f = i / 2^10 + j / 2^20 + t 2^-20: two table factors, and 2^(t 2^-20) - 1 by
// its quadratic (the cubic term is below 2^-64).
MCD_HD uint64_t exp2_frac(uint64_t f, uint64_t a, uint64_t b) {
    constexpr uint64_t e1 = 12193974156573ull;  // ln 2 2^-20, units of 2^-64
    constexpr uint32_t e2 = 4030332u;           // (ln 2)^2 / 2 2^-40
    const uint64_t t = f << (2 * kExpBits);
    const uint32_t th = static_cast<uint32_t>(t >> 32), tl = static_cast<uint32_t>(t);
    const uint64_t p1 = e1 + mul_hi32(th, e2);
    const uint64_t e = mul_frac(th, p1) + mul_hi32(tl, static_cast<uint32_t>(p1 >> 32));  // < 2^-20.5
    // (1 + b)(1 + e) - 1; b e as a 32-bit product of their leading bits
    const uint32_t be = mul_hi32(static_cast<uint32_t>(b >> 22), static_cast<uint32_t>(e >> 12));  // units of 2^-62
    const uint64_t x = b + e + (static_cast<uint64_t>(be) << 2);
    return a + mul_hi64(a, x);
}
MCD_HD uint32_t exp2_index_a(uint64_t f) { return static_cast<uint32_t>(f >> (64 - kExpBits)); }
MCD_HD uint32_t exp2_index_b(uint64_t f) {
    return static_cast<uint32_t>(f >> (64 - 2 * kExpBits)) & (kExpEntries - 1);
}

// The bits of the double m 2^(e - 63), m in [2^63, 2^64), rounded to nearest
// (ties up); e in the normal range.
MCD_HD uint64_t double_bits(uint64_t m, int e) {
    return (static_cast<uint64_t>(static_cast<uint32_t>(e + 1022)) << 52) + (m >> 11) + ((m >> 10) & 1u);
}

}  // namespace mcdg
