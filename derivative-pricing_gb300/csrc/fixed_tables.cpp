// fixed_tables.cpp -- the tables of fixed_math.hpp, computed once per process
// in double-double arithmetic and placed in each device's table array.
//
// The quantile z(q) = Phi^-1 satisfies z' = y, y' = z y^2 with y = 1 / phi(z)
// (Steinbrecher and Shaw, "Quantile mechanics", European Journal of Applied
// Mathematics 19, 2008), so its Taylor coefficients at a point follow from z
// and y there by Cauchy products, and the series carries z and y to the next
// interval: from q = 1/2, where z = 0 and y = sqrt(2 pi), to q = 2^-33 without
// an exponential or an error function.  An error in q made on the way stays
// as it is (10^-28 at the end); each interval's degree-5 Taylor term is folded into the lower
// ones by the Chebyshev polynomial of that degree (error c5 / 512).
#include "fixed_tables.hpp"

#include <cmath>

namespace mcdg {

namespace {

struct DD {
    double h, l;
};
DD quick(double a, double b) {
    const double s = a + b;
    return {s, b - (s - a)};
}
DD add(DD a, DD b) {
    const double s = a.h + b.h, t = s - a.h;
    return quick(s, ((a.h - (s - t)) + (b.h - t)) + a.l + b.l);
}
DD mul(DD a, DD b) {
    const double p = a.h * b.h;
    return quick(p, std::fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
DD scale(DD a, double pow2) { return {a.h * pow2, a.l * pow2}; }
DD div_small(DD a, double k) {  // a / k, k a small integer
    const double q = a.h / k;
    const double r = std::fma(-q, k, a.h);
    return quick(q, (r + a.l) / k);
}
// Nearest integer of a * 2^e (a >= 0; slightly negative values give 0).
uint64_t to_units(DD a, int e) {
    const DD x = scale(a, std::ldexp(1.0, e));
    const double f = std::floor(x.h);
    const double rest = (x.h - f) + x.l + 0.5;
    const double whole = std::floor(rest);
    if (f + whole <= 0.0) return 0;
    return static_cast<uint64_t>(f) + static_cast<uint64_t>(static_cast<int64_t>(whole));
}

constexpr int kOrder = 11;  // Taylor terms: (2^-9)^12 = 2^-108

void series(DD z0, DD y0, DD (&z)[kOrder + 1], DD (&y)[kOrder + 1]) {
    DD v[kOrder + 1];  // z y
    z[0] = z0;
    y[0] = y0;
    for (int k = 0; k < kOrder; ++k) {
        DD s{0.0, 0.0}, t{0.0, 0.0};
        for (int j = 0; j <= k; ++j) s = add(s, mul(z[j], y[k - j]));
        v[k] = s;
        for (int j = 0; j <= k; ++j) t = add(t, mul(v[j], y[k - j]));
        z[k + 1] = div_small(y[k], k + 1);
        y[k + 1] = div_small(t, k + 1);
    }
}

DD eval(const DD (&c)[kOrder + 1], DD h) {
    DD r = c[kOrder];
    for (int k = kOrder - 1; k >= 0; --k) r = add(mul(r, h), c[k]);
    return r;
}

void fill_quantile(FixedTables& t) {
    DD z{0.0, 0.0}, y{2.506628274631000502415765284811, -1.8328579980459167e-16};  // sqrt(2 pi)
    DD zs[kOrder + 1], ys[kOrder + 1];
    double at = 0.5, at_low = 0.0;  // the series' point: at + at_low
    series(z, y, zs, ys);
    for (int oct = 0; oct < kQuantOctaves; ++oct) {
        const double a = std::ldexp(1.0, -(oct + 2)), width = a / kQuantSub;
        for (int i = kQuantSub - 1; i >= 0; --i) {
            // right end of the interval, less the last 2^-32 of it (s = ~fraction)
            const double right = a + width * (i + 1), low = -std::ldexp(width, -32);
            const DD h = quick(right - at, low - at_low);
            z = eval(zs, h);
            y = eval(ys, h);
            at = right;
            at_low = low;
            series(z, y, zs, ys);
            // f(s) = -z(right - width s): c_k = -z_k (-width)^k
            DD c[6];
            double w = 1.0;
            for (int k = 0; k < 6; ++k) {
                c[k] = scale(zs[k], -w);
                w *= -width;
            }
            // s^5 = (1280 s^4 - 1120 s^3 + 400 s^2 - 50 s + 1) / 512 + T5*(s) / 512
            const double fold[5] = {1.0 / 512, -50.0 / 512, 400.0 / 512, -1120.0 / 512, 1280.0 / 512};
            for (int k = 0; k < 5; ++k) c[k] = add(c[k], DD{c[5].h * fold[k], 0.0});
            const int e = oct * kQuantSub + i;
            t.lo[e].c0 = to_units(c[0], 61);
            t.lo[e].c1 = to_units(c[1], 61);
            t.hi[e].c2 = to_units(c[2], 61);
            t.hi[e].c3 = static_cast<uint32_t>(to_units(c[3], 61));
            t.hi[e].c4 = static_cast<uint32_t>(to_units(c[4], 61));
        }
    }
}

// 2^(i / 2^10) and 2^(i / 2^20) - 1 by the exponential series of i ln 2 / 2^k.
DD expm1(DD x) {
    DD r{0.0, 0.0};
    for (int k = 30; k >= 1; --k) r = div_small(mul(x, add(r, DD{1.0, 0.0})), k);
    return r;
}

void fill_exp(FixedTables& t) {
    const DD ln2{0.693147180559945286226764, 2.319046813846299558417771e-17};
    for (int i = 0; i < kExpEntries; ++i) {
        const DD x = mul(ln2, DD{static_cast<double>(i), 0.0});
        t.exp_a[i] = to_units(add(DD{1.0, 0.0}, expm1(scale(x, 1.0 / (1 << kExpBits)))), 63);
        t.exp_b[i] = to_units(expm1(scale(x, 1.0 / (1 << (2 * kExpBits)))), 64);
    }
}

// Reciprocals of the intervals' left ends, rounded up, and their logarithms:
// one Newton step of exp(x) = c from the library's logarithm (its error squared
// is below 10^-31).
void fill_log(FixedTables& t) {
    for (uint32_t i = 0; i < kLogEntries; ++i) {
        const uint64_t left = kLogEntries + i;
        t.log_c[i] = static_cast<uint32_t>(((1ull << (31 + kLogBits)) + left - 1) / left);
        const double c = std::ldexp(static_cast<double>(t.log_c[i]), -31), x = -std::log(c);  // x >= 0
        // c exp(x) - 1 = (c - 1) + c expm1(x)
        const DD d = add(DD{c - 1.0, 0.0}, mul(DD{c, 0.0}, expm1(DD{x, 0.0})));
        t.log_l[i] = to_units(add(DD{x, 0.0}, DD{-d.h, -d.l}), 59);
    }
}

}  // namespace

// In static storage: mcd_price_batch_static, which allocates nothing and has no
// status for a failed allocation here, needs the tables too.
const FixedTables& fixed_tables() {
    static FixedTables tables;
    static const bool filled = [] {
        fill_quantile(tables);
        fill_exp(tables);
        fill_log(tables);
        return true;
    }();
    static_cast<void>(filled);
    return tables;
}

}  // namespace mcdg
