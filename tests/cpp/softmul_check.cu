// Host check of the integer-pipe FP64 product and sum (cdet_softmul.cuh): wherever
// they report no exception their bits are the IEEE results, for random factors,
// short significands (where ties occur), powers of two, exponents at the ends
// of the accepted ranges, and values outside them, which must be reported.
// Prints the number of products checked, reported and wrong; exits non-zero
// if one is wrong or too many ordinary products are reported.
#include "cdet_softmul.cuh"

#include <cstdio>
#include <cstring>
#include <cmath>
#include <random>

int main() {
    std::mt19937_64 rng(20261205);
    auto bits = [](double d) { uint64_t u; std::memcpy(&u, &d, 8); return u; };
    auto value = [](uint64_t u) { double d; std::memcpy(&d, &u, 8); return d; };
    const uint64_t frac = (uint64_t{1} << 52) - 1;
    long wrong = 0, reported = 0, checked = 0, ordinary_reported = 0, missed = 0;
    auto check = [&](double x, double b, bool ordinary) {
        const uint64_t xb = bits(x), bb = bits(b);
        if (!cdet::soft_factor_in_range(static_cast<uint32_t>(xb >> 32))) return;
        const cdet::SoftFactor f = cdet::soft_factor(static_cast<uint32_t>(xb >> 32), static_cast<uint32_t>(xb));
        uint32_t hi = 0, lo = 0;
        bool bad = false;
        cdet::soft_mul_bits(f, static_cast<uint32_t>(bb >> 32), static_cast<uint32_t>(bb), hi, lo, bad);
        ++checked;
        if (bad) {
            ++reported;
            if (ordinary) ++ordinary_reported;
            return;
        }
        const int field = static_cast<int>((bb >> 52) & 0x7FF);
        if (field < 300 || field > 1700) ++missed;
        volatile double want = x * b;
        if (bits(want) != ((static_cast<uint64_t>(hi) << 32) | lo)) ++wrong;
    };
    for (int i = 0; i < 4000000; ++i) {
        const uint64_t sx = rng() & (uint64_t{1} << 63), sb = rng() & (uint64_t{1} << 63);
        const uint64_t ex = 923 + rng() % 102, eb = 300 + rng() % 1400;
        const double x = value(sx | (ex << 52) | (rng() & frac));
        const double b = value(sb | (eb << 52) | (rng() & frac));
        check(x, b, true);
        // short significands: exact products and ties
        const int keep_x = rng() % 53, keep_b = rng() % 53;
        const double xs = value(bits(x) & ~((uint64_t{1} << keep_x) - 1));
        const double bs = value(bits(b) & ~((uint64_t{1} << keep_b) - 1));
        check(xs, bs, false);
        check(xs, b, false);
        check(x, bs, false);
        // all ones: the carry out of the significand
        check(value(bits(x) | frac), value(bits(b) | (frac >> (rng() % 53))), false);
    }
    const double edge[] = {0.0, -0.0, 5e-324, 2.2250738585072014e-308, 1e-250, 1e300, INFINITY, -INFINITY, NAN, 1.0, -2.0};
    for (double x : {2.0, -2.0, 1.0, 1.5, -0.75, 1.9999999999999998, 1e-29})
        for (double b : edge) check(x, b, false);
    // sums: exponents apart by 0 to 70, both signs, short significands, near cancellation
    auto check_sum = [&](double x, double y, bool ordinary) {
        const uint64_t xb = bits(x), yb = bits(y);
        uint32_t hi = 0, lo = 0;
        bool bad = false;
        cdet::soft_add_bits(static_cast<uint32_t>(xb >> 32), static_cast<uint32_t>(xb), static_cast<uint32_t>(yb >> 32),
                            static_cast<uint32_t>(yb), hi, lo, bad);
        ++checked;
        if (bad) {
            ++reported;
            if (ordinary) ++ordinary_reported;
            return;
        }
        volatile double want = x + y;
        if (bits(want) != ((static_cast<uint64_t>(hi) << 32) | lo)) ++wrong;
    };
    for (int i = 0; i < 6000000; ++i) {
        const uint64_t sx = rng() & (uint64_t{1} << 63), sy = rng() & (uint64_t{1} << 63);
        const int ex = 300 + static_cast<int>(rng() % 1300);
        const int apart = static_cast<int>(rng() % 3 == 0 ? rng() % 4 : rng() % 71);
        const int ey = ex + (rng() & 1 ? apart : -apart);
        const uint64_t fx = rng() & frac, fy = rng() & frac;
        const double x = value(sx | (static_cast<uint64_t>(ex) << 52) | fx);
        const double y = value(sy | (static_cast<uint64_t>(ey) << 52) | fy);
        check_sum(x, y, apart >= 2);
        const int keep_x = rng() % 53, keep_y = rng() % 53;
        const double xs = value(bits(x) & ~((uint64_t{1} << keep_x) - 1)), ys = value(bits(y) & ~((uint64_t{1} << keep_y) - 1));
        check_sum(xs, ys, false);
        check_sum(xs, y, false);
        check_sum(value(bits(x) | frac), y, false);
        check_sum(x, value(bits(y) & ~frac), false);
        check_sum(x, value(bits(-x) ^ (rng() & ((uint64_t{1} << (rng() % 53)) - 1))), false);  // cancelling
    }
    for (double x : edge)
        for (double y : edge) check_sum(x, y, false);
    for (double x : {1.7976931348623157e308, 1e308, 4e-308, 1e-290, 1.0})
        for (double y : {1.7976931348623157e308, -1e308, 4e-308, -3e-308, 1e-323}) check_sum(x, y, false);
    std::printf("%ld products and sums, %ld reported, %ld ordinary reported, %ld wrong, %ld out of range not reported\n", checked,
                reported, ordinary_reported, wrong, missed);
    return (wrong || missed || ordinary_reported > 4) ? 1 : 0;
}
