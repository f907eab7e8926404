// Host check of the integer-pipe FP64 reciprocal (cdet_softmul.cuh): wherever it
// reports no exception its bits are those of the IEEE quotient 1 / b, for
// random and short significands, significands next to powers of two, the ends
// of the exponent range, and seeds one unit of their last place either way;
// values outside the range must be reported. Prints the numbers checked,
// reported and wrong; exits non-zero if one is wrong or too many are reported.
#include "cdet_softmul.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

int main() {
    std::mt19937_64 rng(20261205);
    auto bits = [](double d) { uint64_t u; std::memcpy(&u, &d, 8); return u; };
    auto value = [](uint64_t u) { double d; std::memcpy(&d, &u, 8); return d; };
    const uint64_t frac = (uint64_t{1} << 52) - 1;
    long wrong = 0, reported = 0, checked = 0, ordinary_reported = 0, missed = 0;
    auto check = [&](double b, bool ordinary) {
        const uint64_t bb = bits(b);
        const uint32_t arg = cdet::soft_rcp_arg(static_cast<uint32_t>(bb >> 32), static_cast<uint32_t>(bb));
        float f;
        std::memcpy(&f, &arg, 4);
        volatile float r = 1.0f / f;
        float rf = r;
        uint32_t seed;
        std::memcpy(&seed, &rf, 4);
        for (int off = -1; off <= 1; ++off) {
            uint32_t hi = 0, lo = 0;
            bool bad = false;
            cdet::soft_rcp_bits(static_cast<uint32_t>(bb >> 32), static_cast<uint32_t>(bb), seed + off, hi, lo, bad);
            ++checked;
            if (bad) {
                ++reported;
                ordinary_reported += ordinary;
                continue;
            }
            const int field = static_cast<int>((bb >> 52) & 0x7FF);
            if (field < 1 || field > 2044 || (bb & frac) == 0) ++missed;
            volatile double want = 1.0 / b;
            if (bits(want) != ((static_cast<uint64_t>(hi) << 32) | lo)) ++wrong;
        }
    };
    for (int i = 0; i < 4000000; ++i) {
        const uint64_t sign = rng() & (uint64_t{1} << 63), field = 1 + rng() % 2043, m = rng() & frac;
        check(value(sign | (field << 52) | m | 1), true);
        check(value(sign | (field << 52) | (m & ~((uint64_t{1} << (rng() % 53)) - 1))), false);
        check(value(sign | (field << 52) | (m >> (rng() % 53))), false);         // just above a power of two
        check(value(sign | (field << 52) | (frac ^ (m >> (rng() % 53)))), false);  // just below one
    }
    for (uint64_t m = 0; m < 4096; ++m) {
        check(value((uint64_t{1023} << 52) | m), m != 0);
        check(value((uint64_t{1023} << 52) | (frac - m)), true);
        check(value((uint64_t{1023} << 52) | (m << 40)), false);
    }
    for (double b : {0.0, -0.0, 5e-324, 2.2250738585072009e-308, 1.7976931348623157e308, 1e308, 4.5e307, -9e307,
                     (double)INFINITY, -(double)INFINITY, (double)NAN, 1.0, -2.0, 0.5})
        check(b, false);
    std::printf("%ld reciprocals, %ld reported, %ld ordinary reported, %ld wrong, %ld not reported\n", checked, reported,
                ordinary_reported, wrong, missed);
    return (wrong || missed || ordinary_reported > 4) ? 1 : 0;
}
