// Host check of the 113-bit integer arithmetic (cdet_widefloat.cuh) against
// binary128 (113 significand bits, one rounding): products, base - l r with
// and without cancellation, inverses, and the packed format's round trip and
// ordering, over random operands, powers of two, all-ones mantissas, equal and
// far-apart exponents, and zeros. Prints the worst relative errors in units of
// 2^-112 and exits non-zero when one exceeds its bound.
#include "cdet_widefloat.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

using namespace cdet;
#ifdef __SIZEOF_FLOAT128__
typedef __float128 f128;
#else
typedef long double f128;  // binary128 on aarch64
#endif

static std::mt19937_64 rng(20261205);

static f128 two(int e) {
    f128 r = 1;
    for (; e > 0; --e) r *= 2;
    for (; e < 0; ++e) r /= 2;
    return r;
}
static f128 value(const Wide& a) {
    f128 v = 0;
    for (int i = 3; i >= 0; --i) v = v * two(32) + static_cast<f128>(a.m[i]);
    v *= two(a.e - 127);
    return a.sign ? -v : v;
}
static bool is_zero(const WidePacked& q) { return (q.x | q.y | q.z | q.w) == 0; }
static f128 value(const WidePacked& q) { return is_zero(q) ? f128(0) : value(wide_unpack(q)); }

static Wide random_wide(int kind, int spread) {
    Wide a;
    for (int i = 0; i < 4; ++i) a.m[i] = static_cast<uint32_t>(rng());
    a.m[3] = (a.m[3] & 0x3FFFFFFFu) | 0x40000000u;
    a.m[0] &= ~0x3FFFu;  // the 113 bits a stored number has
    if (kind == 1) a.m[0] = a.m[1] = a.m[2] = 0, a.m[3] = 0x40000000u;
    if (kind == 2) a.m[0] = 0xFFFFC000u, a.m[1] = a.m[2] = 0xFFFFFFFFu, a.m[3] = 0x7FFFFFFFu;
    if (kind == 3) a.m[0] = a.m[1] = 0, a.m[2] &= 0xFFFFFC00u;  // a double
    a.e = static_cast<int>(rng() % (2 * spread + 1)) - spread;
    a.sign = rng() & 1;
    return a;
}
static f128 absq(f128 x) { return x < 0 ? -x : x; }

int main() {
    const f128 unit = two(-112);
    double worst_mul = 0, worst_sub = 0, worst_inv = 0;
    long bad = 0;
    auto recip = [] __host__ __device__(uint64_t bits) {
        double d;
        std::memcpy(&d, &bits, 8);
        d = 1.0 / d;
        uint64_t r;
        std::memcpy(&r, &d, 8);
        return r;
    };
    for (int it = 0; it < 400000; ++it) {
        const int spreads[] = {0, 2, 40, 120, 1000};
        const Wide a = random_wide(static_cast<int>(rng() % 4), spreads[rng() % 5]);
        const Wide b = random_wide(static_cast<int>(rng() % 4), spreads[rng() % 5]);
        Wide c = random_wide(static_cast<int>(rng() % 4), spreads[rng() % 5]);
        if (value(wide_pack(a)) != value(a)) ++bad;  // the stored format is exact on 113 bits
        const WidePacked pa = wide_pack(a), pb = wide_pack(b);
        if (wide_abs_le(pa, pb) != (absq(value(a)) <= absq(value(b)))) ++bad;
        const f128 prod = value(a) * value(b);
        worst_mul = std::fmax(worst_mul, static_cast<double>(absq(value(wide_pack(wide_mul(a, b))) - prod) / (absq(prod) * unit)));
        if (rng() % 3 == 0) {  // cancellation: c near a b
            c = wide_unpack(wide_pack(wide_mul(a, b)));
            const int flip = static_cast<int>(rng() % 113);
            c.m[(14 + flip) / 32] ^= 1u << ((14 + flip) % 32);
            c.m[3] |= 0x40000000u;
            c.m[3] &= 0x7FFFFFFFu;
        }
        // against the larger of the two terms: what the subtraction can know
        const f128 want = value(c) - prod;
        const f128 scale = absq(value(c)) > absq(prod) ? absq(value(c)) : absq(prod);
        const f128 got = value(wide_pack(wide_sub_prod(a, b, c)));
        worst_sub = std::fmax(worst_sub, static_cast<double>(absq(got - want) / (scale * unit)));
        const f128 inv = 1 / value(a);
        worst_inv = std::fmax(worst_inv, static_cast<double>(absq(value(wide_pack(wide_inverse(a, recip))) - inv) / (absq(inv) * unit)));
    }
    // zeros: products with zero stay below every number, sums ignore them
    const WidePacked zero{0, 0, 0, 0};
    const Wide z = wide_unpack(zero);
    for (int it = 0; it < 1000; ++it) {
        const Wide a = random_wide(0, 900), b = random_wide(0, 900);
        if (!is_zero(wide_pack(wide_mul(z, a))) || !is_zero(wide_pack(wide_mul(z, z)))) ++bad;
        if (value(wide_pack(wide_sub_prod(z, a, b))) != value(b)) ++bad;
        if (!is_zero(wide_pack(wide_sub_prod(z, z, z)))) ++bad;
        Wide na = a;
        na.sign ^= 1;
        if (!is_zero(wide_pack(wide_add(a, na)))) ++bad;
        const double d = std::ldexp(static_cast<double>(rng() >> 11), static_cast<int>(rng() % 1900) - 1000);
        uint64_t bits;
        std::memcpy(&bits, &d, 8);
        if (std::fpclassify(d) == FP_NORMAL && value(wide_from_bits(bits)) != static_cast<f128>(d)) ++bad;
    }
    std::printf("worst errors (2^-112): product %.2f, base - l r %.2f, inverse %.2f; %ld violations\n", worst_mul,
                worst_sub, worst_inv, bad);
    return (bad || worst_mul > 2.0 || worst_sub > 2.5 || worst_inv > 2.0) ? 1 : 0;
}
