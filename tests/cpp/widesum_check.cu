// Host check of the connected recursion's sums (WideSum, cdet_widefloat.cuh)
// against binary128: a recursion of order 8 on subset values that are graded
// (one or two vertices scaled by 2^-s, s up to 500, or single subsets, or
// zeros), each mask's sum from the same dp and a; the same sums in parts and
// in another order, bit for bit; on the farthest scale allowed; and the round-off filter's decision. Prints
// the worst error in units of 2^-112 of the sum of the terms' magnitudes and
// exits non-zero when a check fails.
#include "cdet_widefloat.cuh"

#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

using namespace cdet;
#ifdef __SIZEOF_FLOAT128__
typedef __float128 f128;
#else
typedef long double f128;  // binary128 on aarch64
#endif

static std::mt19937_64 rng(4113);

static f128 two(int e) {
    f128 r = 1;
    for (; e > 0; --e) r *= 2;
    for (; e < 0; ++e) r /= 2;
    return r;
}
static f128 value(const Wide& a) {
    if (a.e < kWideZero / 2) return 0;
    f128 v = 0;
    for (int i = 3; i >= 0; --i) v = v * two(32) + static_cast<f128>(a.m[i]);
    v *= two(a.e - 127);
    return a.sign ? -v : v;
}
static Wide random_wide(int e) {
    Wide a;
    for (int i = 0; i < 4; ++i) a.m[i] = static_cast<uint32_t>(rng());
    a.m[3] = (a.m[3] & 0x3FFFFFFFu) | 0x40000000u;
    a.m[0] &= ~0x3FFFu;  // the 113 bits a stored number has
    a.e = e;
    a.sign = rng() & 1;
    return a;
}

struct Term {
    uint32_t m[4];
    int32_t exponent;
    bool negative;
};

// slack: how far above the largest exponent the scale lies
static Wide sum_of(const std::vector<Term>& terms, int parts, bool reversed, double threshold, int thr_log, int slack = 0) {
    int32_t bound = -(1 << 24);
    for (const Term& t : terms) bound = t.exponent > bound ? t.exponent : bound;
    bound += slack;
    std::vector<WideSum> part(parts);
    for (size_t i = 0; i < terms.size(); ++i) {
        const Term& t = terms[reversed ? terms.size() - 1 - i : i];
        part[i % parts].add(t.m, bound - t.exponent, t.negative);
    }
    for (int k = 1; k < parts; ++k) part[0].merge(part[k]);
    return part[0].value(bound, threshold, thr_log);
}

int main() {
    constexpr int n = 8;
    constexpr uint32_t count = 1u << n;
    const int grades[] = {0, 17, 44, 90, 200, 500};
    double worst = 0, worst_slack = 0;
    long bad = 0, filtered = 0;
    for (int it = 0; it < 60; ++it) {
        const int s = grades[it % 6], kind = (it / 6) % 5;
        std::vector<Wide> a(count), dp(count / 2);
        for (uint32_t m = 1; m < count; ++m) {
            int e = static_cast<int>(rng() % 7) - 3;
            if (kind <= 1 && (m & 4u)) e -= s;               // one vertex
            if (kind == 1 && (m & 1u)) e -= 2 * s;           // vertex 0 as well
            if (kind == 2 && rng() % 4 == 0) e -= s;         // single subsets
            a[m] = random_wide(e);
            if (kind == 3 && rng() % 5 == 0) a[m] = wide_unpack(WidePacked{0u, 0u, 0u, 0u});
            if (kind == 4 && (m & 2u)) a[m] = wide_unpack(WidePacked{0u, 0u, 0u, 0u});
        }
        dp[0] = a[1];
        for (uint32_t rest = 1; rest < count / 2; ++rest) {  // (a submask is a smaller number)
            std::vector<Term> terms;
            auto push = [&](const uint32_t (&m)[4], int32_t e, bool neg) {
                Term t;
                std::memcpy(t.m, m, sizeof(t.m));
                t.exponent = e;
                t.negative = neg;
                terms.push_back(t);
            };
            const Wide& am = a[(rest << 1) | 1u];
            push(am.m, am.e - 1, am.sign != 0);
            f128 want = value(am), mag = want < 0 ? -want : want;
            for (uint32_t sm = (rest - 1u) & rest;; sm = (sm - 1u) & rest) {
                const Wide &x = dp[sm], &y = a[(rest ^ sm) << 1];
                uint32_t pm[4];
                mul_top(x.m, y.m, pm);
                push(pm, x.e + y.e, x.sign == y.sign);
                const f128 p = value(x) * value(y);
                want -= p;
                mag += p < 0 ? -p : p;
                if (sm == 0) break;
            }
            const Wide got = sum_of(terms, 1, false, 0.0, 0);
            for (int parts = 1; parts <= 5; parts += 2) {
                const Wide other = sum_of(terms, parts, true, 0.0, 0);
                if (std::memcmp(&other, &got, sizeof(Wide)) != 0) ++bad;
            }
            const f128 err = value(got) > want ? value(got) - want : want - value(got);
            if (mag == 0) {
                if (value(got) != 0) ++bad;
            } else {
                const double e = static_cast<double>(err / (mag * two(-112)));
                worst = e > worst ? e : worst;
                const Wide far = sum_of(terms, 1, false, 0.0, 0, kSumSlack);
                const f128 d = value(far) > want ? value(far) - want : want - value(far);
                const double es = static_cast<double>(d / (mag * two(-112)));
                worst_slack = es > worst_slack ? es : worst_slack;
                // the filter, away from its threshold
                const f128 ratio = (want < 0 ? -want : want) / mag;
                const Wide cut = sum_of(terms, 1, false, 0.25, -2), cut_far = sum_of(terms, 1, false, 0.25, -2, kSumSlack);
                if (ratio < 0.2499 && (value(cut) != 0 || value(cut_far) != 0)) ++bad;
                if (ratio > 0.2501 && std::memcmp(&cut, &got, sizeof(Wide)) != 0) ++bad;
                if (ratio > 0.2501 && std::memcmp(&cut_far, &far, sizeof(Wide)) != 0) ++bad;
                filtered += ratio < 0.2499;
            }
            dp[rest] = got;
        }
    }
    std::printf("worst error %.2f x 2^-112 of the magnitudes, %.2f on the farthest scale; %ld sums below the filter's "
                "threshold; %ld violations\n", worst, worst_slack, filtered, bad);
    // binary128's own sum of up to 2^7 terms: each of its roundings 2^-113 of the partial sum
    return (bad || filtered < 100 || worst > 256.0 || worst_slack > 256.0) ? 1 : 0;
}
