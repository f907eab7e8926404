// 113-bit floating point on the integer pipes.
//
// The double-double integrand behind the split assembly needs about 106 bits
// through the minors and the connected recursion. A double-double pair update
// is 16 FP64 operations, and GB300's FP64 pipe takes 64 to 74 clocks of a
// sub-partition for each; the same update on 32-bit integer multiplies is
// about 110 clocks in all. These are the pieces.
//
// A number in registers (Wide) is sign, exponent and a mantissa M of four
// words with its leading one at bit 126: (-1)^sign M 2^(e - 127). In memory
// (uint4) it is sign, a 15-bit exponent (bias 16384) and the 112 bits below
// the leading one, so that stored magnitudes compare as 128-bit integers.
// Stored results are truncated: relative error below 2^-112 (a double-double
// sum's is a few 2^-104). Zero is the all-zero word; unpacked it reads as
// a number so small that every alignment shifts it out. Functions are __host__ too, so
// that the arithmetic can be checked without a GPU.
#pragma once

#include <cstdint>

namespace cdet {

struct Wide {
    uint32_t m[4];  // m[3] the most significant
    int32_t e;
    uint32_t sign;  // 0 or 1
};
struct alignas(16) WidePacked {
    uint32_t x, y, z, w;
};

constexpr int kWideBias = 16384;
constexpr int kWideFlush = -16000;       // results below 2^kWideFlush are stored as zero
constexpr int32_t kWideZero = -(1 << 20);  // the exponent a zero unpacks to

// (hi:lo) << s and >> s for s in 0..31, one word of the result
__host__ __device__ __forceinline__ uint32_t shl_word(uint32_t lo, uint32_t hi, int s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, s);
#else
    return s ? (hi << s) | (lo >> (32 - s)) : hi;
#endif
}
__host__ __device__ __forceinline__ uint32_t shr_word(uint32_t lo, uint32_t hi, int s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_r(lo, hi, s);
#else
    return s ? (lo >> s) | (hi << (32 - s)) : lo;
#endif
}
__host__ __device__ __forceinline__ int leading_zeros(uint32_t x) {
#ifdef __CUDA_ARCH__
    return __clz(static_cast<int>(x));
#else
    return x ? __builtin_clz(x) : 32;
#endif
}

// a += b + carry-in (0 or 1), least significant word first
template <int N>
__host__ __device__ __forceinline__ void add_words(uint32_t (&a)[N], const uint32_t (&b)[N], uint32_t carry_in) {
#ifdef __CUDA_ARCH__
    static_assert(N >= 3 && N <= 6, "one carry chain per length");
    if constexpr (N == 3) {
        asm("{.reg .u32 t;\n"
            " add.cc.u32 t, %6, 0xffffffff;\n"
            " addc.cc.u32 %0, %0, %3;\n"
            " addc.cc.u32 %1, %1, %4;\n"
            " addc.u32 %2, %2, %5;}"
            : "+r"(a[0]), "+r"(a[1]), "+r"(a[2])
            : "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(carry_in));
    } else if constexpr (N == 4) {
        asm("{.reg .u32 t;\n"
            " add.cc.u32 t, %8, 0xffffffff;\n"
            " addc.cc.u32 %0, %0, %4;\n"
            " addc.cc.u32 %1, %1, %5;\n"
            " addc.cc.u32 %2, %2, %6;\n"
            " addc.u32 %3, %3, %7;}"
            : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3])
            : "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(carry_in));
    } else if constexpr (N == 5) {
        asm("{.reg .u32 t;\n"
            " add.cc.u32 t, %10, 0xffffffff;\n"
            " addc.cc.u32 %0, %0, %5;\n"
            " addc.cc.u32 %1, %1, %6;\n"
            " addc.cc.u32 %2, %2, %7;\n"
            " addc.cc.u32 %3, %3, %8;\n"
            " addc.u32 %4, %4, %9;}"
            : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4])
            : "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(carry_in));
    } else {
        asm("{.reg .u32 t;\n"
            " add.cc.u32 t, %12, 0xffffffff;\n"
            " addc.cc.u32 %0, %0, %6;\n"
            " addc.cc.u32 %1, %1, %7;\n"
            " addc.cc.u32 %2, %2, %8;\n"
            " addc.cc.u32 %3, %3, %9;\n"
            " addc.cc.u32 %4, %4, %10;\n"
            " addc.u32 %5, %5, %11;}"
            : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5])
            : "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(carry_in));
    }
#else
    uint64_t c = carry_in;
    for (int i = 0; i < N; ++i) {
        c += static_cast<uint64_t>(a[i]) + b[i];
        a[i] = static_cast<uint32_t>(c);
        c >>= 32;
    }
#endif
}

__host__ __device__ __forceinline__ Wide wide_unpack(const WidePacked& q) {
    Wide r;
    r.m[3] = (shl_word(q.z, q.w, 14) & 0x3FFFFFFFu) | 0x40000000u;
    r.m[2] = shl_word(q.y, q.z, 14);
    r.m[1] = shl_word(q.x, q.y, 14);
    r.m[0] = q.x << 14;
    const int32_t field = static_cast<int32_t>((q.w >> 16) & 0x7FFFu);
    r.e = field ? field - kWideBias : kWideZero;
    r.sign = q.w >> 31;
    return r;
}

// Packs a mantissa with its leading one at bit 126.
__host__ __device__ __forceinline__ WidePacked wide_pack(const Wide& a) {
    WidePacked q;
    q.x = shr_word(a.m[0], a.m[1], 14);
    q.y = shr_word(a.m[1], a.m[2], 14);
    q.z = shr_word(a.m[2], a.m[3], 14);
    q.w = (a.sign << 31) | (static_cast<uint32_t>(a.e + kWideBias) << 16) | ((a.m[3] >> 14) & 0xFFFFu);
    if (a.e < kWideFlush) q = WidePacked{0u, 0u, 0u, 0u};
    return q;
}

__host__ __device__ __forceinline__ Wide wide_from_bits(uint64_t bits) {  // of a finite double; subnormals as zero
    Wide r;
    const int field = static_cast<int>((bits >> 52) & 0x7FFu);
    const uint64_t mant = (bits & ((uint64_t{1} << 52) - 1)) | (uint64_t{1} << 52);
    r.m[3] = static_cast<uint32_t>(mant >> 22);
    r.m[2] = static_cast<uint32_t>(mant) << 10;
    r.m[1] = r.m[0] = 0;
    r.e = field ? field - 1022 : kWideZero;
    r.sign = static_cast<uint32_t>(bits >> 63);
    return r;
}

// The upper four words of the eight-word product: ten of the sixteen partial
// products; what is left out is below 4 units of the last word kept.
__host__ __device__ __forceinline__ void mul_top(const uint32_t (&a)[4], const uint32_t (&b)[4], uint32_t (&p)[4]) {
    auto wide = [](uint32_t x, uint32_t y) { return static_cast<uint64_t>(x) * y; };
    auto high = [](uint64_t x) { return x >> 32; };
    const uint64_t x = wide(a[3], b[1]) + high(wide(a[3], b[0])) + high(wide(a[2], b[1]));
    const uint64_t y = wide(b[3], a[1]) + high(wide(b[3], a[0])) + high(wide(b[2], a[1]));
    const uint64_t q0 = wide(a[2], b[2]);
    const uint64_t q1 = wide(a[2], b[3]) + high(q0);
    const uint64_t q2 = wide(a[3], b[2]) + static_cast<uint32_t>(q1);
    uint64_t hi = wide(a[3], b[3]) + high(q1) + high(q2);
    uint64_t lo = (q2 << 32) | static_cast<uint32_t>(q0);
#ifdef __CUDA_ARCH__
    asm("add.cc.u64 %0, %0, %2;\n addc.u64 %1, %1, 0;\n add.cc.u64 %0, %0, %3;\n addc.u64 %1, %1, 0;"
        : "+l"(lo), "+l"(hi)
        : "l"(x), "l"(y));
#else
    lo += x;
    hi += lo < x;
    lo += y;
    hi += lo < y;
#endif
    p[0] = static_cast<uint32_t>(lo);
    p[1] = static_cast<uint32_t>(lo >> 32);
    p[2] = static_cast<uint32_t>(hi);
    p[3] = static_cast<uint32_t>(hi >> 32);
}

// a b with the leading one wherever mul_top leaves it (bit 124 or 125): the
// value is p 2^(e - 126).
__host__ __device__ __forceinline__ Wide wide_mul_raw(const Wide& a, const Wide& b) {
    Wide r;
    mul_top(a.m, b.m, r.m);
    r.e = a.e + b.e;
    r.sign = a.sign ^ b.sign;
    return r;
}
__host__ __device__ __forceinline__ Wide wide_mul(const Wide& a, const Wide& b) {
    Wide r = wide_mul_raw(a, b);
    const int s = (r.m[3] & 0x20000000u) ? 1 : 2;  // leading one to bit 126
    r.m[3] = shl_word(r.m[2], r.m[3], s);
    r.m[2] = shl_word(r.m[1], r.m[2], s);
    r.m[1] = shl_word(r.m[0], r.m[1], s);
    r.m[0] <<= s;
    r.e += 1 - s;
    return r;
}

// words >> d (d >= 0) within N words, least significant first
template <int N>
__host__ __device__ __forceinline__ void shift_right_words(uint32_t (&t)[N], int d) {
    const int ws = d >> 5, bs = d & 31;
#pragma unroll
    for (int i = 0; i < N; ++i) t[i] = i + 1 < N ? shr_word(t[i], t[i + 1], bs) : t[i] >> bs;
    if (ws & 1) {
#pragma unroll
        for (int i = 0; i < N; ++i) t[i] = i + 1 < N ? t[i + 1] : 0u;
    }
    if (ws & 2) {
#pragma unroll
        for (int i = 0; i < N; ++i) t[i] = i + 2 < N ? t[i + 2] : 0u;
    }
    if (ws >= 4) {
#pragma unroll
        for (int i = 0; i < N; ++i) t[i] = ((ws & ~7) == 0 && i + 4 < N) ? t[i + 4] : 0u;
    }
}

// t (N words, two's complement when `negative`) to magnitude
template <int N>
__host__ __device__ __forceinline__ void negate_if(uint32_t (&t)[N], bool negative) {
    const uint32_t m = negative ? 0xFFFFFFFFu : 0u;
    const uint32_t zero[N] = {};
#pragma unroll
    for (int i = 0; i < N; ++i) t[i] ^= m;
    add_words(t, zero, m & 1u);
}

// Moves the leading one of N words to bit 126 of the upper four words (32 N -
// 2 of all); returns the left shift (-1 .. ), 32 N when t is zero.
template <int N>
__host__ __device__ __forceinline__ int normalise_words(uint32_t (&t)[N]) {
    int shift = 0;
    while (t[N - 1] == 0 && shift < 32 * N) {
#pragma unroll
        for (int i = N - 1; i > 0; --i) t[i] = t[i - 1];
        t[0] = 0;
        shift += 32;
    }
    const int lz = leading_zeros(t[N - 1]);
    if (lz == 0) {
#pragma unroll
        for (int i = 0; i < N; ++i) t[i] = i + 1 < N ? shr_word(t[i], t[i + 1], 1) : t[i] >> 1;
    } else if (lz < 32) {
#pragma unroll
        for (int i = N - 1; i >= 0; --i) t[i] = i > 0 ? shl_word(t[i - 1], t[i], lz - 1) : t[i] << (lz - 1);
    }
    return shift + lz - 1;
}

// x + y, the mantissas below 2^127 and not necessarily normalised (value
// m 2^(e - 127)); one guard word, so the error is below 2^-157 of the larger
// operand's range.
__host__ __device__ __forceinline__ Wide wide_add(Wide x, Wide y) {
    if (x.e < y.e) {
        const Wide t = x;
        x = y;
        y = t;
    }
    uint32_t a[5] = {0u, x.m[0], x.m[1], x.m[2], x.m[3]};
    uint32_t b[5] = {0u, y.m[0], y.m[1], y.m[2], y.m[3]};
    shift_right_words(b, x.e - y.e);
    const uint32_t mask = x.sign != y.sign ? 0xFFFFFFFFu : 0u;
#pragma unroll
    for (int i = 0; i < 5; ++i) b[i] ^= mask;
    add_words(a, b, mask & 1u);
    const bool negative = mask && (a[4] >> 31);
    negate_if(a, negative);
    const int shift = normalise_words(a);
    Wide r;
#pragma unroll
    for (int i = 0; i < 4; ++i) r.m[i] = a[i + 1];
    r.e = shift >= 159 ? kWideZero : x.e - shift;
    r.sign = x.sign ^ (negative ? 1u : 0u);
    return r;
}

// base - l r
__host__ __device__ __forceinline__ Wide wide_sub_prod(const Wide& l, const Wide& r, const Wide& base) {
    Wide p = wide_mul_raw(l, r);
    p.e += 1;  // p 2^(e - 126)
    p.sign ^= 1u;
    return wide_add(base, p);
}

// 1 / a from a double's reciprocal of the leading 53 bits and two Newton
// steps: relative error below 2^-115. `reciprocal` is the caller's 1 / x for
// doubles x in [1, 2).
template <class Reciprocal>
__host__ __device__ __forceinline__ Wide wide_inverse(const Wide& a, Reciprocal reciprocal) {
    // D = m 2^-126 in [1, 2); r ~ 1 / D as R 2^-126, R in (2^125, 2^126]
    const uint64_t d_bits = (uint64_t{0x3FF} << 52) | (static_cast<uint64_t>(a.m[3] & 0x3FFFFFFFu) << 22) | (a.m[2] >> 10);
    const uint64_t r_bits = reciprocal(d_bits);  // bits of a double in (0.5, 1]
    Wide r = wide_from_bits(r_bits);             // m 2^(e - 127), e = 0 (or 1 for exactly 1)
    if (r.e == 0) {                              // to R 2^-126
#pragma unroll
        for (int i = 0; i < 4; ++i) r.m[i] = i < 3 ? shr_word(r.m[i], r.m[i + 1], 1) : r.m[i] >> 1;
    }
#pragma unroll 1
    for (int step = 0; step < 2; ++step) {
        uint32_t t[4], c[4];
        mul_top(a.m, r.m, t);  // D r 2^124
        // rho = 2^124 - t
        uint32_t rho[4] = {~t[0], ~t[1], ~t[2], ~t[3]};
        const uint32_t one[4] = {0u, 0u, 0u, 0x10000000u};
        add_words(rho, one, 1u);
        const bool negative = rho[3] >> 31;
        negate_if(rho, negative);
        mul_top(r.m, rho, c);  // R rho / 2^128; the correction is R rho / 2^124
#pragma unroll
        for (int i = 3; i >= 0; --i) c[i] = i > 0 ? shl_word(c[i - 1], c[i], 4) : c[i] << 4;
        if (negative) {
#pragma unroll
            for (int i = 0; i < 4; ++i) c[i] = ~c[i];
        }
        add_words(r.m, c, negative ? 1u : 0u);
    }
    // r = R 2^-126, a = D 2^(a.e - 1): 1 / a = R 2^(2 - a.e - 127)
    uint32_t n[4] = {r.m[0], r.m[1], r.m[2], r.m[3]};
    const int shift = normalise_words(n);
    Wide out;
#pragma unroll
    for (int i = 0; i < 4; ++i) out.m[i] = n[i];
    out.e = 2 - a.e - shift;
    out.sign = a.sign;
    return out;
}

__host__ __device__ __forceinline__ int bit_length(const uint32_t* t, int words) {
    for (int i = words - 1; i >= 0; --i)
        if (t[i]) return 32 * i + 32 - leading_zeros(t[i]);
    return 0;
}

// A sum of up to 2^9 + 1 terms on a fixed-point scale: 192 bits in two's
// complement with a unit of 2^(bound - 178), `bound` at least every term's
// exponent, and the sum of the terms' magnitudes with a unit of 2^(bound - 114).
// Integer additions: the terms may be taken in any order and in parts (merge)
// without changing a bit. Terms far below the bound lose bits: it has to lie
// within kSumSlack of some term's exponent, so that the magnitudes reach
// 2^(bound - 50); the sum's error is then below 2^-118 of them, theirs below
// 2^-54.
constexpr int kSumWords = 6;
constexpr int kSumHeadroom = 12;  // bits between the largest term and the sign
constexpr int kMagWords = 4;      // the magnitudes keep the upper four words
constexpr int kSumSlack = 48;
struct WideSum {
    uint32_t acc[kSumWords] = {}, mag[kMagWords] = {};

    // +-m 2^(bound - below - 126), m < 2^127, below >= 0
    __host__ __device__ __forceinline__ void add(const uint32_t (&m)[4], int below, bool negative) {
        uint32_t t[kSumWords] = {0u, 0u, m[0], m[1], m[2], m[3]};
        shift_right_words(t, below + kSumHeadroom);
        const uint32_t top[kMagWords] = {t[2], t[3], t[4], t[5]};
        add_words(mag, top, 0u);
        const uint32_t x = negative ? 0xFFFFFFFFu : 0u;
#pragma unroll
        for (int i = 0; i < kSumWords; ++i) t[i] ^= x;
        add_words(acc, t, x & 1u);
    }
    __host__ __device__ __forceinline__ void merge(const WideSum& o) {
        add_words(acc, o.acc, 0u);
        add_words(mag, o.mag, 0u);
    }
    // The sum; zero where its magnitude is below threshold (> 0; thr_log its
    // ilogb) times the sum of the terms' magnitudes, and where all terms are
    // the zeros of wide_unpack.
    __host__ __device__ __forceinline__ Wide value(int32_t bound, double threshold, int thr_log) const {
        uint32_t a[kSumWords];
#pragma unroll
        for (int i = 0; i < kSumWords; ++i) a[i] = acc[i];
        const bool negative = a[kSumWords - 1] >> 31;
        negate_if(a, negative);
        bool keep = bound > kWideZero / 2;
        if (threshold > 0.0) {
            constexpr int kLow = 32 * (kSumWords - kMagWords);
            if (bit_length(a, kSumWords) < kLow + bit_length(mag, kMagWords) + thr_log + 2) {
                // near or below the threshold: compare as doubles
                double av = 0.0, mv = 0.0;
                for (int i = kSumWords - 1; i >= 0; --i) av = av * 4294967296.0 + static_cast<double>(a[i]);
                for (int i = kMagWords - 1; i >= 0; --i) mv = mv * 4294967296.0 + static_cast<double>(mag[i]);
                keep = keep && !(av < threshold * (mv * 18446744073709551616.0));  // 2^kLow
            }
        }
        const int shift = normalise_words(a);
        Wide r;
#pragma unroll
        for (int i = 0; i < 4; ++i) r.m[i] = a[i + 2];
        // a 2^(bound - 178), its leading one moved to bit 190 = m 2^(e - 127), m the upper four words
        r.e = keep && shift < 32 * kSumWords - 1 ? bound + kSumHeadroom + 1 - shift : kWideZero;
        r.sign = negative ? 1u : 0u;
        return r;
    }
};

// |a| <= |b| for stored numbers
__host__ __device__ __forceinline__ bool wide_abs_le(const WidePacked& a, const WidePacked& b) {
    const uint64_t ah = (static_cast<uint64_t>(a.w & 0x7FFFFFFFu) << 32) | a.z;
    const uint64_t bh = (static_cast<uint64_t>(b.w & 0x7FFFFFFFu) << 32) | b.z;
    const uint64_t al = (static_cast<uint64_t>(a.y) << 32) | a.x, bl = (static_cast<uint64_t>(b.y) << 32) | b.x;
    return ah < bh || (ah == bh && al <= bl);
}

}  // namespace cdet
