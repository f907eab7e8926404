// Correctly rounded FP64 products, sums and reciprocals on the integer pipes.
//
// GB300 retires about two FP64 lane operations per clock and SM, so a warp's
// FP64 instruction holds its sub-partition's FP64 pipe for 64 to 74 clocks.
// The integer pipes are idle meanwhile, and a 53 x 53 bit product with its
// rounding is about 25 of their instructions (45 clocks of a sub-partition
// alone, hidden completely behind two FP64 additions; measured on a Clenshaw
// step: product and two additions on the FP64 pipe 104 ns per warp step,
// product here 70 ns). soft_mul therefore takes one of the three operations
// of the reference's Clenshaw step off the pipe that bounds it.
//
// The result is the IEEE round-to-nearest-even product, the same bits as
// __dmul_rn, whenever `bad` stays clear. `bad` is set (never cleared) when
// the value may need more than the common path: b zero, subnormal, infinite,
// NaN or of extreme exponent, or the discarded bits within 2^-32 ulp of a
// tie. The caller then repeats the work with __dmul_rn.
#pragma once

#include <cstdint>

namespace cdet {

// The fixed factor x, unpacked once: its 53-bit significand at the top of 64
// bits, its sign, and its exponent field as an increment of the other
// factor's high word.
struct SoftFactor {
    uint32_t hi, lo, sign, exponent;
};

// |x| in [2^-100, 2): every product with |b| in (2^-723, 2^677) is normal.
__host__ __device__ __forceinline__ bool soft_factor_in_range(uint32_t x_hi) {
    const uint32_t field = (x_hi >> 20) & 0x7FFu;
    return field >= 1023u - 100u && field <= 1024u;
}

__host__ __device__ __forceinline__ SoftFactor soft_factor(uint32_t x_hi, uint32_t x_lo) {
    SoftFactor f;
    const uint32_t top = (x_hi & 0xFFFFFu) | 0x100000u;
    f.hi = (top << 11) | (x_lo >> 21);
    f.lo = x_lo << 11;
    f.sign = x_hi & 0x80000000u;
    f.exponent = (((x_hi >> 20) & 0x7FFu) - 1023u) << 20;
    return f;
}

// With B the 53-bit significand of b and X the 64-bit one of x, B X lies in
// [2^115, 2^117): its high word pair holds the 53 significant bits, or 52 of
// them (`small`), in which case everything moves up one bit and the exponent
// down one. Half an ulp is added below the kept bits; the carry runs into the
// exponent field where the significand overflows.
__host__ __device__ __forceinline__ void soft_mul_bits(const SoftFactor& x, uint32_t b_hi, uint32_t b_lo,
                                                       uint32_t& r_hi, uint32_t& r_lo, bool& bad) {
    const uint32_t bh = (b_hi & 0xFFFFFu) | 0x100000u;
    const uint64_t p0 = static_cast<uint64_t>(b_lo) * x.lo;
    const uint64_t p1 = static_cast<uint64_t>(b_lo) * x.hi + (p0 >> 32);
    const uint64_t p2 = static_cast<uint64_t>(bh) * x.lo + static_cast<uint32_t>(p1);
    const uint64_t p3 = static_cast<uint64_t>(bh) * x.hi + (p1 >> 32) + (p2 >> 32);
    const uint32_t w0 = static_cast<uint32_t>(p0), w1 = static_cast<uint32_t>(p2);
    const uint32_t w2 = static_cast<uint32_t>(p3), w3 = static_cast<uint32_t>(p3 >> 32);
    const bool small = w3 < 0x100000u;
#ifdef __CUDA_ARCH__
    const uint32_t s = small ? 1u : 0u;
    const uint32_t v3 = __funnelshift_l(w2, w3, s);
    const uint32_t v2 = __funnelshift_l(w1, w2, s);
    const uint32_t v1 = __funnelshift_l(w0, w1, s);
#else
    const uint32_t v3 = small ? (w3 << 1) | (w2 >> 31) : w3;
    const uint32_t v2 = small ? (w2 << 1) | (w1 >> 31) : w2;
    const uint32_t v1 = small ? (w1 << 1) | (w0 >> 31) : w1;
#endif
    bad |= v1 == 0x80000000u;                                  // a tie, or within 2^-32 ulp above one
    bad |= (b_hi << 1) - (300u << 21) > (1400u << 21);         // b's exponent field outside 300..1700
    const uint32_t field = ((b_hi & 0xFFF00000u) ^ x.sign) + (small ? x.exponent - 0x100000u : x.exponent);
#ifdef __CUDA_ARCH__
    asm("{.reg .u32 d;\n"
        " add.cc.u32 d, %2, 0x80000000;\n"
        " addc.cc.u32 %0, %3, 0;\n"
        " addc.u32 %1, %4, %5;}"
        : "=&r"(r_lo), "=r"(r_hi)
        : "r"(v1), "r"(v2), "r"(v3), "r"(field));
#else
    const uint64_t kept = ((static_cast<uint64_t>(v3) << 32) | v2) + (v1 >> 31);
    r_lo = static_cast<uint32_t>(kept);
    r_hi = static_cast<uint32_t>(kept >> 32) + field;
#endif
}

// x + y, correctly rounded, on the integer pipes: about 55 of their
// instructions, more than an FP64 addition's time on its own pipe, so a kernel
// takes it for a share of its additions only. The operand of larger magnitude
// keeps its place in a window of three words (21 + 32 bits and 32 guard bits),
// the other is shifted down to it and added or subtracted. `bad` as for the
// product: an operand zero, subnormal, infinite, NaN or near the ends of the
// exponent range, 21 or more bits cancelled, operands whose order the upper
// words do not tell, or, where a shift by 32 or more has dropped bits below the
// window, discarded bits within a few units of a tie. Exact ties (frequent:
// nearby exponents discard a bit or two) round to even here.
__host__ __device__ __forceinline__ void soft_add_bits(uint32_t x_hi, uint32_t x_lo, uint32_t y_hi, uint32_t y_lo,
                                                       uint32_t& r_hi, uint32_t& r_lo, bool& bad) {
    const bool swap = (x_hi & 0x7FFFFFFFu) < (y_hi & 0x7FFFFFFFu);
    const uint32_t bh = swap ? y_hi : x_hi, bl = swap ? y_lo : x_lo;
    const uint32_t sh = swap ? x_hi : y_hi, sl = swap ? x_lo : y_lo;
    const uint32_t small_field = sh & 0x7FF00000u;
    uint32_t d = ((bh & 0x7FF00000u) - small_field) >> 20;
    d = d < 63u ? d : 63u;
    const uint32_t mb = (bh & 0xFFFFFu) | 0x100000u, ms = (sh & 0xFFFFFu) | 0x100000u;
    const bool far = d >= 32u;
    const uint32_t w2 = far ? 0u : ms, w1 = far ? ms : sl, w0 = far ? sl : 0u;
    const uint32_t m = static_cast<uint32_t>(static_cast<int32_t>(bh ^ sh) >> 31);  // all ones: subtract
#ifdef __CUDA_ARCH__
    const uint32_t z2 = __funnelshift_r(w2, 0u, d) ^ m, z1 = __funnelshift_r(w1, w2, d) ^ m;
    const uint32_t z0 = __funnelshift_r(w0, w1, d) ^ m;
    uint32_t s0, s1, s2;
    asm("{.reg .u32 t;\n"
        " add.cc.u32 t, %3, 1;\n"
        " addc.cc.u32 %0, %4, 0;\n"
        " addc.cc.u32 %1, %5, %6;\n"
        " addc.u32 %2, %7, %8;}"
        : "=&r"(s0), "=&r"(s1), "=r"(s2)
        : "r"(m), "r"(z0), "r"(z1), "r"(bl), "r"(z2), "r"(mb));
    const uint32_t n = static_cast<uint32_t>(__clz(static_cast<int>(s2))) - 10u;
    const uint32_t v2 = __funnelshift_l(s1, s2, n), v1 = __funnelshift_l(s0, s1, n), v0 = s0 << (n & 31u);
    const uint32_t k1 = __funnelshift_r(v1, v2, 1), rest = __funnelshift_r(v0, v1, 1);
#else
    const uint32_t c = d & 31u;
    auto right = [c](uint32_t lo, uint32_t hi) { return c ? (lo >> c) | (hi << (32 - c)) : lo; };
    const uint32_t z2 = right(w2, 0u) ^ m, z1 = right(w1, w2) ^ m, z0 = right(w0, w1) ^ m;
    uint64_t carry = static_cast<uint64_t>(z0) + (m & 1u);
    const uint32_t s0 = static_cast<uint32_t>(carry);
    carry = (carry >> 32) + bl + z1;
    const uint32_t s1 = static_cast<uint32_t>(carry);
    const uint32_t s2 = static_cast<uint32_t>((carry >> 32) + mb + z2);
    const uint32_t n = (s2 ? static_cast<uint32_t>(__builtin_clz(s2)) : 32u) - 10u;
    const uint32_t e = n & 31u;
    const uint32_t v2 = e ? (s2 << e) | (s1 >> (32 - e)) : s2, v1 = e ? (s1 << e) | (s0 >> (32 - e)) : s1, v0 = s0 << e;
    const uint32_t k1 = (v1 >> 1) | (v2 << 31), rest = (v0 >> 1) | (v1 << 31);
#endif
    bad |= s2 - 1u >= 0x3FFFFFu;                          // negative, or 21 bits and more cancelled
    bad |= far && rest - 0x7FFFFFFCu <= 8u;
    bad |= (bh << 1) - (64u << 21) > (1936u << 21);       // the larger exponent field outside 64..2000
    bad |= small_field == 0u;
    const uint32_t field = (bh & 0xFFF00000u) - (n << 20);
    const uint32_t keep = rest == 0x80000000u ? 0xFFFFFFFEu : 0xFFFFFFFFu;  // a tie rounds up, then to even
#ifdef __CUDA_ARCH__
    asm("{.reg .u32 t;\n"
        " add.cc.u32 t, %2, 0x80000000;\n"
        " addc.cc.u32 %0, %3, 0;\n"
        " addc.u32 %1, %4, %5;}"
        : "=&r"(r_lo), "=r"(r_hi)
        : "r"(rest), "r"(k1), "r"(v2 >> 1), "r"(field));
    r_lo &= keep;
#else
    const uint64_t kept = ((static_cast<uint64_t>(v2 >> 1) << 32) | k1) + (rest >> 31);
    r_lo = static_cast<uint32_t>(kept) & keep;
    r_hi = static_cast<uint32_t>(kept >> 32) + field;
#endif
}

// 1 / b, correctly rounded, on the integer pipes (about 50 instructions, where
// the FP64 one holds its pipe for eight). From a 24-bit reciprocal a little
// below 1/b, q0, the residual e = 1 - b q0 in (0, 2^-21) gives q0 (1 + e + e^2)
// within one unit of the last place; the exact remainder 2^105 - B Q, whose
// magnitude is below 2^54, then says whether that neighbour or the next is the
// nearest (a reciprocal is never a tie).
// seed: the FP32 bits of an approximation, within a unit or so of its last
// place, of the reciprocal of soft_rcp_arg(b). `bad` (set, never cleared): a
// power of two, a zero, subnormal, infinite or NaN b, a subnormal result, or a
// seed further off than that.
__host__ __device__ __forceinline__ uint32_t soft_rcp_arg(uint32_t b_hi, uint32_t b_lo) {
    return 0x3F800001u + (((b_hi & 0xFFFFFu) << 3) | (b_lo >> 29));  // rounded up
}

__host__ __device__ __forceinline__ void soft_rcp_bits(uint32_t b_hi, uint32_t b_lo, uint32_t seed, uint32_t& r_hi,
                                                       uint32_t& r_lo, bool& bad) {
    const uint64_t B = (static_cast<uint64_t>((b_hi & 0xFFFFFu) | 0x100000u) << 32) | b_lo;  // 2^52 b
    const uint32_t top = static_cast<uint32_t>(B >> 21), bottom = b_lo << 11;
    const uint32_t below = seed - 2u;
    const uint32_t q0 = ((below > 0x3F000000u ? below : 0x3F000000u) << 8) | 0x80000000u;    // 2^32 / b
    const uint64_t t = (uint64_t{1} << 63) + 512u -
                       (static_cast<uint64_t>(top) * q0 + ((static_cast<uint64_t>(bottom) * q0) >> 32));
    bad |= static_cast<uint32_t>(t >> 42) != 0u;
    const uint32_t e = static_cast<uint32_t>(t >> 10);                                       // 2^53 e
    const uint32_t e2 = static_cast<uint32_t>((static_cast<uint64_t>(e) * e) >> 32);         // 2^74 e^2
    const uint64_t c = static_cast<uint64_t>(q0) * e + ((static_cast<uint64_t>(q0) * e2) >> 21) + 0x80000000u;
    uint64_t Q = (static_cast<uint64_t>(q0) << 21) + (c >> 32);                              // 2^53 / b
    const int64_t r2 = static_cast<int64_t>((0u - B * Q) << 1);
    Q -= static_cast<uint64_t>((static_cast<int64_t>(B) - r2) >> 63);  // 2 R > B: the next above
    Q += static_cast<uint64_t>((static_cast<int64_t>(B) + r2) >> 63);  // 2 R < -B: the next below
    const uint32_t field = (b_hi >> 20) & 0x7FFu;
    bad |= field - 1u >= 2043u;
    bad |= B == uint64_t{1} << 52;
    r_lo = static_cast<uint32_t>(Q);
    r_hi = (b_hi & 0x80000000u) + ((2044u - field) << 20) + static_cast<uint32_t>(Q >> 32);
}

#ifdef __CUDACC__
// 1 / b, correctly rounded, for any b.
__device__ __forceinline__ double soft_rcp(double b) {
    const uint32_t b_hi = static_cast<uint32_t>(__double2hiint(b)), b_lo = static_cast<uint32_t>(__double2loint(b));
    uint32_t hi, lo;
    float seed;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(seed) : "f"(__uint_as_float(soft_rcp_arg(b_hi, b_lo))));
    bool bad = false;
    soft_rcp_bits(b_hi, b_lo, __float_as_uint(seed), hi, lo, bad);
    if (bad) return __drcp_rn(b);
    return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
}
__device__ __forceinline__ double soft_mul(const SoftFactor& x, double b, bool& bad) {
    uint32_t hi, lo;
    soft_mul_bits(x, static_cast<uint32_t>(__double2hiint(b)), static_cast<uint32_t>(__double2loint(b)), hi, lo, bad);
    return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
}
__device__ __forceinline__ double soft_add(double x, double y, bool& bad) {
    uint32_t hi, lo;
    soft_add_bits(static_cast<uint32_t>(__double2hiint(x)), static_cast<uint32_t>(__double2loint(x)),
                  static_cast<uint32_t>(__double2hiint(y)), static_cast<uint32_t>(__double2loint(y)), hi, lo, bad);
    return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
}
#endif

}  // namespace cdet
