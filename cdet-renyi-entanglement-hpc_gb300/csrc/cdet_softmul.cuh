// A correctly rounded FP64 product on the integer pipes.
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

#ifdef __CUDACC__
__device__ __forceinline__ double soft_mul(const SoftFactor& x, double b, bool& bad) {
    uint32_t hi, lo;
    soft_mul_bits(x, static_cast<uint32_t>(__double2hiint(b)), static_cast<uint32_t>(__double2loint(b)), hi, lo, bad);
    return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
}
#endif

}  // namespace cdet
