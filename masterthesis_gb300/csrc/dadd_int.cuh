// Exact binary64 addition on the 32-bit integer pipe.
//
// GB300's FP64 pipe retires about 1.8 lane operations per clock per SM, the
// integer pipe 64: an FP64 stencil sweep keeps the FP64 pipe busy while the
// integer pipe idles.  dadd_same_sign_bits computes a + b, rounded to
// nearest even exactly as the FP64 adder does (the same bits), from the
// operands' bit patterns with integer instructions only.  It covers the case
// that dominates the neighbour sums of a smooth field -- both operands of
// one sign, exponents at most 10 apart, the smaller exponent field in
// [1, 2035] (magnitudes from 2^-1022 to about 2^1013) -- and reports every
// other case (zeros, subnormals, infinities, NaNs, opposite signs, distant
// exponents, huge magnitudes) through `ok`, for the caller to add in FP64
// instead.
//
// Method (textbook IEEE addition with guard bits): place each significand
// (hidden bit included) at bits 62-d..10-d of a 64-bit word, d <= 10 its
// distance from the larger exponent, so that no bit is shifted out and the
// sum is exact; add; round to nearest even at bit 10, or at bit 11 when the sum
// carried into bit 63; pack: the rounded significand's hidden bit is added
// into the exponent field, so a rounding carry raises the exponent by
// itself.
//
// The operands are aligned to the larger exponent where they stand; ordering
// them by magnitude first took four selects and a comparison more (90
// instead of 128 integer-ALU instructions per node of a sweep, 117 to 122
// GLUP/s for two rows per thread).
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define SCAFES_HD __host__ __device__ __forceinline__
#else
#define SCAFES_HD inline
#endif

namespace scafes {

SCAFES_HD uint64_t dadd_same_sign_bits(uint64_t a, uint64_t b, bool& ok) {
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a;
    const uint32_t bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
    const uint32_t ea = ah >> 20, eb = bh >> 20;  // sign and exponent field
    const uint32_t e = ea > eb ? ea : eb, m = ea > eb ? eb : ea;
    // The smaller exponent in [1, 2035] and at most 10 apart.  With opposite
    // signs the larger is the negative one's, 2048 + its exponent, which is
    // more than 10 above any exponent <= 2035, so the test covers the signs;
    // the larger exponent is at most 2045.
    ok = e - m <= 10u && (m & 0x7ffu) - 1u < 2035u;
    uint32_t pa = 1024u >> ((e - ea) & 31u), pb = 1024u >> ((e - eb) & 31u);
#if defined(__CUDA_ARCH__)
    // Keeps the alignment a multiply (the FMA pipe) rather than a shift (the
    // integer ALU, which the adder keeps busier).
    asm("" : "+r"(pa), "+r"(pb));
#endif
    // ma * 2^(10 - da) + mb * 2^(10 - db), one of da, db zero: exact, below 2^64.
    uint64_t s = (uint64_t)al * pa + (uint64_t)bl * pb;
    s += (uint64_t)(((ah & 0x000fffffu) | 0x00100000u) * pa + ((bh & 0x000fffffu) | 0x00100000u) * pb) << 32;
    const uint32_t c = (uint32_t)(s >> 63);
    const uint32_t sh = 10u + c;
    // + (half - 1) + the last kept bit: rounds half to even.
    s += (uint64_t)(0x1ffu + 0x200u * c + (((uint32_t)s >> sh) & 1u));
    const uint64_t r = s >> sh;  // 53 bits, or 2^53 after a rounding carry
    return ((uint64_t)((e + c - 1u) << 20) << 32) + r;
}

// a + b for operands of any signs: RN of the exact sum where `ok`, which
// holds when the exponents are at most 9 apart or one operand is zero (or
// subnormal, and then lost below the other's last bit), and the larger
// exponent field is in [64, 2045] or the sum is zero.  For the differences of
// neighbours in fields that change sign.  The significands are aligned to the
// larger exponent with 9 guard bits (so nothing is shifted out), added as
// signed 64-bit numbers, and the magnitude is normalised by its leading
// zeros and rounded half to even.  A zero sum has the FP64 adder's sign: -0
// only where both operands are -0.
SCAFES_HD uint64_t dadd_bits(uint64_t a, uint64_t b, bool& ok) {
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a;
    const uint32_t bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
    const uint32_t z0 = ah & bh & 0x80000000u;  // the high word of a zero sum
    const uint32_t ta = ah & 0x7ff00000u, tb = bh & 0x7ff00000u;
    const uint32_t e = ta > tb ? ta : tb, m = ta > tb ? tb : ta;
    const uint32_t sa = (e - ta) >> 20, sb = (e - tb) >> 20;
#if defined(__CUDA_ARCH__)
    // PTX shifts clamp: 0 from 32 on.
    uint32_t pa, pb;
    asm("shr.u32 %0, 512, %1;" : "=r"(pa) : "r"(sa));
    asm("shr.u32 %0, 512, %1;" : "=r"(pb) : "r"(sb));
#else
    const uint32_t pa = sa < 32 ? 512u >> sa : 0u, pb = sb < 32 ? 512u >> sb : 0u;
#endif
    // The hidden bit, absent with a zero exponent field.
    const uint32_t mah = (ah & 0x000fffffu) | (ta < 0x00100000u ? ta : 0x00100000u);
    const uint32_t mbh = (bh & 0x000fffffu) | (tb < 0x00100000u ? tb : 0x00100000u);
    const uint64_t A = (uint64_t)al * pa + ((uint64_t)(mah * pa) << 32);
    const uint64_t B = (uint64_t)bl * pb + ((uint64_t)(mbh * pb) << 32);
    const int64_t d = (int32_t)(ah ^ bh) >> 31;  // all ones when the signs differ
    const int64_t s = (int64_t)(A + ((B ^ (uint64_t)d) - (uint64_t)d));
    const int64_t n = s >> 63;
    const uint64_t mag = (uint64_t)((s ^ n) - n);
#if defined(__CUDA_ARCH__)
    const int lz = __clzll((long long)mag);
#else
    const int lz = mag ? __builtin_clzll(mag) : 64;
#endif
    uint64_t r = mag << ((lz - 1) & 63);  // leading bit at 62
    r += (uint64_t)(0x1ffu + (((uint32_t)r >> 10) & 1u));
    r >>= 10;
    const uint32_t top = e - 0x04000000u;  // exponent field - 64
    // A zero sum is right at any exponent but that of infinities and NaNs.
    ok = (e - m <= 0x00900000u || m == 0u) && (top <= 0x7bd00000u || (mag == 0u && e < 0x7ff00000u));
    const uint32_t hi = ((uint32_t)(r >> 32) + e + ((uint32_t)(1 - lz) << 20)) | ((ah ^ (uint32_t)n) & 0x80000000u);
    // The low word of a zero sum is zero already.  Where the sign is formed
    // decides what the compiler spills: a Yee step at 128 x 120 x 113 takes 62.5
    // us with it formed first, 63.0 formed here, 66 with both words selected,
    // and 62.1 with the sign dropped.
    return ((uint64_t)(mag ? hi : z0) << 32) | (uint32_t)r;
}

// A constant factor prepared for dmul_bits: its significand's 53 bits at the
// top of 64, what its exponent and sign add to the high word of the other
// factor, and the exponent fields (in place) for which the product and both
// factors are normal numbers: [lo, lo + range].
struct IntFactor {
    uint32_t ch, cl, k, lo, range;
};

inline IntFactor make_int_factor(double c) {
    uint64_t b;
    __builtin_memcpy(&b, &c, 8);
    const int ec = (int)(b >> 52 & 0x7ff);
    const uint64_t m = ((b & 0xfffffffffffffull) | (1ull << 52)) << 11;
    IntFactor f;
    f.ch = (uint32_t)(m >> 32);
    f.cl = (uint32_t)m;
    f.k = ((uint32_t)(ec - 1023) << 20) + (uint32_t)(b >> 63 << 31);
    const int lo = 1025 - ec > 1 ? 1025 - ec : 1, hi = 3067 - ec < 2046 ? 3067 - ec : 2046;
    const bool normal = ec >= 1 && ec <= 2046 && lo <= hi;
    f.lo = normal ? (uint32_t)lo << 20 : 0xfff00000u;  // never matched
    f.range = normal ? (uint32_t)(hi - lo) << 20 : 0u;
    return f;
}

// c * u, rounded to nearest even as by the FP64 multiplier, where `ok` (u,
// c and the product normal numbers).  The 53 x 53 bit product is formed
// exactly in four 32 x 32 multiplications (the FMA pipe); its top 53 bits are
// rounded with the rest.
SCAFES_HD uint64_t dmul_bits(const IntFactor& c, uint64_t u, bool& ok) {
    const uint32_t uh = (uint32_t)(u >> 32), ul = (uint32_t)u;
    const uint32_t mh = (uh & 0x000fffffu) | 0x00100000u;
    const uint64_t p0 = (uint64_t)ul * c.cl;
    const uint64_t p1 = (uint64_t)ul * c.ch + (p0 >> 32);
    const uint64_t p2 = (uint64_t)mh * c.cl + (uint32_t)p1;
    const uint64_t p3 = (uint64_t)mh * c.ch + (p1 >> 32) + (p2 >> 32);  // the top 52 or 53 bits
    const uint32_t r1 = (uint32_t)p2, r0 = (uint32_t)p0;                // the rest
    const uint32_t th = (uint32_t)(p3 >> 32), tl = (uint32_t)p3;
    const uint32_t s = 1u - (th >> 20);  // one bit short: shift in the next
#if defined(__CUDA_ARCH__)
    const uint32_t nh = __funnelshift_l(tl, th, s), nl = __funnelshift_l(r1, tl, s), nr = __funnelshift_l(r0, r1, s);
#else
    const uint32_t nh = s ? th << 1 | tl >> 31 : th, nl = s ? tl << 1 | r1 >> 31 : tl, nr = s ? r1 << 1 | r0 >> 31 : r1;
#endif
    // Round half to even; a bit of r0 breaks a tie (where its top bit moved
    // into nr, nr is no tie).
    const uint32_t rest = nr | (r0 != 0u ? 1u : 0u);
    const uint32_t up = rest > 0x80000000u - (nl & 1u) ? 1u : 0u;
    const uint64_t m = (((uint64_t)nh << 32) | nl) + up;
    ok = (uh & 0x7ff00000u) - c.lo <= c.range;
    return m + ((uint64_t)((uh & 0xfff00000u) + c.k - (s << 20)) << 32);
}

}  // namespace scafes
