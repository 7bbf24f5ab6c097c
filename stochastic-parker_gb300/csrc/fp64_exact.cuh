// Double-precision operations of the FP64 mover whose result can be had, bit
// for bit, with fewer or no instructions of the FP64 pipe.  That pipe takes
// one warp instruction per 64 cycles and SM sub-partition on GB300 (measured:
// add, multiply, FMA, comparison and the conversions all cost the same),
// while the integer and FP32 pipes take one every 2 cycles; so a product that
// takes about 25 integer instructions is cheaper than the conversion and the
// multiplication it replaces, and it runs beside the FP64 pipe.
//
// Every function says for which operands it is exact; outside of those it
// falls back on the plain operation.  Compiles as host C++ too (CPU test).
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define GPAT_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define GPAT_HD inline
#endif

namespace gpat {

GPAT_HD uint32_t hi_word(double x) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2hiint(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return (uint32_t)(b >> 32);
#endif
}

GPAT_HD uint32_t lo_word(double x) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2loint(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return (uint32_t)b;
#endif
}

GPAT_HD double from_words(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t b = ((uint64_t)hi << 32) | lo;
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}

GPAT_HD uint32_t float_bits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t b;
    std::memcpy(&b, &x, 4);
    return b;
#endif
}

GPAT_HD float bits_float(uint32_t b) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float x;
    std::memcpy(&x, &b, 4);
    return x;
#endif
}

GPAT_HD double fma_rn(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}

GPAT_HD bool finite_bits(double x) { return (hi_word(x) & 0x7ff00000u) != 0x7ff00000u; }

GPAT_HD bool is_zero(double x) { return ((hi_word(x) << 1) | lo_word(x)) == 0u; }

// The high words of doubles as integers in the doubles' order (both zeros 0):
// order(a) < order(b) implies a < b unless one of them is a NaN; equal high
// words say nothing.
GPAT_HD int32_t order(double x) {
    const int32_t h = (int32_t)hi_word(x), s = h >> 31;
    return ((h & 0x7fffffff) ^ s) - s;
}

// lo < x < hi for certain (false for a NaN, and where the high words decide
// nothing): the common case of a boundary test.
GPAT_HD bool surely_inside(double x, double lo, double hi) {
    const int32_t k = order(x);
    return order(lo) < k && k < order(hi);
}

// a < b, a > b
GPAT_HD bool less(double a, double b) {
    const int32_t ka = order(a), kb = order(b);
    if (ka != kb && finite_bits(a) && finite_bits(b)) return ka < kb;
    return a < b;
}

// Whether a float is one that widen() and scaled() do not take: subnormal,
// infinite or NaN.
GPAT_HD bool odd_float(float v) {
    const uint32_t t = (float_bits(v) & 0x7fffffffu) - 0x00800000u;
    return t >= 0x7f000000u && t != 0xff800000u;
}

// (double)v for v zero or normal; a zero is +0.
GPAT_HD double widen(float v) {
    const uint32_t u = float_bits(v);
    const uint32_t h = ((uint32_t)((int32_t)u >> 3) & 0x8fffffffu) + 0x38000000u;
    return from_words((u & 0x7fffffffu) == 0u ? 0u : h, u << 29);
}

// One interpolation weight taken apart for scaled(): the 53-bit mantissa
// (implicit bit included) and the exponent, prepared for adding a float's.  ok
// is false where scaled() does not apply (zero, negative, below 2^-767 or
// above 2^77, not finite).
struct Weight {
    double w;
    uint32_t hi, lo, expo;
    bool ok;
};

GPAT_HD Weight weight(double w) {
    Weight r;
    const uint32_t h = hi_word(w);
    r.w = w;
    r.lo = lo_word(w);
    r.hi = (h & 0xfffffu) | 0x100000u;
    r.ok = h - 0x10000000u < 0x34c00000u;
    // the product's biased exponent for a mantissa product below 2^84, less
    // the float's, less the implicit bit that the mantissa adds
    r.expo = (h & 0x7ff00000u) - (128u << 20);
    return r;
}

// (double)v * w rounded to nearest even, for v zero or normal and w.ok; a zero
// product is +0.  The 24-bit by 53-bit mantissa product is exact in 85 bits;
// it is shifted so that 53 of them stand above the lowest 32, and adding
// 0x7fffffff plus the last kept bit to those 32 rounds by its carry.
GPAT_HD double scaled(float v, const Weight &w) {
    const uint32_t u = float_bits(v);
    const uint32_t m = (u << 8) | 0x80000000u;
    const uint64_t p0 = (uint64_t)m * w.lo;
    const uint64_t p = (uint64_t)m * w.hi + (p0 >> 32);   // in [2^51, 2^53)
    const uint32_t ph = (uint32_t)(p >> 32), pl = (uint32_t)p, pr = (uint32_t)p0;
    const uint32_t s = (ph >> 20) ^ 1u;                   // 1: below 2^52
    const uint32_t e = ((u >> 3) & 0x0ff00000u) + w.expo + (ph & 0x100000u);
#ifdef __CUDA_ARCH__
    uint32_t h = __funnelshift_l(pl, ph, s), l = __funnelshift_l(pr, pl, s);
    const uint32_t r = pr << s, last = 0x7fffffffu + (l & 1u);
    asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %2, %3;\n\taddc.cc.u32 %0, %0, 0;\n\t"
        "addc.u32 %1, %1, %4;\n\t}"
        : "+r"(l), "+r"(h)
        : "r"(r), "r"(last), "r"(e));
#else
    const uint64_t q = (p << s) | (s ? pr >> 31 : 0u);
    const uint64_t low = (uint64_t)(uint32_t)(pr << s) + 0x7fffffffu + (q & 1u);
    const uint64_t t = q + (low >> 32);
    const uint32_t l = (uint32_t)t, h = (uint32_t)(t >> 32) + e;
#endif
    const bool zero = (u & 0x7fffffffu) == 0u;
    return from_words(zero ? 0u : h | (u & 0x80000000u), zero ? 0u : l);
}

// a / b for a divisor known beforehand, with its correctly rounded reciprocal
// rb: one multiplication and two FMAs (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34, 1990).  a zero or in 2^+-900, b normal and far from the ends of
// the range (reciprocal returns 0 otherwise); else the plain division.
GPAT_HD double div_by(double a, double b, double rb) {
    const uint32_t mag = hi_word(a) & 0x7fffffffu;
    if ((mag - 0x07b00000u < 0x70800000u || (mag | lo_word(a)) == 0u) && hi_word(rb) != 0u) {
        const double q = a * rb;
        return fma_rn(fma_rn(-q, b, a), rb, q);
    }
    return a / b;
}

GPAT_HD double reciprocal(double b) {
    const uint32_t mag = hi_word(b) & 0x7fffffffu;
    return mag - 0x39b00000u < 0x0c800000u ? 1.0 / b : 0.0;   // 2^-100 .. 2^100
}

// floor(x) and floor(x) + 1 as a double, for |x| < 2^30 (false otherwise):
// adding 1.5 2^52 rounds to an integer that stands in the low word.
GPAT_HD bool floor_next(double x, int &fl, double &next) {
    if ((hi_word(x) & 0x7fffffffu) >= 0x41d00000u) return false;
    const double magic = 6755399441055744.0;
#ifdef __CUDA_ARCH__
    const double t = __dadd_rd(x, magic);
#else
    const double t = std::floor(x) + magic;
#endif
    fl = (int)lo_word(t);
    next = t - (magic - 1.0);
    return true;
}

// 2 u - 1 for the 53-bit uniform u = ((a >> 5) 2^26 + (b >> 6)) / 2^53: with
// the first of the 53 bits set, 2 u - 1 is the fraction of the others, else
// that fraction less 1; both differences are exact.
GPAT_HD double symmetric_uniform(uint32_t a, uint32_t b) {
    const double one_to_two = from_words(0x3ff00000u | ((a >> 11) & 0xfffffu),
                                         ((a >> 5) << 26) | (b >> 6));
    return one_to_two - ((a >> 31) ? 1.0 : 2.0);
}

// A double's magnitude as a float, its mantissa cut to 20 bits (at most 2^-20
// too small), for magnitudes in 2^-50 .. 2^50; ok is cleared outside of them.
GPAT_HD float rough(double x, bool &ok) {
    const uint32_t mag = hi_word(x) & 0x7fffffffu;
    if (mag - 0x3cd00000u >= 0x06400000u) ok = false;
    return bits_float((mag - 0x38000000u) << 3);
}

}  // namespace gpat
