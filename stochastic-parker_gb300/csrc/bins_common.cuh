// Binning of particles for the distributions, off the FP64 pipe (which would
// take 25 of its instructions for one log10): the same bins and the same
// fixed-point weights as the plain expressions, which decide wherever the
// cheaper form is not certain.
#pragma once

#include <cmath>

#include "device_common.cuh"
#include "fp64_exact.cuh"

namespace gpat {

// floor((log10(p) - pmin_log) / dp_log) through log2 p = e + log2 m in FP32:
// pos = scale (e + log2 m) + offset, off by less than tol.
struct LogBins {
    double pmin_log, dp_log;
    float scale, offset, tol, tol_e;
};

inline LogBins make_log_bins(double pmin_log, double dp_log) {
    LogBins b;
    b.pmin_log = pmin_log;
    b.dp_log = dp_log;
    b.scale = (float)(0.30102999566398120 / dp_log);
    b.offset = (float)(-pmin_log / dp_log);
    // __log2f on [1, 2) and the cut mantissa: 4.1e-7; the roundings of scale,
    // offset and the sums: 2^-22 of their magnitudes.  Four times that.
    b.tol = 2e-6f * (std::fabs(b.scale) + std::fabs(b.offset) + 1.0f);
    b.tol_e = 2e-6f * std::fabs(b.scale);
    return b;
}

__device__ __forceinline__ int log_bin(double p, const LogBins &b) {
    const uint32_t h = hi_word(p);
    if (h - 0x00100000u < 0x7fe00000u) {   // positive and normal
        const float e = (float)((int)(h >> 20) - 1023);
        const float m = bits_float(0x3f800000u | ((h & 0xfffffu) << 3) | (lo_word(p) >> 29));
        const float pos = __fmaf_rn(__log2f(m), b.scale, __fmaf_rn(e, b.scale, b.offset));
        const float k = floorf(pos), frac = pos - k, tol = __fmaf_rn(fabsf(e), b.tol_e, b.tol);
        if (frac > tol && frac < 1.0f - tol && fabsf(pos) < 1e6f) return (int)k;
    }
    return (int)floor((log10(p) - b.pmin_log) / b.dp_log);
}

// floor((x - lo) / d) through FP32: x cut to 24 bits, off by less than tol bins.
struct EvenBins {
    double lo, d, rd;
    float lo_f, inv, tol_x;
};

inline EvenBins make_even_bins(double lo, double d) {
    EvenBins b;
    b.lo = lo;
    b.d = d;
    b.rd = reciprocal(d);
    b.lo_f = (float)lo;
    b.inv = (float)(1.0 / d);
    b.tol_x = 4e-7f * std::fabs(b.inv);
    return b;
}

__device__ __forceinline__ int even_bin(double x, const EvenBins &b) {
    const uint32_t h = hi_word(x), mag = h & 0x7fffffffu;
    if (mag - 0x39b00000u < 0x0c800000u || (mag | lo_word(x)) == 0u) {   // 2^+-100, or 0
        const float v = mag == 0u ? 0.0f
                                  : bits_float((h & 0x80000000u) | ((mag - 0x38000000u) << 3) |
                                               (lo_word(x) >> 29));
        const float pos = (v - b.lo_f) * b.inv;
        const float k = floorf(pos), frac = pos - k;
        const float tol = __fmaf_rn(fabsf(v) + fabsf(b.lo_f), b.tol_x, 1e-6f * fabsf(pos) + 1e-6f);
        if (frac > tol && frac < 1.0f - tol && fabsf(pos) < 1e6f) return (int)k;
    }
    const double q = div_by(x - b.lo, b.d, b.rd);
    int k;
    double next;
    return floor_next(q, k, next) ? k : (int)floor(q);
}

__device__ __forceinline__ bool within_one(double mu) {   // -1 <= mu <= 1
    const uint32_t mag = hi_word(mu) & 0x7fffffffu;
    return mag < 0x3ff00000u || (mag == 0x3ff00000u && lo_word(mu) == 0u);
}

// fixed_split for w in [2^-64, 2^63): the 53-bit mantissa shifted into 64.64
// fixed point, cut below 2^-64; other values by fixed_split itself.
__device__ __forceinline__ void fixed_parts(double w, unsigned long long &h,
                                            unsigned long long &l) {
    const uint32_t hw = hi_word(w);
    const int e = (int)(hw >> 20) - 1023;   // the sign bit puts negative values out of range
    if (e < -64 || e > 62) {
        fixed_split(w, h, l);
        return;
    }
    const unsigned long long m =
        ((unsigned long long)((hw & 0xfffffu) | 0x100000u) << 32) | lo_word(w);
    const int s = e + 12;                   // m 2^(e - 52) in units of 2^-64
    if (s >= 0) {
        l = s < 64 ? m << s : 0ull;
        h = s == 0 ? 0ull : s < 64 ? m >> (64 - s) : m << (s - 64);
    } else {
        l = m >> -s;
        h = 0ull;
    }
}

// Weights in shared memory as eight 16-bit limbs summed in 32-bit words: adds
// that return nothing and carry nothing, one for a weight that is a power of
// two.  A word holds the limbs of 65536 weights.
constexpr int kLimbs = 8;

__device__ __forceinline__ void limbs_add(unsigned int *limb, unsigned long long h,
                                          unsigned long long l) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const unsigned int a = (unsigned int)(l >> (16 * k)) & 0xffffu;
        if (a) atomicAdd(&limb[k], a);
    }
    if (h) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned int a = (unsigned int)(h >> (16 * k)) & 0xffffu;
            if (a) atomicAdd(&limb[4 + k], a);
        }
    }
}

__device__ __forceinline__ void limbs_sum(const unsigned int *limb, unsigned long long &h,
                                          unsigned long long &l) {
    h = 0ull;
    l = 0ull;
#pragma unroll
    for (int k = 0; k < kLimbs; ++k) {
        const unsigned long long v = limb[k];
        if (k < 4)
            add_u128(h, l, k == 0 ? 0ull : v >> (64 - 16 * k), v << (16 * k));
        else
            h += v << (16 * (k - 4));
    }
}

}  // namespace gpat
