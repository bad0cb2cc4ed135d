// Square root and reciprocal of a Cholesky pivot, correctly rounded, from an
// approximate reciprocal square root (host and device).
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define GMGS_HD __host__ __device__ __forceinline__
#else
#define GMGS_HD inline
#endif

namespace gmgs {

GMGS_HD uint64_t bits_of(double v) {
    uint64_t b;
    std::memcpy(&b, &v, sizeof(b));
    return b;
}
GMGS_HD double of_bits(uint64_t b) {
    double v;
    std::memcpy(&v, &b, sizeof(v));
    return v;
}

// s = sqrt(d) and r = 1 / s, both rounded to nearest, for a positive normal d
// well inside the exponent range and y within 2^-21 of 1 / sqrt(d).
//
// One third-order step, y (1 + h / 2 + 3 h^2 / 8) with h = 1 - d y^2 (error h^3),
// leaves y within 0.75 2^-52 of 1 / sqrt(d), relatively.  s0 = d y is refined by
// Markstein's final step s = RN(s0 + (d - s0^2) y / 2), whose residual is exact:
// before rounding it is within 2^-103 of the root, and no square root of a double
// but those that the tests enumerate lies that near to a rounding boundary.
// The same step for the reciprocal, RN(y + y (1 - s y)), goes wrong where 1 / s
// is within 2^-103 of one (s just below a power of two, and a few others), so its
// remainder 2^105 - S R of the 53-bit integers S, R is formed modulo 2^64, exact
// because it is below 2^54, and moves r by a unit where it exceeds S / 2.
// Ten dependent FP64 operations of 64 clocks (the library's square root and
// division of a lane take about 25); the remainder is integer work.
GMGS_HD void sqrt_reciprocal(double d, double y, double& s, double& r) {
    const double h = std::fma(-(d * y), y, 1.0);
    y = std::fma(y, h * std::fma(0.375, h, 0.5), y);
    const double s0 = d * y;
    s = std::fma(std::fma(-s0, s0, d), of_bits(bits_of(y) - (1ull << 52)), s0);
    r = std::fma(y, std::fma(-s, y, 1.0), y);
    // (a power of two s has a power of two r, S R = 2^104 and rest 0 as well)
    constexpr uint64_t ONE = 1ull << 52;
    const uint64_t sb = bits_of(s), rb = bits_of(r);
    const uint64_t S = (sb & (ONE - 1)) | ONE, R = (rb & (ONE - 1)) | ONE;
    const uint64_t twice = 0 - 2 * (S * R);                                // 2 (2^105 - S R): 2^105 is 0 modulo 2^64
    r = of_bits(rb + ((S - twice) >> 63) - ((S + twice) >> 63));           // the sign bits of S - twice, S + twice
}

}  // namespace gmgs
