// Fixed-point sums for the FP64 kernels: 96 bits for the operator (fine64.cu),
// 64 bits for the transfers (k_up64, k_restrict).
//
// GB300's FP64 unit takes 19 clocks of the SM per warp instruction; the integer
// units take a quarter of a clock.  Sums of a few FP64 values on a common scale
// are therefore formed as 96-bit integers: exact, three instructions each.
#pragma once

#include "gmgs_internal.cuh"

namespace gmgs {

struct I96 {
    uint32_t a, b, c;      // low, middle, high word (two's complement)
};

__device__ __forceinline__ I96 operator+(const I96& x, const I96& y) {
    I96 r;
    asm("add.cc.u32 %0, %3, %6;\n\taddc.cc.u32 %1, %4, %7;\n\taddc.u32 %2, %5, %8;"
        : "=r"(r.a), "=r"(r.b), "=r"(r.c)
        : "r"(x.a), "r"(x.b), "r"(x.c), "r"(y.a), "r"(y.b), "r"(y.c));
    return r;
}
__device__ __forceinline__ I96 operator-(const I96& x, const I96& y) {
    I96 r;
    asm("sub.cc.u32 %0, %3, %6;\n\tsubc.cc.u32 %1, %4, %7;\n\tsubc.u32 %2, %5, %8;"
        : "=r"(r.a), "=r"(r.b), "=r"(r.c)
        : "r"(x.a), "r"(x.b), "r"(x.c), "r"(y.a), "r"(y.b), "r"(y.c));
    return r;
}
template <int N>
__device__ __forceinline__ I96 shl(const I96& x) {
    return {x.a << N, __funnelshift_l(x.a, x.b, N), __funnelshift_l(x.b, x.c, N)};
}

// v 2^(83 - 1022 + ...) : v as a multiple of 2^(E - 1105), where the biased
// exponent of |v| is at most E (|v| < 2^(E - 1022), so |result| < 2^83).  Exact
// for exponents from E - 30 on, below that truncated to the unit.
__device__ __forceinline__ I96 to_fixed(double v, int E) {
    const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
    const int e = (int)((hi >> 20) & 0x7ffu);
    const uint32_t m = e ? (hi & 0xfffffu) | 0x100000u : 0u;      // a subnormal is far below the unit
    const uint32_t l = e ? lo : 0u;
    const int s = 30 + e - E;
    I96 r;
    if (s >= 0) {
        r = {l << s, __funnelshift_l(l, m, s), __funnelshift_l(m, 0u, s)};
    } else {
        const int t = min(-s, 63);
        const uint32_t x = t < 32 ? l : m, y = t < 32 ? m : 0u;
        r = {__funnelshift_r(x, y, t & 31), y >> (t & 31), 0u};
    }
    const uint32_t sg = (uint32_t)((int32_t)hi >> 31);            // two's complement of negative values
    r.a ^= sg;
    r.b ^= sg;
    r.c ^= sg;
    return r - I96{sg, sg, sg};
}

// floor-like x C / 2^64 for an unsigned 64-bit C (low, high word): the partial
// products below 2^32 of the quotient's unit are dropped, so the result is low
// by less than 3 units
__device__ __forceinline__ I96 mul_frac(const I96& x, uint2 C) {
    const uint64_t p = (uint64_t)x.b * C.y + __umulhi(x.b, C.x) + __umulhi(x.a, C.y);
    const uint64_t q = (uint64_t)x.c * C.x, r = (uint64_t)x.c * C.y;
    const uint32_t sg = (uint32_t)((int32_t)x.c >> 31);
    const I96 u = {(uint32_t)p, (uint32_t)(p >> 32), 0u}, w = {(uint32_t)q, (uint32_t)(q >> 32), 0u};
    const I96 z = {0u, (uint32_t)r, (uint32_t)(r >> 32)};
    const I96 t = (u + w) + z;                                    // of x as an unsigned number:
    return t - I96{0u, C.x & sg, C.y & sg};                       // 2^96 too large when x is negative
}

// x 2^Q in FP64, rounded to nearest; ex: Q + 1023 + 95, the biased exponent of 2^95 2^Q
__device__ __forceinline__ double to_double(I96 x, int ex) {
    const uint32_t sg = (uint32_t)((int32_t)x.c >> 31);
    x.a ^= sg;
    x.b ^= sg;
    x.c ^= sg;
    x = x - I96{sg, sg, sg};
    if (x.c == 0u) {
        x = {0u, x.a, x.b};
        ex -= 32;
        if (x.c == 0u) {
            x = {0u, 0u, x.b};
            ex -= 32;
        }
    }
    if (x.c == 0u) return 0.0;
    const int z = __clz((int)x.c);
    uint32_t h = __funnelshift_l(x.b, x.c, z), l = __funnelshift_l(x.a, x.b, z);
    ex -= z;
    const uint32_t l2 = l + 0x400u;                               // round at bit 10
    if (l2 < l) {
        h += 1u;
        if (h == 0u) {
            h = 0x80000000u;
            ++ex;
        }
    }
    const uint32_t dh = ((uint32_t)(ex - 1) << 20) + (h >> 11);   // the leading one adds 1 to the exponent
    return __hiloint2double((int)(dh | (sg & 0x80000000u)), (int)__funnelshift_r(l2, h, 11));
}

// Weighted sums of a few values as 64-bit integers: value v weighs 2^-k and
// counts in units of 2^(E - 1083), E the largest biased exponent of the sum's
// values.  |v| 2^-k < 2^60 units, so the weights may add up to 8.  A value is
// exact down to E - 7, below that its last bits are cut off: at most 2^-60 of
// the largest value, where an FP64 sum rounds by up to 2^-53 at each addition.
// (Only where large values cancel exactly can FP64 keep more of the small ones:
// its rounding errors may all be zero there.)
// E within SUM64_MIN .. SUM64_MAX only (no zeros, subnormals, infinities, NaN).
constexpr int SUM64_MIN = 128, SUM64_MAX = 2000;
constexpr int SUM64_DROP = 4096;      // a k that drops the value, whatever it is

__device__ __forceinline__ int abs_hi(double v) { return __double2hiint(v) & 0x7fffffff; }
__device__ __forceinline__ bool sum64_holds(int E) { return E >= SUM64_MIN && E <= SUM64_MAX; }

// k: 2^-k, or SUM64_DROP
__device__ __forceinline__ long long sum64_term(double v, int E, int k) {
    const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
    const int t = min(E - (int)((hi >> 20) & 0x7ffu) + k, 63);        // zeros and subnormals: below the unit
    const uint32_t m = (hi & 0xfffffu) | 0x100000u;
    const unsigned long long M = ((unsigned long long)__funnelshift_l(lo, m, 7) << 32) | (lo << 7);
    const long long x = (long long)(M >> t), sg = (long long)((int32_t)hi >> 31);
    return (x ^ sg) - sg;
}
// x 2^-k units in FP64, rounded to nearest
__device__ __forceinline__ double sum64_value(long long x, int E, int k) {
    const long long sg = x >> 63;
    const unsigned long long u = (unsigned long long)((x ^ sg) - sg);
    if (u == 0) return 0.0;
    const int z = __clzll((long long)u);
    unsigned long long n = u << z;                                    // 2^63 <= n < 2^64
    int ex = E + 3 - z - k;                                           // z = 4: |v| in [2^(E - 1023), 2^(E - 1022))
    const unsigned long long n2 = n + 0x400u;                         // round at bit 10
    if (n2 < n) {
        n = 1ull << 63;
        ++ex;
    } else {
        n = n2;
    }
    const uint32_t h = (uint32_t)(n >> 32), l = (uint32_t)n;
    const uint32_t dh = ((uint32_t)ex << 20) + (h >> 11);             // the leading one adds 1 to the exponent
    return __hiloint2double((int)(dh | ((uint32_t)(int32_t)sg & 0x80000000u)), (int)__funnelshift_r(l, h, 11));
}

}  // namespace gmgs
