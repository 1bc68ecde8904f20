// verlet_axis.cuh -- one coordinate's verlet update (integrators/src/verlet.rs:
// 24-82) in f64 in the reference's operation order, and the correctly rounded
// division by a constant that it needs.
#pragma once

#include <stdint.h>
#include <string.h>

namespace pg {

// A divisor that stays the same over many divisions, as the integer division of
// mantissas uses it: GB300 issues two f64 operations per clock and SM, and a
// correctly rounded f64 division is a chain of them (three per body were 60 of
// the 94 us that verlet took at 1,048,580 bodies), while the integer units do 64.
// Division by an invariant with a precomputed reciprocal: Moeller & Granlund,
// "Improved division by invariant integers" (IEEE Trans. Computers 60, 2011).
struct Divisor {
    double value;
    uint64_t d, v;     // mantissa with its top bit at 63; floor((2^128 - 1) / d) - 2^64
    int32_t exponent;  // biased; 0: not a normal number (plain division)
    uint32_t pad;
};

inline Divisor make_divisor(double value)
{
    Divisor r;
    memset(&r, 0, sizeof r);
    r.value = value;
    uint64_t bits;
    memcpy(&bits, &value, sizeof bits);
    const int e = (int)(bits >> 52) & 0x7ff;
    if (e == 0 || e == 0x7ff) return r;
    r.exponent = e;
    r.d = ((bits & 0xfffffffffffffull) | (1ull << 52)) << 11;
    r.v = (uint64_t)((~(unsigned __int128)0 - ((unsigned __int128)r.d << 64)) / r.d);
    return r;
}

#ifdef __CUDACC__

// n / d.value, correctly rounded (the bits of __ddiv_rn).
__device__ __forceinline__ double divide(double n, const Divisor &d)
{
    const uint64_t bits = (uint64_t)__double_as_longlong(n);
    const int e = (int)(bits >> 52) & 0x7ff;
    // quotient of the mantissas: q = floor(2^63 n / d), 2^62 < q < 2^64, with the
    // remainder's part in the rounding
    const uint64_t u = ((bits & 0xfffffffffffffull) | (1ull << 52)) << 10;
    const uint64_t low = d.v * u;
    uint64_t q = __umul64hi(d.v, u) + u + 1ull;
    uint64_t r = 0ull - q * d.d;
    if (r > low) {
        --q;
        r += d.d;
    }
    if (r >= d.d) {
        ++q;
        r -= d.d;
    }
    const int shift = 10 + (int)(q >> 63);
    uint64_t m = q >> shift;
    const uint64_t rest = q & ((1ull << shift) - 1ull), half = 1ull << (shift - 1);
    // nearest, ties (no remainder at all) to even
    m += rest > half || (rest == half && (r != 0ull || (m & 1ull)));
    const int ex = e - d.exponent + 1023 + (shift - 11);
    if (e == 0 || e == 0x7ff || d.exponent == 0 || ex < 1 || ex > 2045)
        return __ddiv_rn(n, d.value);
    // m has its top bit at 52 (or, rounded up, is 2^53: the carry goes on)
    const uint64_t sign = (bits ^ (uint64_t)__double_as_longlong(d.value)) & (1ull << 63);
    return __longlong_as_double((long long)(sign | (((uint64_t)(ex - 1) << 52) + m)));
}

// 2 x, exact: the exponent of a normal number below the largest.
__device__ __forceinline__ double twice(double x)
{
    const uint64_t bits = (uint64_t)__double_as_longlong(x);
    const uint32_t e = (uint32_t)(bits >> 52) & 0x7ffu;
    if (e - 1u < 2045u) return __longlong_as_double((long long)(bits + (1ull << 52)));
    return __dadd_rn(x, x);
}

// verlet.rs:33-39 (initial, Taylor step) and verlet.rs:64-70 (regular).
__device__ __forceinline__ void verlet_axis(double &x, double &v, double &p, double a,
                                            const Divisor &dt, double dt2, bool initial)
{
    double xn, vn;
    if (initial) {
        // x + vx*dt + 0.5*a*dt^2 ; vx + a*dt
        xn = __dadd_rn(__dadd_rn(x, __dmul_rn(v, dt.value)), __dmul_rn(__dmul_rn(0.5, a), dt2));
        vn = __dadd_rn(v, __dmul_rn(a, dt.value));
    } else {
        // 2*x - prev + a*dt^2 ; (x' - x)/dt
        xn = __dadd_rn(__dsub_rn(twice(x), p), __dmul_rn(a, dt2));
        vn = divide(__dsub_rn(xn, x), dt);
    }
    p = x;
    x = xn;
    v = vn;
}

#endif

}  // namespace pg
