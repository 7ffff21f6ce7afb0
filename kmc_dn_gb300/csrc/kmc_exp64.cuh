// kmc_exp64.cuh -- FP64 exponentials as mantissa and exponent, for the FP64 hop
// loop, and comparisons on the integer pipe, for it and the FP64 mean field.  A
// warp's FP64 instruction holds its SM quarter's unit for 64 cycles on this
// part, a comparison, a conversion or a negation as much as a multiplication.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace kmc {
namespace {

// x > 0 for finite and infinite x, false for NaN (as the comparison is), on
// the integer pipe.
__device__ __forceinline__ bool positive(double x)
{
    return static_cast<unsigned long long>(__double_as_longlong(x)) - 1ull < 0x7ff0000000000000ull;
}

// x >= y of positive finite values, on the integer pipe.
__device__ __forceinline__ bool not_less(double x, long long y_bits)
{
    return __double_as_longlong(x) >= y_bits;
}

// exp(x + y) = m * 2^k, 2^(-1/256) <= m < 2, y a small correction of x, by
// table and short polynomial (Tang, "Table-driven implementation of the
// exponential function in IEEE floating-point arithmetic", ACM TOMS 15, 1989):
// x = (128 k + j) ln2/128 + r, |r| <= ln2/256, m = 2^(j/128) (1 + p(r)), the
// table entries with their low parts.  |x| < 2^17, where n ln2/128 has 58 bits
// and the part of it that the subtraction leaves is exact: within 0.51 ulp of
// m throughout (tests/test_exp64.py; exp() 0.87 on 4e6 arguments in (-708, 0]).
constexpr int kExpTable = 128;
__device__ __forceinline__ double exp_split(double x, double y, const double2 *table, int &k)
{
    const double shift = 0x1.8p52;
    const double t = fma(x, 0x1.71547652b82fep+7, shift);        // 128/ln2
    const int n = __double2loint(t);
    const double nf = t - shift;
    // ln2/128 in a 33-bit part, whose products with small n are exact, and the rest
    double r = fma(nf, -0x1.473de6af278edp-41, fma(nf, -0x1.62e42fefp-8, x));
    if (__double_as_longlong(y) << 1) r += y;      // not for a zero: an add saved
    double q = fma(r, 1.0 / 120.0, 1.0 / 24.0);
    q = fma(fma(q, r, 1.0 / 6.0), r, 0.5);
    const double p = fma(q, r * r, r);
    const double2 T = table[n & (kExpTable - 1)];
    k = n >> 7;
    return T.x + fma(T.x, p, T.y);
}

// Entry j of that table, 2^(j/128) as hi + lo: the product of 2^(2^b/128)
// over the bits of j in double-double arithmetic.
__device__ double2 exp_table_entry(int j)
{
    const double hi[7] = {0x1.0163da9fb3335p+0, 0x1.02c9a3e778061p+0, 0x1.059b0d3158574p+0, 0x1.0b5586cf9890fp+0,
                          0x1.172b83c7d517bp+0, 0x1.306fe0a31b715p+0, 0x1.6a09e667f3bcdp+0};
    const double lo[7] = {0x1.b61299ab8cdb7p-54,  -0x1.19083535b085dp-56, 0x1.d73e2a475b465p-55,
                          0x1.8a62e4adc610bp-54,  -0x1.19041b9d78a76p-55, 0x1.6f46ad23182e4p-55,
                          -0x1.bdd3413b26456p-54};
    double x = 1.0, y = 0.0;
#pragma unroll
    for (int b = 0; b < 7; ++b) {
        if ((j >> b) & 1) {
            const double m = x * hi[b];
            const double e = fma(x, hi[b], -m) + (x * lo[b] + y * hi[b]);
            x = m + e;
            y = e - (x - m);
        }
    }
    return make_double2(x, y);
}

// |x| at and beyond which the split exponential is not used.
__device__ __forceinline__ bool splittable(double x)
{
    return (__double2hiint(x) & 0x7fffffff) < 0x41000000;
}

// x / kT as the correctly rounded quotient (reciprocal product and one
// residual, Markstein) and what it misses; `unit`: kT = 1.
__device__ __forceinline__ double over_kT(double x, bool unit, double kT, double inv_kT, double &rest)
{
    rest = 0.0;
    if (unit) return x;
    const double y0 = x * inv_kT;
    const double y = fma(fma(-y0, kT, x), inv_kT, y0);
    rest = fma(-y, kT, x) * inv_kT;
    return y;
}

// min(cap, g 2^ex), the rate of a pair from the product g of its factors'
// mantissas (cap = tc*nu, g includes it) and the sum of their exponents.
__device__ __forceinline__ double scaled_min(double g, int ex, double cap)
{
    const int er = __double2hiint(g) >> 20, e = er + ex;
    double r;
    if (static_cast<unsigned>(er - 1) < 2046u && static_cast<unsigned>(e - 1) < 2046u)
        r = __hiloint2double(__double2hiint(g) + (ex << 20), __double2loint(g));
    else if (__double_as_longlong(g) == 0)
        r = 0.0;                // a pair without a transition constant
    else if (er >= 2047 || e >= 2047)
        r = cap;
    else
        r = scalbn(g, ex);      // subnormal or about to be
    if (static_cast<unsigned long long>(__double_as_longlong(r)) >
        static_cast<unsigned long long>(__double_as_longlong(cap)))
        r = cap;
    return r;
}

}  // namespace
}  // namespace kmc
