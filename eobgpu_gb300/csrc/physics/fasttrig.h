// Sine and cosine without FP64 instructions.
//
// On GB300 an FP64 instruction costs an SM sub-partition 64 issue cycles, a
// conversion to or from a double as much, an integer one 2 and a 32 x 32 + 64 bit
// product 4, so the device library's sincos is the largest single piece of a
// waveform sample (38 FP64 instructions; 11 with a table and FP64 sums).
// Here the phase becomes an integer, units of 2^-64 turn, by one wide product with
// 2^64 / (2 pi) to 126 bits; sine and cosine of its nearest multiple of 1 / 2048
// turn come from a quarter-wave table in units of 2^-61 (S. Gal's method, as
// in Tang's log of fastlog.h), and the angle-addition formulas take the remainder
// |r| <= pi / 2048 with
//   sin r = r - r^3 / 6 + r^5 / 120,  cos r - 1 = -r^2 / 2 + r^4 / 24
// in 64-bit integers: within 2^-59.6 of the turn's values (2.4 million turns emulated reach
// 2^-59.69), 2^-59.2 with the turn's own cut-off, then rounded to a double: half an
// ulp and 2^-59.2 absolute of the exact values for |x| < 2^40 (tests/test_gpu_sincos.py,
// tests/test_gpu_phase_turns.py).  Larger, infinite and NaN arguments take the library's
// sincos.  Host: the library.
#pragma once
#include "fac_coeffs.h"
#include "trig_table.h"

namespace eob {

typedef long long i64;
typedef unsigned long long u64;

#ifdef __CUDACC__
__device__ const i64 kSinFix[513] = EOB_SINFIX_INIT;
__device__ const double kArgGammaD[7][EOB_ARG_GAMMA_N] = EOB_ARG_GAMMA_INIT;
__device__ const double kArgGammaLowD[7][EOB_ARG_GAMMA_LOW_N] = EOB_ARG_GAMMA_LOW_INIT;

// |x| < 2^127 truncated to a float, below 2^-126 to zero, by integer operations
__device__ __forceinline__ float f32_trunc(double x)
{
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned a = hi & 0x7fffffffu;
    return __uint_as_float(a < (897u << 20) ? 0u : (hi & 0x80000000u) | ((a - (896u << 20)) << 3) | (lo >> 29));
}

// the rare arguments, out of line
static __device__ __noinline__ double2 eob_sincos_large(double x)
{
    double2 r;
    sincos(x, &r.x, &r.y);
    return r;
}

// x / (2 pi) mod 1 in units of 2^-64, |x| < 2^40: the 53-bit mantissa times
// 2^64 / (2 pi) (62 integer and 64 fraction bits), shifted by the exponent
__device__ __forceinline__ u64 turns_of(double x)
{
    const i64 b = __double_as_longlong(x);
    const int e = (int)((b >> 52) & 0x7ff);
    const u64 m = ((u64)b & 0xfffffffffffffull) | (e ? 0x10000000000000ull : 0ull);
    const u64 low = m * 0x28be60db9391054aull, lo = low + __umul64hi(m, 0x7f09d5f47d4d3770ull);
    const u64 hi = __umul64hi(m, 0x28be60db9391054aull) + (lo < low ? 1 : 0);
    const int s = 1075 - e;  // 12 .. 1075
    u64 u = s < 64 ? (lo >> s) | (hi << (64 - s)) : (s < 128 ? hi >> (s - 64) : 0ull);
    return b < 0 ? 0ull - u : u;
}

// sin and cos of 2 pi t / 2^64 in units of 2^-61
__device__ __forceinline__ void sincos_fix(u64 t, i64 *s, i64 *c)
{
    const u64 v = t + (1ull << 52);
    const unsigned k = (unsigned)(v >> 53);
    const i64 rem = (i64)(v & ((1ull << 53) - 1)) - (1ll << 52);
    const i64 r = __mul64hi(rem << 9, 0x6487ed5110b4611all);  // 2 pi 2^60: the remainder, units of 2^-69
    const u64 z = (u64)__mul64hi(r, r);                       // r^2, units of 2^-74
    const unsigned zt = (unsigned)(z >> 24);
    const unsigned z2 = __umulhi(zt, zt);                     // r^4, units of 2^-68
    // cos r - 1 = -r^2 / 2 + r^4 / 24 and (sin r - r) / r = -r^2 / 6 + r^4 / 120, units of 2^-74
    const i64 c1 = (i64)(((u64)z2 * 2863311531u) >> 30) - (i64)(z >> 1);
    const i64 w = (i64)(((u64)z2 * 2290649225u) >> 32) - (i64)__umul64hi(z, 3074457345618258603ull);
    const i64 sr = r + (__mul64hi(r, w << 8) >> 18);
    const int i = k & 511;
    const i64 st = __ldg(&kSinFix[i]), ct = __ldg(&kSinFix[512 - i]);
    const i64 sv = st + (__mul64hi(ct, sr) >> 5) + (__mul64hi(st, c1) >> 10);
    const i64 cv = ct - (__mul64hi(st, sr) >> 5) + (__mul64hi(ct, c1) >> 10);
    const i64 sa = (k & 512) ? cv : sv, ca = (k & 512) ? sv : cv;
    *s = (k & 1024) ? -sa : sa;
    *c = ((k + 512) & 1024) ? -ca : ca;
}

// v 2^-61 as a double, |v| < 2^62, rounded to nearest
__device__ __forceinline__ double unit_value(i64 v)
{
    const u64 a = (u64)(v < 0 ? -v : v);
    const int z = __clzll((i64)a);
    const u64 m = a << (z & 63);
    // leading bit 2^(63 - z - 61); it carries into the exponent field, and so does a rounding up
    const u64 b = ((u64)(unsigned)(1024 - z) << 52) + (m >> 11) + ((m >> 10) & 1);
    return __longlong_as_double(a == 0 ? 0ll : (i64)(b | ((u64)v & 0x8000000000000000ull)));
}
#endif
static constexpr double kArgGammaH[7][EOB_ARG_GAMMA_N] = EOB_ARG_GAMMA_INIT;
static constexpr double kArgGammaLowH[7][EOB_ARG_GAMMA_LOW_N] = EOB_ARG_GAMMA_LOW_INIT;

#ifdef __CUDACC__
// |x| >= 2^40, infinite or NaN
__device__ __forceinline__ bool turns_refuse(double x)
{
    return (unsigned)(__double2hiint(x) & 0x7fffffff) >= 0x42700000u;
}

// The phase x of a sample, for sines and cosines of m x + add: m times the integer
// phase is exact mod 1, and a rotation takes about 100 integer instructions, where
// a complex product from one multiple to the next takes 4 FP64 ones (twice their
// issue time) and a double product and sum with m converted 3.
struct PhaseTurns {
    u64 t;
    double x;
    bool large;
    __device__ __forceinline__ explicit PhaseTurns(double phi) : x(phi)
    {
        large = turns_refuse(phi);
        t = large ? 0ull : turns_of(phi);
    }
    __device__ __forceinline__ void fix(u64 turns, double *s, double *c) const
    {
        i64 sf, cf;
        sincos_fix(turns, &sf, &cf);
        *s = unit_value(sf);
        *c = unit_value(cf);
    }
    __device__ __forceinline__ void wide(double arg, double *s, double *c) const
    {
        const double2 r = eob_sincos_large(arg);
        *s = r.x;
        *c = r.y;
    }
    __device__ __forceinline__ void multiple(int m, double *s, double *c) const
    {
        if (large) wide(m * x, s, c);
        else fix((u64)(i64)m * t, s, c);
    }
    __device__ __forceinline__ void multiple(int m, double add, double *s, double *c) const
    {
        if (large || turns_refuse(add)) wide(fma((double)m, x, add), s, c);
        else fix((u64)(i64)m * t + turns_of(add), s, c);
    }
};
#endif

EOB_HD void eob_sincos(double x, double *s, double *c)
{
#ifdef __CUDA_ARCH__
    if (turns_refuse(x)) {
        const double2 r = eob_sincos_large(x);
        *s = r.x;
        *c = r.y;
        return;
    }
    i64 sf, cf;
    sincos_fix(turns_of(x), &sf, &cf);
    *s = unit_value(sf);
    *c = unit_value(cf);
#else
    *s = sin(x);
    *c = cos(x);
#endif
}

// arg Gamma(l + 1 + i y) / y for z = (y / (l + 1))^2 in [0, EOB_ARG_GAMMA_ZMAX]
EOB_HD double arg_gamma_over_y(int l, double z)
{
#ifdef __CUDA_ARCH__
    const double *a = kArgGammaD[l - 2];
#else
    const double *a = kArgGammaH[l - 2];
#endif
    double p = a[EOB_ARG_GAMMA_N - 1];
#pragma unroll
    for (int k = EOB_ARG_GAMMA_N - 2; k >= 0; --k) p = fma(p, z, a[k]);
    return p;
}

// the same for z <= EOB_ARG_GAMMA_ZLOW
EOB_HD double arg_gamma_over_y_low(int l, double z)
{
#ifdef __CUDA_ARCH__
    const double *a = kArgGammaLowD[l - 2];
#else
    const double *a = kArgGammaLowH[l - 2];
#endif
    double p = a[EOB_ARG_GAMMA_LOW_N - 1];
#pragma unroll
    for (int k = EOB_ARG_GAMMA_LOW_N - 2; k >= 0; --k) p = fma(p, z, a[k]);
    return p;
}

}  // namespace eob
