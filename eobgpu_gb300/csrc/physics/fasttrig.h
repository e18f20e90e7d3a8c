// Sine and cosine for FP64 issue rate: 11 FP64 instructions.
//
// On GB300 an FP64 instruction costs an SM sub-partition 64 issue cycles, so
// the device library's sincos is the largest single piece of a waveform
// sample.  Here the argument is reduced to the nearest multiple of 2 pi / 2048
// (Cody and Waite with fused products: the first is exact, since the step's
// last place divides every intermediate value), the sine and cosine of the
// multiple come from a quarter-wave table of 513 correctly rounded entries
// (S. Gal's method, as in Tang's log of fastlog.h), and the angle-addition
// formulas take the remainder |r| <= pi / 2048:
//   sin r = r + (-r^3 / 6 + r^5 / 120),  cos r - 1 = -r^2 / 2 + r^4 / 24,
// the bracketed terms (below 6e-10 and 3e-13) in single precision, whose
// rounding they bring below 1e-16.  Within 2.2e-16 absolute of the exact values
// for |x| < 2^40 (tests/test_gpu_sincos.py); larger, infinite and NaN
// arguments take the library's sincos.  Host: the library.
#pragma once
#include "fac_coeffs.h"
#include "trig_table.h"

namespace eob {

#ifdef __CUDACC__
__device__ const double kSinQ[513] = EOB_SINQ_INIT;
__device__ const double kArgGammaD[7][EOB_ARG_GAMMA_N] = EOB_ARG_GAMMA_INIT;
#endif
static constexpr double kArgGammaH[7][EOB_ARG_GAMMA_N] = EOB_ARG_GAMMA_INIT;

#ifdef __CUDACC__
// the rare arguments, out of line
static __device__ __noinline__ double2 eob_sincos_large(double x)
{
    double2 r;
    sincos(x, &r.x, &r.y);
    return r;
}
#endif

#ifdef __CUDACC__
// Conversions by integer operations (a conversion instruction takes an FP64
// issue slot): |x| < 2^127 truncated to a float, below 2^-126 to zero; a float
// (zero as 2^-127) as a double.
__device__ __forceinline__ float f32_trunc(double x)
{
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned a = hi & 0x7fffffffu;
    return __uint_as_float(a < (897u << 20) ? 0u : (hi & 0x80000000u) | ((a - (896u << 20)) << 3) | (lo >> 29));
}

__device__ __forceinline__ double f64_of(float f)
{
    const unsigned b = __float_as_uint(f);
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20))), (int)(b << 29));
}
#endif

EOB_HD void eob_sincos(double x, double *s, double *c)
{
#ifdef __CUDA_ARCH__
    constexpr double kShift = 6755399441055744.0;  // 1.5 2^52
    const unsigned xe = (unsigned)__double2hiint(x) & 0x7fffffffu;
    if (xe >= 0x42700000u) {  // |x| >= 2^40, inf, NaN
        const double2 r = eob_sincos_large(x);
        *s = r.x;
        *c = r.y;
        return;
    }
    const double t = fma(x, EOB_TRIG_INV, kShift);
    const double kd = t - kShift;
    const int k = __double2loint(t);
    const double r = fma(-kd, EOB_TRIG_STEP_LO, fma(-kd, EOB_TRIG_STEP_HI, x));
    const int i = k & 511;
    const double st = __ldg(&kSinQ[i]), ct = __ldg(&kSinQ[512 - i]);
    const float rf = f32_trunc(r), q = rf * rf;
    const double r2 = r * r;
    const double sr = r + f64_of(rf * q * fmaf(q, 1.0f / 120.0f, -1.0f / 6.0f));
    const double c1 = fma(-0.5, r2, f64_of(q * q * (1.0f / 24.0f)));
    const double sv = fma(ct, sr, fma(st, c1, st)), cv = fma(-st, sr, fma(ct, c1, ct));
    // quadrant of the multiple: a swap and two sign bits
    const bool odd = (k & 512) != 0;
    const double sa = odd ? cv : sv, ca = odd ? sv : cv;
    const int sneg = (int)(((unsigned)k << 21) & 0x80000000u);
    const int cneg = (int)(((unsigned)(k + 512) << 21) & 0x80000000u);
    *s = __hiloint2double(__double2hiint(sa) ^ sneg, __double2loint(sa));
    *c = __hiloint2double(__double2hiint(ca) ^ cneg, __double2loint(ca));
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

}  // namespace eob
