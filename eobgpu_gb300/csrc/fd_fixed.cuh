// The frequency-domain residual of one (bin, detector) on the integer units.
//
// |d - (F+ h+ + Fx hx) e^{-2 pi i f tau}|^2 / S takes 17 to 24 FP64 instructions,
// and GB300 issues one in 64 cycles per SM sub-partition; a 32 x 32 + 64 bit
// product takes 4.  Here the projection, the rotation and the difference are block
// floating point: 64-bit integers with one exponent per vector, and the FP64 pipe keeps the
// square and its weight: 3 instructions per (bin, detector), beside about 60 integer
// products and shifts that issue meanwhile.
//
//  * The residual is held to 2^-56 of max|F| max|h| (their powers of two) and 2^-60 of |d|;
//    with what the products cut off its error is 2^-55.7 of the former (rms; 2^-54.2 at
//    most, emulated), where FP64 rounds five times to 2^-53 of |F+ h+| + |Fx hx|.  Bins
//    where both products are well below that maximum (kApart) take the FP64 expression.
//  * dot_hi: a sum of two 64-bit products' upper halves from six 32-bit ones (the
//    products of the low halves, below the last place, left out).
//  * The delay phase: df tau, rounded once, as an integer of 128 bits, whose product with
//    the bin is exact to 2^-64 turn; sine and cosine come from fasttrig.h in units
//    of 2^-61, and the next bin of a thread by a rotation (2^-56 a step at most, up to
//    15 steps).
//    A vector's components share an exponent, so a residual of exactly equal
//    terms is 2^-56 of their size rather than zero.
//  * The residual becomes a double again with its exponent, so weights, sums,
//    infinite PSDs and the range are FP64's own.  Infinities, NaN and values above
//    2^960 take the FP64 expression, one bin at a time; subnormals count as zero
//    (their square is).
#pragma once
#include "eob_device.cuh"

namespace eob {

constexpr int kFixTop = 1023 + 960;  // largest exponent field of the integer path

// (a b + c d) / 2^64 for |a|, |c| < 2^62 and |b|, |d| <= 2^61, -3.75 to +0.75 units off: the
// shift (-1), the products of low halves (-2), the lowest bits (3/4 either way)
__device__ __forceinline__ i64 dot_hi(i64 a, i64 b, i64 c, i64 d)
{
    const int ah = (int)(a >> 32), bh = (int)(b >> 32), ch = (int)(c >> 32), dh = (int)(d >> 32);
    const int al = (int)((unsigned)a >> 1), bl = (int)((unsigned)b >> 1);
    const int cl = (int)((unsigned)c >> 1), dl = (int)((unsigned)d >> 1);
    const i64 p = (i64)ah * bh + (i64)ch * dh;
    const i64 q = (i64)ah * bl + (i64)al * bh + ((i64)ch * dl + (i64)cl * dh);
    return p + (q >> 31);
}

// u cycles per bin (mod 1, |u| < 2^10: turn_ok) in units of 2^-64 turn and, below them,
// 2^-128: a double down to 2^-75 fits, so that the phase of bin i, i u, is exact to the
// last 2^-64 turn.  In 2^-64 alone the cut-off rest, times i, was 6.6e-13 rad in bin 2^21 at
// df = 1/1024, tau = 1 ms.
struct Turns {
    u64 hi, lo;
    // of bin i
    __device__ __forceinline__ u64 at(int i) const
    {
        const unsigned k = (unsigned)i;
        const u64 p = (u64)k * (unsigned)(lo >> 32) + (((u64)k * (unsigned)lo) >> 32);
        return (u64)k * hi + (p >> 32);
    }
};

__device__ __forceinline__ bool turn_ok(double u)
{
    return (unsigned)(__double2hiint(u) & 0x7fffffff) < 0x40900000u;
}

__device__ __forceinline__ Turns turn_of(double u)
{
    const i64 b = __double_as_longlong(u);
    const int e = (int)((b >> 52) & 0x7ff);
    const u64 m = ((u64)b & 0xfffffffffffffull) | (e ? 0x10000000000000ull : 0ull);
    const int sh = e - 1023 - 52 + 128;  // |u| = m 2^sh 2^-128; below 86
    Turns t;
    t.hi = sh >= 64 ? m << min(sh - 64, 63) : (sh > 11 ? m >> (64 - sh) : 0ull);
    t.lo = sh >= 64 ? 0ull : (sh >= 0 ? m << sh : (sh > -64 ? m >> -sh : 0ull));
    if (b < 0) {
        t.lo = 0ull - t.lo;
        t.hi = ~t.hi + (t.lo == 0ull ? 1ull : 0ull);
    }
    return t;
}

// (c, s) turned by (rc, rs)
__device__ __forceinline__ void rotate(i64 *s, i64 *c, i64 rs, i64 rc)
{
    const i64 cn = dot_hi(*c, rc, -*s, rs) << 3;
    *s = dot_hi(*s, rc, *c, rs) << 3;
    *c = cn;
}

__device__ __forceinline__ int exponent_of(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// x in units of 2^(e - 1023 - 52 - up) for an exponent field e >= that of x: |result| < 2^(53 + up)
__device__ __forceinline__ i64 fix_of(double x, int e, int up)
{
    const i64 b = __double_as_longlong(x);
    const int f = (int)((b >> 52) & 0x7ff);
    const u64 m = (u64)((b & 0xfffffffffffffll) | 0x10000000000000ll) << up;
    const u64 v = m >> min(e - f, 63);
    return f == 0 ? 0 : (b < 0 ? -(i64)v : (i64)v);
}

// |v| 2^u as a double (rounded to nearest; zero below the normal range)
__device__ __forceinline__ double size_of(i64 v, int u)
{
    const u64 a = (u64)(v < 0 ? -v : v);
    const int z = __clzll((i64)a);
    const u64 m = a << (z & 63);
    const int e = 1023 + u + 63 - z;
    // the mantissa's leading one carries into the exponent field, and so does a rounding up
    const u64 b = ((u64)(unsigned)(e - 1) << 52) + (m >> 11) + ((m >> 10) & 1);
    return __longlong_as_double((a == 0 || e < 1) ? 0ll : (i64)b);
}

// One (bin, detector) of the data: in units of 2^e, |.| < 2^61, and 1 / S (32 bytes).
struct __align__(16) FdData {
    i64 re, im;
    double w;
    int e;
    __device__ __forceinline__ bool slow() const { return e > kFixTop - 1023 - 60; }
};

__device__ __forceinline__ FdData fd_data(double2 d, double S)
{
    const int f = max(exponent_of(d.x), exponent_of(d.y));
    return {fix_of(d.x, f, 8), fix_of(d.y, f, 8), 1.0 / S, f - 1023 - 60};
}

// The polarisations share an exponent, and so do the patterns. Where the larger of one
// meets the smaller of the other by more than kApart bits each, F+ h+ and Fx hx are both
// that far below the product of the exponents and would lose as many bits: a detector at the
// null of a pattern, a source near edge-on. Either side carries a mask; a bin is slow where
// they meet.
constexpr int kApart = 2;
constexpr int kPlus = 1, kCross = 2, kBin = 4, kDet = 8, kAll = -1;

__device__ __forceinline__ int apart(int plus, int cross)
{
    const int d = plus - cross;  // by the signs of the differences
    return (((kApart - d) >> 31) & kPlus) | (((kApart + d) >> 31) & kCross);
}

// What the residual needs of a (binary, detector): the patterns in units of
// 2^e, |.| < 2^61, the phase per bin and its rotation over `stride` bins.
struct FdDetector {
    i64 fp, fx, rs, rc;
    Turns step;
    int e, mask;
    __device__ __forceinline__ bool slow() const { return mask == kAll; }
};

__device__ __forceinline__ FdDetector fd_detector(double fp, double fx, double cycles_per_bin, int stride)
{
    FdDetector q;
    const int p = exponent_of(fp), x = exponent_of(fx), e = max(p, x);
    const bool slow = !turn_ok(cycles_per_bin) || e > 1023 + 20 || (e < 1023 - 60 && e > 0);
    q.mask = slow ? kAll : kDet | apart(x, p);  // a weak plus pattern meets a strong h+
    q.fp = fix_of(fp, e, 8);
    q.fx = fix_of(fx, e, 8);
    q.e = e - 1023 - 60;
    q.step = turn_of(cycles_per_bin);
    sincos_fix(q.step.at(stride), &q.rs, &q.rc);
    return q;
}

// The polarisations of one bin in units of 2^e, |.| < 2^62
struct FdStrain {
    i64 pr, pi, xr, xi;
    int e, mask;
};

__device__ __forceinline__ FdStrain fd_strain(double2 p, double2 x)
{
    const int f = max(exponent_of(p.x), exponent_of(p.y)), g = max(exponent_of(x.x), exponent_of(x.y)), e = max(f, g);
    return {fix_of(p.x, e, 9), fix_of(p.y, e, 9), fix_of(x.x, e, 9), fix_of(x.y, e, 9), e - 1023 - 61,
            ((kFixTop - e) >> 31) | kBin | apart(f, g)};
}

__device__ __forceinline__ bool fd_slow(const FdStrain &h, const FdDetector &q, const FdData &d)
{
    return (h.mask & q.mask) != 0 || d.slow();
}

// |d - (F+ h+ + Fx hx) (c - i s)|^2
__device__ __forceinline__ double fd_power(const FdStrain &h, const FdDetector &q, i64 s, i64 c, const FdData &d)
{
    // the projection, |.| < 2^62, in units of 2^(h.e + q.e + 62), and it rotated, |.| < 2^60, of 2^(h.e + q.e + 65)
    const i64 gr = dot_hi(h.pr, q.fp, h.xr, q.fx) << 2, gi = dot_hi(h.pi, q.fp, h.xi, q.fx) << 2;
    const i64 tr = dot_hi(gr, c, gi, s), ti = dot_hi(gi, c, -gr, s);
    const int et = h.e + q.e + 65;
    const int u = max(et, d.e), st = min(u - et, 63), sd = min(u - d.e, 63);
    const double rr = size_of((d.re >> sd) - (tr >> st), u), ri = size_of((d.im >> sd) - (ti >> st), u);
    return fma(rr, rr, ri * ri);
}

// the same in FP64, for what the integers do not take; the sines and cosines are theirs unless the detector
// is slow itself
static __device__ __noinline__ double fd_power_slow(double2 hp, double2 hx, double fp, double fx, double2 d,
                                                    double cycles, bool detector, i64 si, i64 ci)
{
    double s = unit_value(si), c = unit_value(ci);
    if (detector) sincos(2.0 * kPi * cycles, &s, &c);
    const double gr = fma(fp, hp.x, fx * hx.x), gi = fma(fp, hp.y, fx * hx.y);
    const double rr = d.x - fma(gr, c, gi * s), ri = d.y - fma(gi, c, -gr * s);
    return fma(rr, rr, ri * ri);
}

}  // namespace eob
