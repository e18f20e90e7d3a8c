// Synthesis on the uniform grid and the likelihood, from the splines of
// k_post.cu:
//
//  k_scan_chunks  per-binary work items of kChunk samples (kStrainChunk where
//                 the strain is written), exclusive scan; the data's sum of
//                 squares (and FP32 copy) on blocks of their own.
//  k_synth_lnl    one block per run of chunks: spline evaluation on the
//                 uniform grid (eob/seobnrv4phm.py:274-386, 2310-2372), mode sum
//                 (BBHWaveformTD, :715-721) and the white-noise residual, reduced
//                 to one partial per chunk; the strain is never written to memory.
//  k_synth_strain the strain itself, summed or per mode.
//  k_synth_mixed_* the same with the amplitudes, the trigonometry and the
//                 residual in FP32.
//  k_finalize     one warp per binary, partials summed in a fixed order
//                 (deterministic).
#include "eob_device.cuh"
#include "packing.cuh"

namespace eob {

namespace {

constexpr int kSynthThreads = 256;
constexpr int kDataBlock = 2048;   // samples of the data per block of k_scan_chunks
constexpr int kMaxDataBlocks = 64;
// samples per work item of the strain modes: one per thread, as these batches
// are small (64 binaries of 8k samples: 512 items of 1024 for 152 SMs, whose
// last wave was two thirds empty)
constexpr int kStrainChunk = kSynthThreads;
constexpr int kFill = 4096;        // samples past the templates' ends per fill item

struct SynthArgs {
    int B, N, K;
    int mms[kMaxModes];
    double dt, amp;
    const double *data;   // lnL mode
    double *out;          // strain modes
    int vec;              // out is 16-byte aligned
};

// samples of a binary's template on the grid
__device__ __forceinline__ int used_samples(int np, int N) { return np <= 0 ? 0 : min(np, N); }

// Block 0: work items of `size` samples per binary and their exclusive scan.
// Blocks 1 ..: partial sums of data^2 (to the spline scratch, free by now) and
// the FP32 copy.  One block for everything took 42 us of a 1.5 ms pass at N = 2^17
// (a chain of 128 loads per thread), the split 6 us.
__global__ void __launch_bounds__(kScanThreads) k_scan_chunks(Ws w, int B, int N, int size, const double *data,
                                                               int mixed, int ndata)
{
    __shared__ long long sm[34];
    __shared__ double s_sq[kScanThreads / 32];
    const int tid = threadIdx.x;
    if (blockIdx.x > 0) {
        double sq = 0.0;
        for (int k = (blockIdx.x - 1) * kScanThreads + tid; k < N; k += ndata * kScanThreads) {
            const double d = data[k];
            sq = fma(d, d, sq);
            if (mixed) w.dataf[k] = (float)d;
        }
        for (int off = 16; off > 0; off >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, off);
        if ((tid & 31) == 0) s_sq[tid >> 5] = sq;
        __syncthreads();
        if (tid < 32) {
            sq = s_sq[tid];
            for (int off = 16; off > 0; off >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, off);
            if (tid == 0) w.cD[blockIdx.x - 1] = sq;
        }
        return;
    }
    const int per = (B + kScanThreads - 1) / kScanThreads;
    const int b0 = min(B, tid * per);
    const int b1 = min(B, b0 + per);
    long long chunks = 0;
    for (int b = b0; b < b1; ++b) chunks += (used_samples(w.npts[b], N) + size - 1) / size;
    long long total;
    long long co = block_exclusive_scan<kScanThreads>(chunks, sm, &total);
    for (int b = b0; b < b1; ++b) {
        w.chunk_off[b] = co;
        co += (used_samples(w.npts[b], N) + size - 1) / size;
    }
    if (tid == 0) {
        w.chunk_off[B] = total;
        w.queue[2] = (unsigned long long)total;
    }
}

// interval i in [lo, hi] with x[i] <= t < x[i+1] (searchsorted right - 1),
// given that it lies there; t, x >= 0: integer comparison of the IEEE bit
// patterns keeps the FP64 pipe free.
__device__ __forceinline__ int knot_index(const double *x, int lo, int hi, double t)
{
    const long long tb = __double_as_longlong(t);
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__double_as_longlong(x[mid]) <= tb) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// k >= 0 as a double, by integer operations (a conversion takes an FP64 issue slot)
__device__ __forceinline__ double index_value(int k)
{
    const int z = __clz(k);
    const unsigned long long m = (unsigned long long)(unsigned)k << (z + 21) & 0xfffffffffffffull;
    return k ? __longlong_as_double((long long)(m | ((unsigned long long)(1023 + 31 - z) << 52))) : 0.0;
}

// t_k = k dT + t0, at most tend (compared on the bits)
__device__ __forceinline__ double grid_time(int k, double dT, double t0, double tend)
{
    const double t = fma(index_value(k), dT, t0);
    return __double_as_longlong(t) > __double_as_longlong(tend) ? tend : t;
}

__device__ __forceinline__ double cubic(const double *y, const double *c1, const double *c2, const double *c3, size_t o,
                                        double x)
{
    return fma(fma(fma(c3[o], x, c2[o]), x, c1[o]), x, y[o]);
}

__device__ __forceinline__ void put_sample(const SynthArgs &sa, size_t i, double re, double im)
{
    if (sa.vec) {
        reinterpret_cast<double2 *>(sa.out)[i] = make_double2(re, im);
    } else {
        sa.out[2 * i] = re;
        sa.out[2 * i + 1] = im;
    }
}

// the merger-ringdown of one mode x = t - t_match after the match point
// (compute_MR_mode_free, eob/seobnrv4phm.py:1830-1843); tanh z = 1 - 2 / (1 + e^{2z})
__device__ __forceinline__ void ringdown_mode(const ImrRec &c, double x, double *hr, double *hi)
{
    const double z = fma(c.c1f, x, c.c2f);
    const double th = z >= 20.0 ? 1.0 : 1.0 - 2.0 * eob_rcp(1.0 + exp(2.0 * z));  // NaN stays NaN
    const double A = fma(c.c1c, th, c.c2c);
    const double ph = c.phi_match - c.d1c * eob_log(fma(c.d2f, exp(-c.d1f * x), 1.0) / (1.0 + c.d2f)) - c.om_re * x;
    const double mag = c.eta * A * exp(-c.om_im * x);
    double sp, cp;
    eob_sincos(ph, &sp, &cp);
    *hr = mag * cp;
    *hi = mag * sp;
}

// A block's run of chunks: consecutive work items, so that the binary and
// its knots change rarely; the runs of all blocks are equal within one chunk.
struct ChunkRun {
    long long c, end;
    int b;
    __device__ ChunkRun(const Ws &w, int B)
    {
        const long long C = (long long)w.queue[2];
        c = C * blockIdx.x / gridDim.x;
        end = C * (blockIdx.x + 1) / gridDim.x;
        b = c < end ? find_segment(w.chunk_off, B, c) : 0;
    }
    __device__ void next(const Ws &w)
    {
        ++c;
        while (c < end && c >= w.chunk_off[b + 1]) ++b;
    }
};

// the knot intervals of a chunk's first and last sample, by two threads
__device__ __forceinline__ void chunk_knots(const double *x, int n, int kbeg, int kend, double dT, double t0,
                                            double tend, int *s_range)
{
    if (threadIdx.x < 2)
        s_range[threadIdx.x] = knot_index(x, 0, n - 1, grid_time(threadIdx.x ? kend - 1 : kbeg, dT, t0, tend));
    __syncthreads();
}

// fixed-order sum of a value over the block's threads, on thread 0 (13 FP64
// instructions a block; a shuffle tree in every warp takes 48)
__device__ __forceinline__ double block_sum(double v, double *s_red)
{
    s_red[threadIdx.x] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x < 32) {
#pragma unroll
        for (int q = 0; q < kSynthThreads / 32; ++q) s += s_red[threadIdx.x + 32 * q];
        for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    }
    return s;
}

// What a block keeps of the binary it works on.
struct BinaryGrid {
    int np, n, last;   // samples; knots; samples from the splines (the ringdown follows)
    bool imr;
    size_t base;
    const double *x;
    double dT, t0, tend;
    __device__ BinaryGrid(const Ws &w, int b, double dt)
    {
        np = w.npts[b];
        n = w.nsteps[b];
        base = (size_t)w.row_off[b];
        // with the merger-ringdown: samples 0 .. idx are the NQC-corrected
        // inspiral, idx + 1 .. np - 1 the ringdown, zero beyond (per mode too)
        imr = w.imr_bin && w.imr_bin[b].on;
        last = imr ? min(np, w.imr_bin[b].idx + 1) : np;
        x = w.tin + base;
        dT = dt / (w.bins[b].Mt * kMTSUN_SI);
        t0 = np > 0 ? x[0] : 0.0;
        tend = np > 0 ? x[n - 1] : 0.0;
    }
};

// The modes of one sample in interval o = base + i at offset xx: per mode
// (MODE 2) into `put`, else their sum.  The phase takes 3 FP64 instructions, a mode
// 8 to 10 (two amplitude splines 6, the rotation 2 or 4; the NQC correction about 30
// for a sample and 9 for a mode); one mode took 62 with the library's sincos and products
// for the powers of xx.  Sines and cosines come from the integer phase
// (fasttrig.h), shared by modes of one m that follow one another.  FP64 issue
// (66 % of the slots) and the integers (33 % of all issue slots) bound it: 1024 ragged
// binaries, (2,2), 11 M samples: 1.43 -> 0.28 ms; 64 binaries, five modes with the
// merger-ringdown, strain of 24576 samples: 0.50 -> 0.14 ms.
template <int MODE, class Put>
__device__ __forceinline__ void spline_sample(const Ws &w, const SynthArgs &sa, const ImrRec *recs, size_t Rc, size_t o,
                                              double xx, double *hsum, double *hsum_i, Put put)
{
    const double phi = cubic(w.ys, w.cA, w.cB, w.cC, o, xx);
    double h = 0.0, hi = 0.0;
    const PhaseTurns phase(phi);
    if (!recs) {
        double sp = 0.0, cp = 0.0;
        for (int q = 0; q < sa.K; ++q) {
            if (q == 0 || sa.mms[q] != sa.mms[q - 1]) phase.multiple(sa.mms[q], &sp, &cp);
            const double re = cubic(w.ys, w.cA, w.cB, w.cC, (size_t)(1 + 2 * q) * Rc + o, xx);
            const double im = cubic(w.ys, w.cA, w.cB, w.cC, (size_t)(2 + 2 * q) * Rc + o, xx);
            // (re + i im) e^{-i m phi}
            if (MODE == 2) put(q, fma(re, cp, im * sp), fma(im, cp, -(re * sp)));
            else {
                h = fma(re, cp, fma(im, sp, h));
                if (MODE == 1) hi = fma(im, cp, fma(-re, sp, hi));
            }
        }
    } else {
        // NQC correction (EOBNonQCCorrection, eob/seobnrv4phm.py:1686-1700):
        // modulus 1 + (p_r / (r om))^2 (a1 + a2 / r + a3 / r^(3/2)), phase
        // p_r / (r om) (b1 + b2 p_r^2)
        const double om = fma(fma(3.0 * w.cC[o], xx, 2.0 * w.cB[o]), xx, w.cA[o]);
        const double rr = cubic(w.imr_ys, w.imr_cA, w.imr_cB, w.imr_cC, o, xx);
        const double pr = cubic(w.imr_ys, w.imr_cA, w.imr_cB, w.imr_cC, Rc + o, xx);
        const double rs = eob_rsqrt(rr), ir = rs * rs, ir32 = ir * rs;
        const double p0 = pr * eob_rcp(rr * om), p02 = p0 * p0, pr2 = pr * pr;
        for (int q = 0; q < sa.K; ++q) {
            const double re = cubic(w.ys, w.cA, w.cB, w.cC, (size_t)(1 + 2 * q) * Rc + o, xx);
            const double im = cubic(w.ys, w.cA, w.cB, w.cC, (size_t)(2 + 2 * q) * Rc + o, xx);
            const double mag = fma(p02, fma(recs[q].a3, ir32, fma(recs[q].a2, ir, recs[q].a1)), 1.0);
            double sp, cp;
            phase.multiple(sa.mms[q], -p0 * fma(recs[q].b2, pr2, recs[q].b1), &sp, &cp);
            const double a = fma(re, cp, im * sp) * mag, b = MODE == 0 ? 0.0 : fma(im, cp, -(re * sp)) * mag;
            if (MODE == 2) put(q, a, b);
            else {
                h += a;
                if (MODE == 1) hi += b;
            }
        }
    }
    *hsum = h;
    *hsum_i = hi;
}

// lnL: a run of chunks per block, one partial per chunk
__global__ void __launch_bounds__(kSynthThreads, 4) k_synth_lnl(Ws w, SynthArgs sa)
{
    __shared__ double s_red[kSynthThreads];
    __shared__ int s_range[2];
    const size_t Rc = (size_t)w.L.Bc * (size_t)w.L.Lc;
    ChunkRun run(w, sa.B);
    while (run.c < run.end) {
        const int b = run.b;
        const BinaryGrid g(w, b, sa.dt);
        const ImrRec *recs = g.imr ? w.imr_rec + (size_t)b * w.L.Kc : nullptr;
        for (; run.c < run.end && run.b == b; run.next(w)) {
            const int kbeg = (int)(run.c - w.chunk_off[b]) * kChunk;
            const int kend = min(used_samples(g.np, sa.N), kbeg + kChunk);
            __syncthreads();  // the last chunk's shared values are done with
            if (kbeg < g.last) chunk_knots(g.x, g.n, kbeg, min(kend, g.last), g.dT, g.t0, g.tend, s_range);
            double acc = 0.0;
            for (int k = kbeg + threadIdx.x; k < kend; k += kSynthThreads) {
                double h = 0.0, hi;
                if (k < g.last) {
                    const double t = grid_time(k, g.dT, g.t0, g.tend);
                    const int i = knot_index(g.x, s_range[0], s_range[1], t);
                    spline_sample<0>(w, sa, recs, Rc, g.base + i, t - g.x[i], &h, &hi, [](int, double, double) {});
                } else {
                    const double xr = (k - (g.last - 1)) * g.dT;
                    for (int q = 0; q < sa.K; ++q) {
                        double hr;
                        ringdown_mode(recs[q], xr, &hr, &hi);
                        h += hr;
                    }
                }
                const double hk = sa.amp * h;
                acc = fma(hk, hk - 2.0 * sa.data[k], acc);
            }
            acc = block_sum(acc, s_red);
            if (threadIdx.x == 0) w.partial[run.c] = acc;
        }
    }
}

// Strain (MODE 1: summed, 2: per mode): the templates in work items of one
// sample per thread, then the rest of every row: zero, or, per mode without
// the merger-ringdown, the value at the last knot (the uniform-grid hold
// of SEOBNRv4PHM.__call__).
template <int MODE>
__global__ void __launch_bounds__(kSynthThreads) k_synth_strain(Ws w, SynthArgs sa)
{
    __shared__ int s_range[2];
    const size_t Rc = (size_t)w.L.Bc * (size_t)w.L.Lc;
    const long long C = (long long)w.queue[2];
    for (long long c = blockIdx.x; c < C; c += gridDim.x) {
        const int b = find_segment(w.chunk_off, sa.B, c);
        const BinaryGrid g(w, b, sa.dt);
        const ImrRec *recs = g.imr ? w.imr_rec + (size_t)b * w.L.Kc : nullptr;
        const int kbeg = (int)(c - w.chunk_off[b]) * kStrainChunk, k = kbeg + threadIdx.x;
        const int kend = min(used_samples(g.np, sa.N), kbeg + kStrainChunk);
        __syncthreads();
        if (kbeg < g.last) chunk_knots(g.x, g.n, kbeg, min(kend, g.last), g.dT, g.t0, g.tend, s_range);
        if (k >= kend) continue;
        const auto put = [&](int q, double re, double im) {
            put_sample(sa, ((size_t)b * sa.K + q) * (size_t)sa.N + k, re, im);
        };
        double h = 0.0, hi = 0.0;
        if (k < g.last) {
            const double t = grid_time(k, g.dT, g.t0, g.tend);
            const int i = knot_index(g.x, s_range[0], s_range[1], t);
            spline_sample<MODE>(w, sa, recs, Rc, g.base + i, t - g.x[i], &h, &hi, put);
        } else {
            const double xr = (k - (g.last - 1)) * g.dT;
            for (int q = 0; q < sa.K; ++q) {
                double hr, him;
                ringdown_mode(recs[q], xr, &hr, &him);
                if (MODE == 2) put(q, hr, him);
                h += hr;
                hi += him;
            }
        }
        if (MODE == 1) put_sample(sa, (size_t)b * sa.N + k, h, hi);
    }
    const int segs = (sa.N + kFill - 1) / kFill;
    for (long long z = blockIdx.x; z < (long long)sa.B * segs; z += gridDim.x) {
        const int b = (int)(z / segs), lo = (int)(z % segs) * kFill, hi = min(sa.N, lo + kFill);
        const int from = max(lo, used_samples(w.npts[b], sa.N));
        if (from >= hi) continue;
        double hr[kMaxModes] = {}, hm[kMaxModes] = {};
        if (MODE == 2 && w.npts[b] > 0) {
            const BinaryGrid g(w, b, sa.dt);
            double s, si;
            if (!g.imr)
                spline_sample<2>(w, sa, nullptr, Rc, g.base + g.n - 1, 0.0, &s, &si, [&](int q, double re, double im) {
#pragma unroll
                    for (int p = 0; p < kMaxModes; ++p)
                        if (p == q) {
                            hr[p] = re;
                            hm[p] = im;
                        }
                });
        }
#pragma unroll
        for (int q = 0; q < kMaxModes; ++q) {
            if (q >= (MODE == 2 ? sa.K : 1)) break;
            const size_t at = (MODE == 2 ? (size_t)b * sa.K + q : (size_t)b) * (size_t)sa.N;
            for (int k = from + threadIdx.x; k < hi; k += kSynthThreads) put_sample(sa, at + k, hr[q], hm[q]);
        }
    }
}

// 2 pi u / 2^36 in [-pi, pi) as the nearest float, for the signed low 36 bits
// of u: their upper 16 and lower 20 bits times the constant in two floats,
// exact but for 1e-11 before the last rounding
__device__ __forceinline__ float turns_to_radians(unsigned long long u)
{
    const long long v = (long long)(u << 28);
    const float hi = (float)(int)(v >> 48), lo = (float)((unsigned)(v >> 28) & 0xfffffu);
    return fmaf(hi, 0x1.921fb6p-14f, fmaf(hi, -0x1.777a5cp-39f, lo * 0x1.921fb6p-34f));
}

// PLAIN: vector loads, no negative m.  Anything else a sample has to allow for (an
// unaligned workspace, signed products) costs 0.5 and 0.7 % of the kernel.
template <bool PLAIN>
__device__ __forceinline__ float4 load_f32(const float *p)
{
    if constexpr (PLAIN) return *reinterpret_cast<const float4 *>(p);
    else return make_float4(p[0], p[1], p[2], p[3]);
}

// Mixed precision: the phase spline and its reduction mod 2 pi run in FP64; the
// amplitude splines (FP32 coefficient copies written at spline
// build), sin/cos and the residual run in FP32.  One fused product with
// 1 / (2 pi) in FP64 leaves the phase in units of 2^-36 turn (9e-11 rad) in the
// low bits of the sum with 1.5 2^16; multiples of it are integer products,
// which wrap as the angle does, so every mode's reduction is free (the FP64
// reduction of each took 5 instructions of the 37 a five-mode sample had; 10 are
// left: 4096 binaries, five modes, 12 M samples: 0.95 -> 0.36 ms).
template <bool PLAIN>
__device__ __forceinline__ void mixed_sample(const Ws &w, const SynthArgs &sa, size_t Rc, size_t o, double xx,
                                             float *h_re, float *h_im)
{
    const double phi = cubic(w.ys, w.cA, w.cB, w.cC, o, xx);
    // to nearest (ties away): the truncated bits and the next one
    float xf = __uint_as_float(__float_as_uint(f32_trunc(xx)) + (((unsigned)__double2loint(xx) >> 28) & 1u));
    unsigned long long turn;
    if ((unsigned)(__double2hiint(phi) & 0x7fffffff) < 0x41000000u) {  // |phi| < 2^17
        turn = (unsigned long long)__double_as_longlong(fma(phi, 0.15915494309189533577, 98304.0));
    } else {
        const double u = phi * 0.15915494309189533577;
        turn = (unsigned long long)__double_as_longlong(u - rint(u) + 98304.0);
        if ((__double2hiint(phi) & 0x7ff00000) == 0x7ff00000) xf = __int_as_float(0x7fffffff);  // no number: NaN
    }
    float h = 0.0f, hi = 0.0f;
    for (int q = 0; q < sa.K; ++q) {
        const float4 a = load_f32<PLAIN>(w.f32 + 4 * ((size_t)(2 * q) * Rc + o));
        const float4 c = load_f32<PLAIN>(w.f32 + 4 * ((size_t)(2 * q + 1) * Rc + o));
        const float re = fmaf(xf, fmaf(xf, fmaf(xf, a.w, a.z), a.y), a.x);
        const float im = fmaf(xf, fmaf(xf, fmaf(xf, c.w, c.z), c.y), c.x);
        float sp, cp;
        const int m = sa.mms[q];
        sincosf(turns_to_radians(PLAIN ? (unsigned)m * turn : (unsigned long long)(long long)m * turn), &sp, &cp);
        // (re + i im) e^{-i m phi}
        h = fmaf(re, cp, fmaf(im, sp, h));
        hi = fmaf(im, cp, fmaf(-re, sp, hi));
    }
    *h_re = h;
    *h_im = hi;
}

// lnL with a Kahan-compensated FP32 sum per thread and FP64 chunk partials.
// The FP32 copies exist only if the spline build ran with precision 1
// (workspace flag queue[6]), and the merger-ringdown runs in FP64 only;
// otherwise the lnL comes out NaN.
template <bool PLAIN>
__global__ void __launch_bounds__(kSynthThreads) k_synth_mixed_lnl(Ws w, SynthArgs sa)
{
    __shared__ double s_red[kSynthThreads];
    __shared__ int s_range[2];
    const bool have_f32 = w.queue[6] == 1ull;
    const size_t Rc = (size_t)w.L.Bc * (size_t)w.L.Lc;
    ChunkRun run(w, sa.B);
    while (run.c < run.end) {
        const int b = run.b;
        const BinaryGrid g(w, b, sa.dt);
        for (; run.c < run.end && run.b == b; run.next(w)) {
            const int kbeg = (int)(run.c - w.chunk_off[b]) * kChunk;
            const int kend = (have_f32 && !g.imr) ? min(used_samples(g.np, sa.N), kbeg + kChunk) : kbeg;
            __syncthreads();  // the last chunk's shared values are done with
            if (kbeg < kend) chunk_knots(g.x, g.n, kbeg, kend, g.dT, g.t0, g.tend, s_range);
            float acc = 0.0f, comp = 0.0f;
            for (int k = kbeg + threadIdx.x; k < kend; k += kSynthThreads) {
                const double t = grid_time(k, g.dT, g.t0, g.tend);
                const int i = knot_index(g.x, s_range[0], s_range[1], t);
                float h, hi;
                mixed_sample<PLAIN>(w, sa, Rc, g.base + i, t - g.x[i], &h, &hi);
                const float hk = (float)sa.amp * h;
                const float term = hk * (hk - 2.0f * w.dataf[k]);
                // Kahan summation
                const float yv = term - comp;
                const float tv = acc + yv;
                comp = (tv - acc) - yv;
                acc = tv;
            }
            const double sum = block_sum((double)acc - (double)comp, s_red);
            if (threadIdx.x == 0) w.partial[run.c] = kbeg < kend ? sum : __longlong_as_double(0x7ff8000000000000ll);
        }
    }
}

// summed strain, zero past each waveform's end (and without the FP32 copies)
template <bool PLAIN>
__global__ void __launch_bounds__(kSynthThreads) k_synth_mixed_strain(Ws w, SynthArgs sa)
{
    __shared__ int s_range[2];
    const bool have_f32 = w.queue[6] == 1ull;
    const size_t Rc = (size_t)w.L.Bc * (size_t)w.L.Lc;
    const long long C = (long long)w.queue[2];
    for (long long c = blockIdx.x; c < C; c += gridDim.x) {
        const int b = find_segment(w.chunk_off, sa.B, c);
        const BinaryGrid g(w, b, sa.dt);
        const int kbeg = (int)(c - w.chunk_off[b]) * kStrainChunk, k = kbeg + threadIdx.x;
        const int kend = min(used_samples(g.np, sa.N), kbeg + kStrainChunk);
        __syncthreads();
        chunk_knots(g.x, g.n, kbeg, kend, g.dT, g.t0, g.tend, s_range);
        if (k >= kend) continue;
        float h = 0.0f, hi = 0.0f;
        if (have_f32) {
            const double t = grid_time(k, g.dT, g.t0, g.tend);
            const int i = knot_index(g.x, s_range[0], s_range[1], t);
            mixed_sample<PLAIN>(w, sa, Rc, g.base + i, t - g.x[i], &h, &hi);
        }
        put_sample(sa, (size_t)b * sa.N + k, (double)h, (double)hi);
    }
    const int segs = (sa.N + kFill - 1) / kFill;
    for (long long z = blockIdx.x; z < (long long)sa.B * segs; z += gridDim.x) {
        const int b = (int)(z / segs), lo = (int)(z % segs) * kFill, hi = min(sa.N, lo + kFill);
        for (int k = max(lo, used_samples(w.npts[b], sa.N)) + threadIdx.x; k < hi; k += kSynthThreads)
            put_sample(sa, (size_t)b * sa.N + k, 0.0, 0.0);
    }
}

// one warp per binary
__global__ void __launch_bounds__(128) k_finalize(Ws w, int B, int ndata, double *lnl, int *status_out)
{
    const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (b >= B) return;
    if (lane == 0 && status_out) status_out[b] = w.status[b];
    if (!lnl) return;
    double s = 0.0, dsq = 0.0;
    for (long long c = w.chunk_off[b] + lane; c < w.chunk_off[b + 1]; c += 32) s += w.partial[c];
    for (int q = lane; q < ndata; q += 32) dsq += w.cD[q];
    s += dsq;
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (lane == 0) lnl[b] = w.npts[b] <= 0 ? __longlong_as_double(0x7ff8000000000000LL) : -0.5 * s;
}

}  // namespace

cudaError_t launch_synth(const Ws &w, const RunArgs &a, int mode, double *out, cudaStream_t s)
{
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int mixed = (mode != 2 && a.opt.precision == 1 && !a.opt.imr) ? 1 : 0;
    int ndata = 0;
    if (mode == 0) {
        // at least 12 doubles of scratch: 4 rows of 3 series
        const size_t room = (size_t)w.L.Bc * w.L.Lc * w.L.nsubs;
        ndata = (a.N + kDataBlock - 1) / kDataBlock;
        if (ndata > kMaxDataBlocks) ndata = kMaxDataBlocks;
        if ((size_t)ndata > room) ndata = (int)room;
    }
    k_scan_chunks<<<1 + ndata, kScanThreads, 0, s>>>(w, a.B, a.N, mode == 0 ? kChunk : kStrainChunk, a.data, mixed,
                                                     ndata);
    SynthArgs sa;
    sa.B = a.B;
    sa.N = a.N;
    sa.K = a.K;
    for (int j = 0; j < kMaxModes; ++j) sa.mms[j] = a.mms[j];
    sa.dt = a.dt;
    sa.amp = a.amp;
    sa.data = a.data;
    sa.out = out;
    sa.vec = (reinterpret_cast<uintptr_t>(out) & 15) == 0 ? 1 : 0;
    void (*kern)(Ws, SynthArgs) = mode == 0 ? k_synth_lnl : mode == 2 ? k_synth_strain<2> : k_synth_strain<1>;
    if (mixed) {
        bool plain = w.f32_vec();
        for (int j = 0; j < a.K; ++j) plain = plain && a.mms[j] >= 0;
        if (mode == 0) kern = plain ? k_synth_mixed_lnl<true> : k_synth_mixed_lnl<false>;
        else kern = plain ? k_synth_mixed_strain<true> : k_synth_mixed_strain<false>;
    }
    const int blocks = mode == 0 ? resident_blocks(kern, kSynthThreads) : nsm * 8;
    kern<<<blocks, kSynthThreads, 0, s>>>(w, sa);
    k_finalize<<<(a.B + 3) / 4, 128, 0, s>>>(w, a.B, ndata, mode == 0 ? a.lnl : nullptr, a.status_out);
    return cudaGetLastError();
}

}  // namespace eob
