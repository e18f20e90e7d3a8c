// After the integrator: packing, multipoles on the trajectory, batched
// not-a-knot splines, and the fused synthesis + likelihood pass.
//
//  k_scan_*    one block: per-binary row counts and waveform sample counts,
//              exclusive scans (packed ragged layout), sum of data^2.
//  k_modes     one thread per packed trajectory row: h_lm e^{i m phi} for the
//              requested modes (get_hlms, eob/seobnrv4phm.py:2138-2221, and
//              the de-rotation of compute_full_waveform, :2331).
//  k_spline    one block per binary (and group of series): not-a-knot cubic
//              splines with the reference's tridiagonal set-up
//              (src/interpolate.cu:10-267), the matrix factorised once per
//              binary and solved by scans (spline_block.cuh).
//  k_synth     one block per 1024-sample chunk of one binary: spline
//              evaluation on the uniform grid (eob/seobnrv4phm.py:274-386,
//              2310-2372), mode sum (BBHWaveformTD, :715-721) and the
//              white-noise residual, reduced to one partial per chunk; in
//              likelihood mode the strain is never written to memory.
//  k_finalize  per binary, partials summed in a fixed order (deterministic).
#include "eob_device.cuh"
#include "spline_block.cuh"

namespace eob {

constexpr int kScanThreads = 1024;

__device__ __forceinline__ double t_in_of(double t_M, double Mt)
{
    // reference: t[s] = t_M * mt * MTSUN_SI, then t / (M * MTSUN_SI)
    return (t_M * Mt * kMTSUN_SI) / (Mt * kMTSUN_SI);
}

// number of uniform samples of binary b: int((t_end - t_0) / dT) + 1
__device__ int binary_npts(const double *tr, int L, double Mt, double dt)
{
    const double t0 = t_in_of(tr[0], Mt);
    const double t1 = t_in_of(tr[(size_t)(L - 1) * kTrajStride], Mt);
    const double dT = dt / (Mt * kMTSUN_SI);
    return (int)((t1 - t0) / dT) + 1;
}

// block-wide exclusive scan helper: returns the exclusive prefix of v over the block
template <int NT>
__device__ long long block_exclusive_scan(long long v, long long *sm, long long *total)
{
    const int tid = threadIdx.x;
    sm[tid] = v;
    __syncthreads();
    for (int off = 1; off < NT; off <<= 1) {
        const long long add = (tid >= off) ? sm[tid - off] : 0;
        __syncthreads();
        sm[tid] += add;
        __syncthreads();
    }
    const long long incl = sm[tid];
    if (total) *total = sm[NT - 1];
    __syncthreads();
    return incl - v;
}

// rows and uniform-grid sample counts per binary; packed row offsets
__global__ void __launch_bounds__(kScanThreads) k_scan_rows(Ws w, int B, double dt)
{
    __shared__ long long sm[kScanThreads];
    const int tid = threadIdx.x;
    const int per = (B + kScanThreads - 1) / kScanThreads;
    const int b0 = tid * per;
    const int b1 = min(B, b0 + per);
    long long rows = 0;
    for (int b = b0; b < b1; ++b) {
        const int L = w.nsteps[b];
        int st = w.status[b];
        int np = 0;
        if (L >= 3 && !(st & (EOB_ST_NAN | EOB_ST_TRIES | EOB_ST_SHORT))) {
            np = binary_npts(w.traj + (size_t)b * w.L.Lc * kTrajStride, L, w.bins[b].Mt, dt);
            if (np < 1) np = 0;
        } else {
            st |= EOB_ST_SHORT;
            w.status[b] = st;
        }
        w.npts[b] = np;
        rows += (np > 0) ? L : 0;
    }
    long long total;
    long long ro = block_exclusive_scan<kScanThreads>(rows, sm, &total);
    for (int b = b0; b < b1; ++b) {
        w.row_off[b] = ro;
        ro += (w.npts[b] > 0) ? w.nsteps[b] : 0;
    }
    if (tid == 0) {
        w.row_off[B] = total;
        w.queue[1] = (unsigned long long)total;
        *(unsigned long long *)w.partial = 0;  // k_modes counts its close rows here
    }
}

// synthesis work items: chunks of kChunk samples of min(npts, N) samples per
// binary (all N samples when cover_all); sum of data^2
__global__ void __launch_bounds__(kScanThreads) k_scan_chunks(Ws w, int B, int N, int cover_all, const double *data,
                                                               int mixed)
{
    __shared__ long long sm[kScanThreads];
    __shared__ double s_sq[kScanThreads];
    const int tid = threadIdx.x;
    const int per = (B + kScanThreads - 1) / kScanThreads;
    const int b0 = tid * per;
    const int b1 = min(B, b0 + per);
    long long chunks = 0;
    for (int b = b0; b < b1; ++b) {
        const int np = w.npts[b];
        const int nuse = (np <= 0) ? 0 : (cover_all ? N : (np < N ? np : N));
        chunks += (nuse + kChunk - 1) / kChunk;
    }
    double sq = 0.0;
    if (data)
        for (int k = tid; k < N; k += kScanThreads) {
            sq += data[k] * data[k];
            if (mixed) w.dataf[k] = (float)data[k];
        }
    s_sq[tid] = sq;
    long long total;
    long long co = block_exclusive_scan<kScanThreads>(chunks, sm, &total);
    for (int b = b0; b < b1; ++b) {
        w.chunk_off[b] = co;
        const int np = w.npts[b];
        const int nuse = (np <= 0) ? 0 : (cover_all ? N : (np < N ? np : N));
        co += (nuse + kChunk - 1) / kChunk;
    }
    for (int off = kScanThreads / 2; off > 0; off >>= 1) {
        if (tid < off) s_sq[tid] += s_sq[tid + off];
        __syncthreads();
    }
    if (tid == 0) {
        w.chunk_off[B] = total;
        w.queue[2] = (unsigned long long)total;
        w.queue[3] = (unsigned long long)__double_as_longlong(s_sq[0]);
    }
}

// index b with off[b] <= v < off[b+1]
__device__ __forceinline__ int find_segment(const long long *off, int B, long long v)
{
    int lo = 0, hi = B;  // answer in [lo, hi)
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (off[mid] <= v) lo = mid; else hi = mid;
    }
    return lo;
}

// rows closer than this to a neighbour [M] keep the log-Gamma sums (mode_eval.h); the
// fine pass steps by 0.05 and halves
constexpr double kCloseRows = 0.04;

struct ModeArgs {
    int K;
    int ells[kMaxModes], mms[kMaxModes];
    ModeConst mc[kMaxModes];
    int imr;  // also r and p_r as series for the merger-ringdown attachment
};

// Rows closer than kCloseRows to a neighbour are listed (in the spline
// scratch, which is free until the splines) for k_modes_close: the two
// evaluations in one kernel cost the others their registers and half the
// instruction cache (five modes, 4096 binaries, splines included: 5.8 ms
// against 4.2 ms).  FP64 issue bounds both: five modes and the Hamiltonian
// take 645 FP64 instructions a row in the closed form, 2427 by the sums on
// every row (4096 binaries: 9.32 ms -> 2.49 + 0.56 ms; 1024 ragged binaries,
// (2,2) alone: 0.77 -> 0.36 + 0.07 ms).
__global__ void __launch_bounds__(128) k_modes(Ws w, int B, ModeArgs ma)
{
    const long long R = (long long)w.queue[1];
    const size_t Rc = (size_t)w.L.Bc * (size_t)w.L.Lc;
    long long *list = (long long *)w.cD;
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < R; r += (long long)gridDim.x * blockDim.x) {
        const int b = find_segment(w.row_off, B, r);
        const int i = (int)(r - w.row_off[b]);
        const BinaryRec &rec = w.bins[b];
        const double *row = w.traj + ((size_t)b * w.L.Lc + i) * kTrajStride;
        const double rr = row[1], phi = row[2], pr = row[3], pphi = row[4];
        const bool close = (i > 0 && row[0] - row[-kTrajStride] < kCloseRows) ||
                           (i + 1 < w.nsteps[b] && row[kTrajStride] - row[0] < kCloseRows);
        w.tin[r] = t_in_of(row[0], rec.Mt);
        w.ys[r] = phi;
        if (ma.imr) {
            w.imr_ys[r] = rr;
            w.imr_ys[Rc + r] = pr;
        }
        if (close) {
            list[atomicAdd((unsigned long long *)w.partial, 1ull)] = r;
            continue;
        }
        HamEval e;
        ham_eval(rec.ham, rr, pr, pphi, &e);
        // v = omega^(1/3); v_phi = r (omega_c^2 r^3)^(-1/3) omega = omega omega_c^(-2/3)
        const double ro = eob_rcbrt(e.dHdL), rc = eob_rcbrt(e.omega_c);
        const ModeRow mr = mode_row(e.dHdL * (ro * ro), e.Hreal, e.dHdL * (rc * rc), pphi, rec.flux.inv2eta, phi);
        for (int j = 0; j < ma.K; ++j) {
            const int l = ma.ells[j], m = ma.mms[j];
            const int li = lm_index(l, m);
            const cdbl hl = mode_term(w.fac[b], l, m, ma.mc[j], mr, rec.pre_re[li], rec.pre_im[li], rec.nu, 0.0, true);
            w.ys[(size_t)(1 + 2 * j) * Rc + r] = hl.re;
            w.ys[(size_t)(2 + 2 * j) * Rc + r] = hl.im;
        }
    }
}

// The listed rows, by the log-Gamma sums: one thread per row, or per row and
// mode while the list is short.
__global__ void __launch_bounds__(128) k_modes_close(Ws w, int B, ModeArgs ma)
{
    // log l! for l = 0..8, summed as mode_eval_sums would
    __shared__ double lfact[kLMax + 1];
    if (threadIdx.x <= kLMax) {
        double f = 0.0;
        for (int q = 2; q <= (int)threadIdx.x; ++q) f += log((double)q);
        lfact[threadIdx.x] = f;
    }
    __syncthreads();
    const long long *list = (const long long *)w.cD;
    const long long C = *(const long long *)w.partial, nt = (long long)gridDim.x * blockDim.x;
    const size_t Rc = (size_t)w.L.Bc * (size_t)w.L.Lc;
    const int per = (C * ma.K <= nt) ? 1 : ma.K, parts = ma.K / per;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < C * parts; c += nt) {
        const long long r = list[c % C];
        const int j0 = (int)(c / C) * per;
        const int b = find_segment(w.row_off, B, r);
        const int i = (int)(r - w.row_off[b]);
        const BinaryRec &rec = w.bins[b];
        const double *row = w.traj + ((size_t)b * w.L.Lc + i) * kTrajStride;
        const double rr = row[1], phi = row[2], pr = row[3], pphi = row[4];
        HamEval e;
        ham_eval(rec.ham, rr, pr, pphi, &e);
        const double v = cbrt(e.dHdL);
        const double vphi_in = 1.0 / (e.omega_c * e.omega_c * rr * rr * rr);
        const double Omega = v * v * v, vh = cbrt(e.Hreal * Omega), vPhi = rr * cbrt(vphi_in) * Omega;
        for (int j = j0; j < j0 + per; ++j) {
            const int l = ma.ells[j], m = ma.mms[j];
            const int li = lm_index(l, m);
            const cdbl hl = mode_eval_sums(w.fac[b], l, m, rec.pre_re[li], rec.pre_im[li], rec.nu, phi, pphi, v, vh,
                                           e.Hreal, vPhi, lfact[l], 0.0, true);
            w.ys[(size_t)(1 + 2 * j) * Rc + r] = hl.re;
            w.ys[(size_t)(2 + 2 * j) * Rc + r] = hl.im;
        }
    }
}

// The splines of one binary in the packed layout, for SplineBlock: series
// 0 .. nmain - 1 are the phase and the modes; nmain, nmain + 1 are r and p_r
// of the merger-ringdown section.
struct PackedSplines {
    static constexpr bool kExact = false, kKeepSlopes = false;
    const Ws &w;
    int n, nmain;
    size_t base, Rc;
    bool mixed;
    __device__ int rows(int) const { return n; }
    __device__ const double *knots(int) const { return w.tin + base; }
    __device__ size_t knot_stride() const { return 1; }
    __device__ size_t row_stride() const { return 1; }
    __device__ SplineSeries series(int, int s) const
    {
        const bool extra = s >= nmain;
        const size_t o = (size_t)(extra ? s - nmain : s) * Rc + base;
        if (extra) return {w.imr_ys + o, w.imr_cA + o, w.imr_cB + o, w.imr_cC + o, w.imr_cD + o};
        return {w.ys + o, w.cA + o, w.cB + o, w.cC + o, w.cD + o};
    }
    __device__ void put(int, int s, int i, const SplineSeries &f, double c1, double c2, double c3) const
    {
        f.c1[i] = c1;
        f.c2[i] = c2;
        f.c3[i] = c3;
        if (mixed && s >= 1 && s < nmain) {
            // FP32 copies of the amplitude series for the mixed-precision synthesis
            const size_t S = (size_t)2 * w.L.Kc * Rc;
            float *q = w.f32 + (size_t)(s - 1) * Rc + base + i;
            q[0] = (float)f.y[i];
            q[S] = (float)c1;
            q[2 * S] = (float)c2;
            q[3 * S] = (float)c3;
        }
    }
    __device__ void put_last(int b, int s, int i, const SplineSeries &f, double, double, double) const
    {
        put(b, s, i, f, 0.0, 0.0, 0.0);
    }
};

constexpr int kSplineThreads = 64, kSplineChunk = 13;
using PackedBlock = SplineBlock<1, kSplineThreads, kSplineChunk>;

// One block per binary and group of `per` series, in the caller's queue order
// (longest first: several tiles long, they would end the launch).  64 threads
// of up to 13 rows: 832 rows a tile, which most trajectories fit (520 rows in
// 9 per thread); 128 threads of 5 rows would spend a quarter more FP64 issue
// slots on the scans.  Measured: 4096 binaries, 11 series, 520 rows: 4.67 ms
// -> 1.09 ms (80 % of the FP64 issue slots); 1024 ragged binaries, 3 series:
// 0.81 -> 0.39 ms (the longest, 4 tiles, ends it).
__global__ void __launch_bounds__(kSplineThreads) k_spline(Ws w, const int *order, int nsubs, int nmain, int per,
                                                           int mixed)
{
    __shared__ PackedBlock::Smem sm;
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) w.queue[6] = (unsigned long long)mixed;
    const int b = order ? order[blockIdx.x] : blockIdx.x;
    const PackedSplines acc{w, w.npts[b] > 0 ? w.nsteps[b] : 0, nmain, (size_t)w.row_off[b],
                            (size_t)w.L.Bc * (size_t)w.L.Lc, mixed != 0};
    const int s0 = blockIdx.y * per;
    PackedBlock::run(acc, sm, s0, min(nsubs, s0 + per));
}

struct SynthArgs {
    int B, N, K;
    int mms[kMaxModes];
    double dt, amp;
    const double *data;   // lnL mode
    double *out;          // strain modes
    int mode;             // 0: lnL, 1: summed strain (zero past the end), 2: per mode, t clamped to the end
};

// interval i with x[i] <= t < x[i+1] (searchsorted right - 1), t, x >= 0:
// integer comparison of the IEEE bit patterns keeps the FP64 pipe free.
__device__ __forceinline__ int knot_index(const double *x, int n, double t)
{
    const long long tb = __double_as_longlong(t);
    int lo = 0, hi = n;  // first index with x > t lies in [lo, hi]
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__double_as_longlong(x[mid]) <= tb) lo = mid + 1; else hi = mid;
    }
    int i = lo - 1;
    if (i < 0) i = 0;
    if (i > n - 1) i = n - 1;
    return i;
}

// the merger-ringdown of one mode x = t - t_match after the match point
// (compute_MR_mode_free, eob/seobnrv4phm.py:1830-1843)
__device__ __forceinline__ void ringdown_mode(const ImrRec &c, double x, double *hr, double *hi)
{
    const double A = c.c1c * tanh(c.c1f * x + c.c2f) + c.c2c;
    const double ph = c.phi_match - c.d1c * log((1 + c.d2f * exp(-c.d1f * x)) / (1 + c.d2f)) - c.om_re * x;
    const double mag = c.eta * A * exp(-c.om_im * x);
    double sp, cp;
    sincos(ph, &sp, &cp);
    *hr = mag * cp;
    *hi = mag * sp;
}

__global__ void __launch_bounds__(256) k_synth(Ws w, SynthArgs sa)
{
    __shared__ double s_red[256 / 32];
    const long long C = (long long)w.queue[2];
    const size_t Rc = (size_t)w.L.Bc * (size_t)w.L.Lc;
    for (long long c = blockIdx.x; c < C; c += gridDim.x) {
        const int b = find_segment(w.chunk_off, sa.B, c);
        const int j = (int)(c - w.chunk_off[b]);
        const int np = w.npts[b];
        // with the merger-ringdown: samples 0 .. idx are the NQC-corrected
        // inspiral, idx + 1 .. np - 1 the ringdown, zero beyond (per mode too)
        const bool imr = w.imr_bin && w.imr_bin[b].on;
        const int idx = imr ? w.imr_bin[b].idx : np;
        const int nuse = (sa.mode == 2) ? sa.N : (np < sa.N ? np : sa.N);
        const int n = w.nsteps[b];
        const size_t base = (size_t)w.row_off[b];
        const double *x = w.tin + base;
        const double Mts = w.bins[b].Mt * kMTSUN_SI;
        const double dT = sa.dt / Mts;
        const double t0 = x[0], tend = x[n - 1];
        const ImrRec *recs = imr ? w.imr_rec + (size_t)b * w.L.Kc : nullptr;
        double acc = 0.0;
        const int kbeg = j * kChunk;
        const int kend = min(nuse, kbeg + kChunk);
        for (int k = kbeg + threadIdx.x; k < kend; k += blockDim.x) {
            double hsum = 0.0, hsum_i = 0.0;
            if (imr && k > idx) {
                if (k < np) {
                    const double xr = (k - idx) * dT;
                    for (int q = 0; q < sa.K; ++q) {
                        double hr, hi;
                        ringdown_mode(recs[q], xr, &hr, &hi);
                        if (sa.mode == 2) {
                            const size_t oo = 2 * (((size_t)b * sa.K + q) * (size_t)sa.N + k);
                            sa.out[oo] = hr;
                            sa.out[oo + 1] = hi;
                        }
                        hsum += hr;
                        hsum_i += hi;
                    }
                } else if (sa.mode == 2) {
                    for (int q = 0; q < sa.K; ++q) {
                        const size_t oo = 2 * (((size_t)b * sa.K + q) * (size_t)sa.N + k);
                        sa.out[oo] = 0.0;
                        sa.out[oo + 1] = 0.0;
                    }
                }
                if (sa.mode == 1) {
                    sa.out[2 * ((size_t)b * sa.N + k)] = hsum;
                    sa.out[2 * ((size_t)b * sa.N + k) + 1] = hsum_i;
                } else if (sa.mode == 0) {
                    const double hk = sa.amp * hsum;
                    acc += hk * hk - 2.0 * sa.data[k] * hk;
                }
                continue;
            }
            double t = k * dT + t0;
            if (t > tend) t = tend;
            const int i = knot_index(x, n, t);
            const double xx = t - x[i], x2 = xx * xx, x3 = x2 * xx;
            const size_t o = base + i;
            const double phi = w.ys[o] + w.cA[o] * xx + w.cB[o] * x2 + w.cC[o] * x3;
            double rr = 0.0, pr = 0.0, om = 0.0;
            if (imr) {
                om = w.cA[o] + 2 * w.cB[o] * xx + 3 * w.cC[o] * x2;
                rr = w.imr_ys[o] + w.imr_cA[o] * xx + w.imr_cB[o] * x2 + w.imr_cC[o] * x3;
                const size_t op = Rc + o;
                pr = w.imr_ys[op] + w.imr_cA[op] * xx + w.imr_cB[op] * x2 + w.imr_cC[op] * x3;
            }
            for (int q = 0; q < sa.K; ++q) {
                const size_t orr = (size_t)(1 + 2 * q) * Rc + o, oi = (size_t)(2 + 2 * q) * Rc + o;
                const double re = w.ys[orr] + w.cA[orr] * xx + w.cB[orr] * x2 + w.cC[orr] * x3;
                const double im = w.ys[oi] + w.cA[oi] * xx + w.cB[oi] * x2 + w.cC[oi] * x3;
                double sp, cp;
                sincos(sa.mms[q] * phi, &sp, &cp);
                // (re + i im) e^{-i m phi}
                double hr = re * cp + im * sp, hi = im * cp - re * sp;
                if (imr) {
                    // NQC correction (EOBNonQCCorrection, eob/seobnrv4phm.py:1686-1700)
                    const ImrRec &cq = recs[q];
                    const double sr = sqrt(rr), rO = rr * om;
                    const double mag = 1.0 + (pr * pr / (rO * rO)) * (cq.a1 + cq.a2 / rr + cq.a3 / (rr * sr));
                    const double nph = cq.b1 * pr / rO + pr * pr * pr / rO * cq.b2;
                    double ns, nc;
                    sincos(nph, &ns, &nc);
                    const double tr = mag * (hr * nc - hi * ns);
                    hi = mag * (hr * ns + hi * nc);
                    hr = tr;
                }
                if (sa.mode == 2) {
                    const size_t oo = 2 * (((size_t)b * sa.K + q) * (size_t)sa.N + k);
                    sa.out[oo] = hr;
                    sa.out[oo + 1] = hi;
                }
                hsum += hr;
                hsum_i += hi;
            }
            if (sa.mode == 1) {
                sa.out[2 * ((size_t)b * sa.N + k)] = hsum;
                sa.out[2 * ((size_t)b * sa.N + k) + 1] = hsum_i;
            } else if (sa.mode == 0) {
                const double hk = sa.amp * hsum;
                acc += hk * hk - 2.0 * sa.data[k] * hk;
            }
        }
        // block reduction (fixed order)
        for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
        if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0 && sa.mode == 0) {
            double s = 0.0;
            for (int q = 0; q < (int)(blockDim.x >> 5); ++q) s += s_red[q];
            w.partial[c] = s;
        }
        __syncthreads();
    }
}

// Mixed precision synthesis: the phase spline and its reduction mod 2 pi run
// in FP64; the amplitude splines (FP32 coefficient copies written at spline
// build), sin/cos and the residual run in FP32.  mode 0 accumulates the lnL
// terms with a Kahan-compensated FP32 sum per thread and FP64 chunk partials;
// mode 1 writes the summed strain (zero past each waveform's end).  The
// FP32 copies exist only if the spline build ran with precision 1 (workspace
// flag queue[6]); otherwise the lnL comes out NaN.
__global__ void __launch_bounds__(256) k_synth_mixed(Ws w, SynthArgs sa)
{
    __shared__ double s_red[256 / 32];
    const long long C = (long long)w.queue[2];
    const bool have_f32 = w.queue[6] == 1ull;
    const size_t Rc = (size_t)w.L.Bc * (size_t)w.L.Lc;
    const size_t S = (size_t)2 * w.L.Kc * Rc;
    const double two_pi_hi = 6.283185307179586232, two_pi_lo = 2.4492935982947064e-16;
    for (long long c = blockIdx.x; c < C; c += gridDim.x) {
        const int b = find_segment(w.chunk_off, sa.B, c);
        const int j = (int)(c - w.chunk_off[b]);
        const int np = w.npts[b];
        const int nuse = np < sa.N ? np : sa.N;
        // the merger-ringdown runs in the FP64 synthesis only
        const bool imr_bin = w.imr_bin && w.imr_bin[b].on;
        const int n = w.nsteps[b];
        const size_t base = (size_t)w.row_off[b];
        const double *x = w.tin + base;
        const double Mts = w.bins[b].Mt * kMTSUN_SI;
        const double dT = sa.dt / Mts;
        const double t0 = x[0], tend = x[n - 1];
        float acc = 0.0f, comp = 0.0f;
        const int kbeg = j * kChunk;
        const int kend = have_f32 ? min(nuse, kbeg + kChunk) : kbeg;
        for (int k = kbeg + threadIdx.x; k < kend; k += blockDim.x) {
            double t = k * dT + t0;
            if (t > tend) t = tend;
            const int i = knot_index(x, n, t);
            const double xx = t - x[i];
            const size_t o = base + i;
            const double phi = w.ys[o] + xx * (w.cA[o] + xx * (w.cB[o] + xx * w.cC[o]));
            const float xf = (float)xx;
            float h = 0.0f, hi = 0.0f;
            for (int q = 0; q < sa.K; ++q) {
                const size_t orr = (size_t)(2 * q) * Rc + o, oi = (size_t)(2 * q + 1) * Rc + o;
                const float re = w.f32[orr] + xf * (w.f32[S + orr] + xf * (w.f32[2 * S + orr] + xf * w.f32[3 * S + orr]));
                const float im = w.f32[oi] + xf * (w.f32[S + oi] + xf * (w.f32[2 * S + oi] + xf * w.f32[3 * S + oi]));
                const double ph = sa.mms[q] * phi;
                const double nn = rint(ph * 0.15915494309189533577);
                const double red = fma(-nn, two_pi_lo, fma(-nn, two_pi_hi, ph));
                float sp, cp;
                sincosf((float)red, &sp, &cp);
                // (re + i im) e^{-i m phi}
                h = fmaf(re, cp, fmaf(im, sp, h));
                hi = fmaf(im, cp, fmaf(-re, sp, hi));
            }
            if (sa.mode == 1) {
                sa.out[2 * ((size_t)b * sa.N + k)] = (double)h;
                sa.out[2 * ((size_t)b * sa.N + k) + 1] = (double)hi;
            } else {
                const float hk = (float)sa.amp * h;
                const float term = hk * (hk - 2.0f * w.dataf[k]);
                // Kahan summation
                const float yv = term - comp;
                const float tv = acc + yv;
                comp = (tv - acc) - yv;
                acc = tv;
            }
        }
        double dacc = (double)acc - (double)comp;
        for (int off = 16; off > 0; off >>= 1) dacc += __shfl_down_sync(0xffffffffu, dacc, off);
        if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = dacc;
        __syncthreads();
        if (threadIdx.x == 0 && sa.mode == 0) {
            double sum = 0.0;
            for (int q = 0; q < (int)(blockDim.x >> 5); ++q) sum += s_red[q];
            w.partial[c] = (have_f32 && !imr_bin) ? sum : __longlong_as_double(0x7ff8000000000000ll);
        }
        __syncthreads();
    }
}

__global__ void k_finalize(Ws w, int B, double *lnl, int *status_out)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= B) return;
    const double dsq = __longlong_as_double((long long)w.queue[3]);
    const int st = w.status[b];
    double s = 0.0;
    for (long long c = w.chunk_off[b]; c < w.chunk_off[b + 1]; ++c) s += w.partial[c];
    const bool bad = (w.npts[b] <= 0);
    if (lnl) lnl[b] = bad ? __longlong_as_double(0x7ff8000000000000LL) : -0.5 * (dsq + s);
    if (status_out) status_out[b] = st;
}

cudaError_t launch_prepare_post(const Ws &w, const RunArgs &a, cudaStream_t s)
{
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    k_scan_rows<<<1, kScanThreads, 0, s>>>(w, a.B, a.dt);
    ModeArgs ma;
    ma.K = a.K;
    for (int j = 0; j < kMaxModes; ++j) { ma.ells[j] = a.ells[j]; ma.mms[j] = a.mms[j]; }
    for (int j = 0; j < a.K; ++j) ma.mc[j] = mode_const(a.ells[j], a.mms[j]);
    ma.imr = (a.opt.imr && w.imr_ys) ? 1 : 0;
    k_modes<<<nsm * 8, 128, 0, s>>>(w, a.B, ma);
    k_modes_close<<<nsm * 4, 128, 0, s>>>(w, a.B, ma);
    const int nmain = 1 + 2 * a.K;
    const int nsubs = nmain + (ma.imr ? 2 : 0);
    // series per block: all of a binary's (its matrix is factorised once),
    // fewer where the batch alone leaves SMs idle
    int per = a.opt.spline_tile;
    if (per < 1 || per > 8) {
        const int groups = a.B >= 2 * nsm ? 1 : (2 * nsm + a.B - 1) / a.B;
        per = (nsubs + groups - 1) / groups;
    }
    k_spline<<<dim3(a.B, (nsubs + per - 1) / per), kSplineThreads, 0, s>>>(w, a.order, nsubs, nmain, per,
                                                                          a.opt.precision == 1 ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_synth(const Ws &w, const RunArgs &a, int mode, double *out, cudaStream_t s)
{
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int mixed = (mode != 2 && a.opt.precision == 1 && !a.opt.imr) ? 1 : 0;
    k_scan_chunks<<<1, kScanThreads, 0, s>>>(w, a.B, a.N, mode == 2 ? 1 : 0, mode == 0 ? a.data : nullptr,
                                             mode == 0 ? mixed : 0);
    if (mode == 1) {
        cudaError_t e = cudaMemsetAsync(out, 0, sizeof(double) * 2 * (size_t)a.B * a.N, s);
        if (e != cudaSuccess) return e;
    }
    SynthArgs sa;
    sa.B = a.B;
    sa.N = a.N;
    sa.K = a.K;
    for (int j = 0; j < kMaxModes; ++j) sa.mms[j] = a.mms[j];
    sa.dt = a.dt;
    sa.amp = a.amp;
    sa.data = a.data;
    sa.out = out;
    sa.mode = mode;
    if (mixed) k_synth_mixed<<<nsm * 8, 256, 0, s>>>(w, sa);
    else k_synth<<<nsm * 8, 256, 0, s>>>(w, sa);
    k_finalize<<<(a.B + 127) / 128, 128, 0, s>>>(w, a.B, mode == 0 ? a.lnl : nullptr, a.status_out);
    return cudaGetLastError();
}

}  // namespace eob
