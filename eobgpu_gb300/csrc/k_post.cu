// After the integrator: packing, multipoles on the trajectory and batched
// not-a-knot splines.
//
//  k_sample_counts  one thread per binary: waveform sample counts.
//  k_scan_rows one block: exclusive scan of the row counts (packed ragged layout).
//  k_modes     one thread per packed trajectory row: h_lm e^{i m phi} for the
//              requested modes (get_hlms, eob/seobnrv4phm.py:2138-2221, and
//              the de-rotation of compute_full_waveform, :2331).
//  k_spline    one block per binary (and group of series): not-a-knot cubic
//              splines with the reference's tridiagonal set-up
//              (src/interpolate.cu:10-267), the matrix factorised once per
//              binary and solved by scans (spline_block.cuh).
//
// The synthesis and likelihood pass that follows is k_synth.cu.
#include "eob_device.cuh"
#include "packing.cuh"
#include "spline_block.cuh"

namespace eob {

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

// Uniform-grid sample counts per binary.  A kernel of its own: three
// divisions are 50 FP64 issue slots for each warp of binaries, which the scan's
// one SM took 64 us for at 4096 binaries (8 us here and 7 us for the scan).
__global__ void __launch_bounds__(128) k_sample_counts(Ws w, int B, double dt)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= B) return;
    const int L = w.nsteps[b];
    const int st = w.status[b];
    int np = 0;
    if (L >= 3 && !(st & (EOB_ST_NAN | EOB_ST_TRIES | EOB_ST_SHORT))) {
        np = binary_npts(w.traj + (size_t)b * w.L.Lc * kTrajStride, L, w.bins[b].Mt, dt);
        if (np < 1) np = 0;
    } else {
        w.status[b] = st | EOB_ST_SHORT;
    }
    w.npts[b] = np;
}

// packed row offsets, and the splines' work order, longest binaries first in steps
// of 64 rows (to chunk_off, which the synthesis fills later).  The caller's `order` is the
// integrator's alone and need not name every binary; in batch order the long splines
// of 1024 ragged binaries end 22 us later.
constexpr int kLengthSteps = 64;

__global__ void __launch_bounds__(kScanThreads) k_scan_rows(Ws w, int B)
{
    __shared__ long long sm[34];
    __shared__ int place[kLengthSteps];
    const int tid = threadIdx.x;
    const int per = (B + kScanThreads - 1) / kScanThreads;
    const int b0 = tid * per;
    const int b1 = min(B, b0 + per);
    long long rows = 0;
    for (int b = b0; b < b1; ++b) rows += (w.npts[b] > 0) ? w.nsteps[b] : 0;
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
    if (tid < kLengthSteps) place[tid] = 0;
    __syncthreads();
    auto step = [&](int b) { return kLengthSteps - 1 - max(0, min(w.nsteps[b] / 64, kLengthSteps - 1)); };
    for (int b = b0; b < b1; ++b) atomicAdd(&place[step(b)], 1);
    __syncthreads();
    if (tid == 0) {
        int at = 0;
        for (int q = 0; q < kLengthSteps; ++q) {
            const int n = place[q];
            place[q] = at;
            at += n;
        }
    }
    __syncthreads();
    int *order = reinterpret_cast<int *>(w.chunk_off);
    for (int b = b0; b < b1; ++b) order[atomicAdd(&place[step(b)], 1)] = b;
}

// rows closer than this to a neighbour [M] keep the log-Gamma sums (mode_eval.h): the
// fine pass steps by 0.05 and halves; the main pass's steps are above 0.2 but at
// its end
constexpr double kCloseRows = 0.2;

struct ModeArgs {
    int K;
    int ells[kMaxModes], mms[kMaxModes];
    ModeConst mc[kMaxModes];
    int imr;  // also r and p_r as series for the merger-ringdown attachment
};

// Rows closer than kCloseRows to a neighbour are listed (in the spline
// scratch, which is free until the splines) for k_modes_close: the two
// evaluations in one kernel cost the others their registers and half the
// instruction cache.  FP64 issue bounds both: five modes and the Hamiltonian
// take 500 FP64 instructions a row in the closed form, 2550 by the sums (4096
// binaries, 2.1 M rows, 4 in 10 listed: 9.32 ms with the sums on every row -> 1.13 + 4.39 ms;
// 1024 ragged binaries, (2,2) alone: 0.77 -> 0.23 + 0.34 ms).
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
            // set-up builds every table with use_hm = 1
            const cdbl hl = mode_term<true>(w.fac[b], l, m, ma.mc[j], mr, rec.pre_re[li], rec.pre_im[li], rec.nu, 0.0,
                                            true);
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
                                           e.Hreal, vPhi, ma.mc[j].y0, lfact[l], 0.0, true);
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
            const float4 v = make_float4((float)f.y[i], (float)c1, (float)c2, (float)c3);
            float *o = w.f32 + 4 * ((size_t)(s - 1) * Rc + base + i);
            if (w.f32_vec()) {
                *reinterpret_cast<float4 *>(o) = v;
            } else {
                o[0] = v.x;
                o[1] = v.y;
                o[2] = v.z;
                o[3] = v.w;
            }
        }
    }
    __device__ void put_last(int b, int s, int i, const SplineSeries &f, double, double, double) const
    {
        put(b, s, i, f, 0.0, 0.0, 0.0);
    }
};

constexpr int kSplineThreads = 64, kSplineChunk = 9, kSplineShort = kSplineThreads * kSplineChunk;
constexpr int kSplineLongThreads = 256;

// One block per binary and group of `per` series, long binaries first.  NT = 64 threads
// of up to 9 rows: 576 rows a tile, which most
// trajectories fit; 128 threads of 5 rows would spend a quarter more FP64 issue
// slots on the scans, and chunks of 13 rows hold their factors in 250 registers (four
// blocks on an SM; six with the 168 of a bound of five, which spills 100 bytes).
// Longer ones go to 256 threads (2304 rows a tile) in a launch of their own: on 64
// threads the longest of a ragged batch, four tiles one after the other, ended the
// launch late; 128 threads, or chunks of 5 rows, took 0.03 to 0.06 ms more.
// 1024 ragged binaries, 3 series: 0.81 ms with a warp per series, 0.39 on 64 threads of
// 13 rows for all, 0.26 so; 4096 binaries, 11 series, 520 rows: 4.67, 1.19
// and 1.08 + 0.03 ms (79 % of the FP64 issue slots).
template <int NT>
__global__ void __launch_bounds__(NT, NT == 64 ? 5 : 1) k_spline(Ws w, int nsubs, int nmain, int per, int mixed)
{
    using Block = SplineBlock<1, NT, kSplineChunk>;
    extern __shared__ __align__(16) char smem[];
    typename Block::Smem &sm = *reinterpret_cast<typename Block::Smem *>(smem);
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) w.queue[6] = (unsigned long long)mixed;
    const int b = reinterpret_cast<const int *>(w.chunk_off)[blockIdx.x];  // k_scan_rows
    const int n = w.npts[b] > 0 ? w.nsteps[b] : 0;
    if ((n > kSplineShort) != (NT > kSplineThreads)) return;
    const PackedSplines acc{w, n, nmain, (size_t)w.row_off[b], (size_t)w.L.Bc * (size_t)w.L.Lc, mixed != 0};
    const int s0 = blockIdx.y * per;
    Block::run(acc, sm, s0, min(nsubs, s0 + per));
}

cudaError_t launch_prepare_post(const Ws &w, const RunArgs &a, cudaStream_t s)
{
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    k_sample_counts<<<(a.B + 127) / 128, 128, 0, s>>>(w, a.B, a.dt);
    k_scan_rows<<<1, kScanThreads, 0, s>>>(w, a.B);
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
    const int mixed = a.opt.precision == 1 ? 1 : 0;
    const dim3 grid(a.B, (nsubs + per - 1) / per);
    using Short = SplineBlock<1, kSplineThreads, kSplineChunk>::Smem;
    using Long = SplineBlock<1, kSplineLongThreads, kSplineChunk>::Smem;
    if (w.L.Lc > kSplineShort) {
        const cudaError_t e = cudaFuncSetAttribute(k_spline<kSplineLongThreads>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Long));
        if (e != cudaSuccess) return e;
        k_spline<kSplineLongThreads><<<grid, kSplineLongThreads, sizeof(Long), s>>>(w, nsubs, nmain, per, mixed);
    }
    k_spline<kSplineThreads><<<grid, kSplineThreads, sizeof(Short), s>>>(w, nsubs, nmain, per, mixed);
    return cudaGetLastError();
}

}  // namespace eob
