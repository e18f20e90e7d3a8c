// Reference-shaped synthesis and likelihood entry points of src/tdinterp.pyx:
//
//   eob_tdinterp2              TDInterp_wrap2 -> TD2 (src/interpolate.cu:441-549)
//   eob_tdinterp               TDInterp_wrap  -> TD  (src/interpolate.cu:323-438)
//   eob_all_in_one_likelihood  all_in_one_likelihood (src/interpolate.cu:553-627)
//
// The first two evaluate per-mode cubic splines (y + c1 x + c2 x^2 + c3 x^3,
// the reference's expression) on a caller time grid, rotate each mode by
// e^{-i m phi} with phi the orbital-phase spline and sum the modes; the third
// forms the frequency-domain residual d - (F+ h+ + Fx hx) e^{-2 pi i f tau}
// and sums |r|^2 / S_n per 1024-bin block of frequencies, one partial per
// (block, binary, channel) in the reference's layout.  Layouts, index
// arithmetic and argument meaning are the reference's, including TD2's sub-
// series stride old_lengths[b] inside a slot of old_length rows; knot indices
// are clamped into the binary's rows (the reference reads whatever memory an
// out-of-range index points at).  Complex
// arrays are interleaved (re, im) doubles.  All three are grid-stride
// streaming kernels: one thread per output sample (four frequency bins for the
// likelihood), coalesced over samples.
#include "eob_device.cuh"
#include "fd_fixed.cuh"

namespace {

constexpr int kMaxTdModes = 20;  // src/interpolate.cu:320 (MAX_EOB_MODES)
constexpr int kSumBins = 1024;   // frequency bins per likelihood partial (NUM_THREADS_SUM)
constexpr int kSumThreads = 256;

__device__ __forceinline__ double cubic(const double *y, const double *c1, const double *c2, const double *c3, size_t j,
                                        double x)
{
    return fma(fma(fma(c3[j], x, c2[j]), x, c1[j]), x, y[j]);
}

// sum_k (re_k + i im_k) e^{-i m_k phi} of one sample; sub-series k of a
// binary's block start at base + k * stride.  The rotations come from the integer
// phase (fasttrig.h); a mode with the m of the one before shares its.  FP64 issue
// bounds it (88 %): two modes take 24 FP64 instructions a sample, 72 with the
// library's sincos and products for the powers of x, 28 with integer sincos and
// complex products from one multiple to the next (128 binaries, two modes, 32768
// samples: 0.36, 0.18 and 0.138 ms).
__device__ __forceinline__ double2 mode_sum(const double *y, const double *c1, const double *c2, const double *c3,
                                            size_t base, size_t stride, int ind, double x, int K, const int *ms)
{
    const double phi = cubic(y, c1, c2, c3, base + 2 * (size_t)K * stride + ind, x);
    double hr = 0.0, hi = 0.0, c, s;
    auto add = [&](int k) {
        const double re = cubic(y, c1, c2, c3, base + (size_t)k * stride + ind, x);
        const double im = cubic(y, c1, c2, c3, base + (size_t)(K + k) * stride + ind, x);
        // (re + i im)(c - i s)
        hr = fma(re, c, fma(im, s, hr));
        hi = fma(im, c, fma(-re, s, hi));
    };
    // One mode: m phi rounded to a double, as the reference's sincos(m phi), which tests and
    // callers compare a single series with; several: exact multiples of the integer phase.
    if (K == 1) {
        eob::eob_sincos(ms[0] * phi, &s, &c);
        add(0);
        return make_double2(hr, hi);
    }
    const eob::PhaseTurns phase(phi);
    for (int k = 0; k < K; ++k) {
        if (k == 0 || ms[k] != ms[k - 1]) phase.multiple(ms[k], &s, &c);
        add(k);
    }
    return make_double2(hr, hi);
}

// Five blocks on an SM (48 registers, 12 bytes spilled): 0.138 ms at the size above, against
// 0.143 ms with 60 registers and four blocks.
__global__ void __launch_bounds__(256, 5) k_td2(double2 *out, const double *dataTime, const double *ts, const double *y, const double *c1,
                      const double *c2, const double *c3, int old_length, const int *old_lengths, int data_length,
                      int B, int K, const int *ms_in, const int *inds, const int *lengths, int max_length)
{
    __shared__ int ms[kMaxTdModes];
    for (int k = threadIdx.x; k < K; k += blockDim.x) ms[k] = ms_in[k];
    __syncthreads();
    for (int b = blockIdx.y; b < B; b += gridDim.y) {
        // a binary's samples stop at max_length and its knot indices stay
        // inside its slot (the reference trusts its caller for both)
        const int n = min(lengths[b], max_length);
        const int olh = min(old_lengths[b], old_length);
        const size_t base = (size_t)b * (2 * K + 1) * (size_t)old_length;
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += blockDim.x * gridDim.x) {
            const int ind = min(max(inds[(size_t)max_length * b + i], 0), old_length - 1);
            const double x = dataTime[i] - ts[(size_t)b * old_length + ind];
            out[(size_t)b * data_length + i] = mode_sum(y, c1, c2, c3, base, (size_t)olh, ind, x, K, ms);
        }
    }
}

// one binary of TDInterp: its own arrays, samples ind_start .. ind_start + n of
// the time grid, written from element data_length of its output (the
// reference's templateChannels[data_length + i])
__global__ void k_td1(double2 *out, const double *dataTime, const double *ts, const double *y, const double *c1,
                      const double *c2, const double *c3, int old_length, int data_length, int K, const int *ms_in,
                      const int *inds, int ind_start, int n)
{
    __shared__ int ms[kMaxTdModes];
    for (int k = threadIdx.x; k < K; k += blockDim.x) ms[k] = ms_in[k];
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += blockDim.x * gridDim.x) {
        const int ind = min(max(inds[i], 0), old_length - 1);
        const double x = dataTime[i + ind_start] - ts[ind];
        out[(size_t)data_length + i] = mode_sum(y, c1, c2, c3, 0, (size_t)old_length, ind, x, K, ms);
    }
}

// |d - h|^2 / S_n summed over blocks of kSumBins frequencies, per (binary,
// channel): blockIdx.x = frequency block, y = group of binaries, z = pair of
// channels.  The residual up to its square on the integer units (fd_fixed.cuh); a
// block keeps its data and 1 / S_n in registers (four bins and NCH channels
// per thread) and carries `group` binaries past them.  96 binaries x 30721 bins x 2
// channels: 0.39 ms in FP64 -> 0.13 ms.
constexpr int kSumGroup = 16;  // most binaries per block

template <int NCH>
__global__ void __launch_bounds__(kSumThreads, 2) k_fd_lnl(double2 *temp_sum, const double2 *hp, const double2 *hc,
                                                           const double2 *data, const double *psd, const double *Fplus,
                                                           const double *Fcross, const double *tshift, double df, int B,
                                                           int group, int ch0, int nch, int N)
{
    using namespace eob;
    constexpr int kBins = kSumBins / kSumThreads, kWarps = kSumThreads / 32;
    __shared__ FdDetector det[kSumGroup][NCH];
    __shared__ double sums[kSumGroup][NCH][kWarps];
    const int tid = threadIdx.x, i0 = blockIdx.x * kSumBins + tid, first = ch0 + blockIdx.z * NCH;
    FdData d[kBins][NCH];
#pragma unroll
    for (int q = 0; q < kBins; ++q)
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
            const size_t at = (size_t)(first + c) * N + min(i0 + q * kSumThreads, N - 1);
            d[q][c] = fd_data(data[at], psd[at]);
        }
    for (int b0 = blockIdx.y * group; b0 < B; b0 += gridDim.y * group) {
        const int nb = min(group, B - b0);
        __syncthreads();
        for (int t = tid; t < nb * NCH; t += kSumThreads) {
            const size_t k = (size_t)(first + t % NCH) * B + b0 + t / NCH;
            det[t / NCH][t % NCH] = fd_detector(Fplus[k], Fcross[k], df * tshift[k], kSumThreads);
        }
        __syncthreads();
        for (int g = 0; g < nb; ++g) {
            const size_t row = (size_t)(b0 + g) * N;
            i64 s[NCH], co[NCH];
            double acc[NCH];
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                sincos_fix(det[g][c].step.at(i0), &s[c], &co[c]);
                acc[c] = 0.0;
            }
#pragma unroll
            for (int q = 0; q < kBins; ++q) {
                const int i = i0 + q * kSumThreads;
                if (i < N) {
                    const double2 p = hp[row + i], x = hc[row + i];
                    const FdStrain h = fd_strain(p, x);
#pragma unroll
                    for (int c = 0; c < NCH; ++c) {
                        const FdDetector &t = det[g][c];
                        if (q > 0) rotate(&s[c], &co[c], t.rs, t.rc);
                        double power;
                        if (fd_slow(h, t, d[q][c])) {
                            const size_t k = (size_t)(first + c) * B + b0 + g;
                            power = fd_power_slow(p, x, Fplus[k], Fcross[k], data[(size_t)(first + c) * N + i],
                                                  df * i * tshift[k], t.slow(), s[c], co[c]);
                        } else {
                            power = fd_power(h, t, s[c], co[c], d[q][c]);
                        }
                        acc[c] = fma(power, d[q][c].w, acc[c]);
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                double t = acc[c];
                for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
                if ((tid & 31) == 0) sums[g][c][tid >> 5] = t;
            }
        }
        __syncthreads();
        for (int t = tid; t < nb * NCH; t += kSumThreads) {
            double v = 0.0;
            for (int k = 0; k < kWarps; ++k) v += sums[t / NCH][t % NCH][k];
            temp_sum[((size_t)blockIdx.x * B + b0 + t / NCH) * nch + first + t % NCH] = make_double2(v, 0.0);
        }
    }
}

int grid_for(long long n, int bs)
{
    long long g = (n + bs - 1) / bs;
    return (int)(g < 1 ? 1 : (g > 65535 ? 65535 : g));
}

int ret(cudaError_t e) { return e == cudaSuccess ? EOB_OK : EOB_E_CUDA; }

}  // namespace

extern "C" {

int eob_tdinterp2(double *templateChannels, const double *dataTime, const double *ts, const double *propArrays,
                  const double *c1, const double *c2, const double *c3, int old_length, const int *old_lengths,
                  int data_length, int numBinAll, int numModes, const int *ls, const int *ms, const int *inds,
                  const int *lengths, int max_length, cudaStream_t stream)
{
    (void)ls;  // the reference reads l but only m enters the rotation
    if (numBinAll < 0 || numModes < 1 || numModes > kMaxTdModes || old_length < 1 || max_length < 0 ||
        data_length < max_length)
        return EOB_E_ARG;
    if (numBinAll == 0 || max_length == 0) return EOB_OK;
    if (!templateChannels || !dataTime || !ts || !propArrays || !c1 || !c2 || !c3 || !old_lengths || !ms || !inds ||
        !lengths)
        return EOB_E_ARG;
    const int bs = 256;
    dim3 grid(grid_for(max_length, bs), numBinAll < 65535 ? numBinAll : 65535);
    k_td2<<<grid, bs, 0, stream>>>((double2 *)templateChannels, dataTime, ts, propArrays, c1, c2, c3, old_length,
                                   old_lengths, data_length, numBinAll, numModes, ms, inds, lengths, max_length);
    return ret(cudaGetLastError());
}

int eob_tdinterp(const long long *templateChannels_ptrs, const double *dataTime, const long long *tsAll,
                 const long long *propArraysAll, const long long *c1All, const long long *c2All,
                 const long long *c3All, const int *old_lengths, int data_length, int numBinAll, int numModes,
                 const int *ls, const int *ms, const long long *inds_ptrs, const int *inds_start,
                 const int *ind_lengths, cudaStream_t stream)
{
    (void)ls;
    if (numBinAll < 0 || numModes < 1 || numModes > kMaxTdModes || data_length < 0) return EOB_E_ARG;
    if (numBinAll == 0) return EOB_OK;
    if (!templateChannels_ptrs || !dataTime || !tsAll || !propArraysAll || !c1All || !c2All || !c3All ||
        !old_lengths || !ms || !inds_ptrs || !inds_start || !ind_lengths)
        return EOB_E_ARG;
    // per-binary metadata are host arrays, as in the reference's host loop
    // (src/interpolate.cu:401-431); one launch per binary on the caller's stream
    const int bs = 256;
    for (int b = 0; b < numBinAll; ++b) {
        const int n = ind_lengths[b];
        if (n < 0 || old_lengths[b] < 1) return EOB_E_ARG;
        if (n == 0) continue;
        k_td1<<<grid_for(n, bs), bs, 0, stream>>>(
            (double2 *)templateChannels_ptrs[b], dataTime, (const double *)tsAll[b], (const double *)propArraysAll[b],
            (const double *)c1All[b], (const double *)c2All[b], (const double *)c3All[b], old_lengths[b], data_length,
            numModes, ms, (const int *)inds_ptrs[b], inds_start[b], n);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return EOB_E_CUDA;
    }
    return EOB_OK;
}

int eob_all_in_one_likelihood(double *temp_sum, const double *hp_fd, const double *hc_fd, const double *data,
                              const double *psd, const double *Fplus, const double *Fcross, const double *time_shift,
                              double df, int num_bin_all, int nchannels, int data_length, cudaStream_t stream)
{
    if (num_bin_all < 0 || nchannels < 0 || data_length < 0) return EOB_E_ARG;
    if (num_bin_all == 0 || nchannels == 0 || data_length == 0) return EOB_OK;
    if (!temp_sum || !hp_fd || !hc_fd || !data || !psd || !Fplus || !Fcross || !time_shift) return EOB_E_ARG;
    const int nblocks = (data_length + kSumBins - 1) / kSumBins;
    // binaries per block: enough blocks for four per SM, then as many binaries
    // as share one conversion of the data
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const long long items = (long long)num_bin_all * nblocks * ((nchannels + 1) / 2);
    long long group = items / (4LL * (nsm > 0 ? nsm : 1));
    group = group < 1 ? 1 : (group > kSumGroup ? kSumGroup : group);
    const long long groups = (num_bin_all + group - 1) / group;
    const int pairs = nchannels / 2;
    for (int z = 0; z < pairs; z += 65535) {
        const dim3 grid(nblocks, (unsigned)(groups < 65535 ? groups : 65535), pairs - z < 65535 ? pairs - z : 65535);
        k_fd_lnl<2><<<grid, kSumThreads, 0, stream>>>((double2 *)temp_sum, (const double2 *)hp_fd,
                                                      (const double2 *)hc_fd, (const double2 *)data, psd, Fplus, Fcross,
                                                      time_shift, df, num_bin_all, (int)group, 2 * z, nchannels,
                                                      data_length);
        if (cudaGetLastError() != cudaSuccess) return EOB_E_CUDA;
    }
    if (nchannels & 1) {
        const dim3 grid(nblocks, (unsigned)(groups < 65535 ? groups : 65535), 1);
        k_fd_lnl<1><<<grid, kSumThreads, 0, stream>>>((double2 *)temp_sum, (const double2 *)hp_fd,
                                                      (const double2 *)hc_fd, (const double2 *)data, psd, Fplus, Fcross,
                                                      time_shift, df, num_bin_all, (int)group, nchannels - 1, nchannels,
                                                      data_length);
    }
    return ret(cudaGetLastError());
}

}  // extern "C"
