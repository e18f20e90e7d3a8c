// The packed ragged layout of the passes after the integrator: offsets per
// binary by exclusive scans, and their search.
#pragma once

namespace eob {

constexpr int kScanThreads = 1024;

// block-wide exclusive scan: the exclusive prefix of v over the NT threads, and
// the total.  sm: 34 entries of shared memory.
template <int NT>
__device__ long long block_exclusive_scan(long long v, long long *sm, long long *total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    long long s = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const long long u = __shfl_up_sync(0xffffffffu, s, off);
        if (lane >= off) s += u;
    }
    if (lane == 31) sm[wid] = s;
    __syncthreads();
    if (wid == 0) {
        long long t = lane < NT / 32 ? sm[lane] : 0;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const long long u = __shfl_up_sync(0xffffffffu, t, off);
            if (lane >= off) t += u;
        }
        sm[lane + 1] = t;
        if (lane == 0) sm[0] = 0;
    }
    __syncthreads();
    *total = sm[NT / 32];
    return s - v + sm[wid];
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

// blocks that fill the device once: a kernel whose blocks take equal runs of the
// work ends in a partial wave on more of them (1216 blocks on 152 SMs x 5: two waves,
// the second 60 % full; the likelihood passes gain 4 and 12 %).  Kernels with
// uneven items (strain, multipoles) run faster with spare blocks.
template <class Kernel>
inline int resident_blocks(Kernel kern, int threads)
{
    int dev = 0, nsm = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, 0);
    return nsm * (per > 0 ? per : 1);
}

}  // namespace eob
