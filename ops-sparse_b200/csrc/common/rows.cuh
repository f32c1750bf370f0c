// Searches in sorted offset arrays by a whole warp.
#pragma once

#include <cuda_runtime.h>

namespace b200sp {

// Largest r in [0, m) with rowPtr[r] - base <= p, given rowPtr[0] - base <= p; p is the same in every lane.  The 32
// lanes probe 32 places per round: a million rows take four dependent loads instead of twenty.
__device__ __forceinline__ int WarpRowOf(const int *__restrict__ rowPtr, int m, long long p, int lane, int base = 0)
{
    int lo = 0;
    for (int hi = m; hi - lo > 1;) {
        const int step = (hi - lo + 31) / 32;
        const long long idx = (long long)lo + (long long)(lane + 1) * step;
        const bool ok = idx < hi && (long long)__ldg(rowPtr + idx) - base <= p;
        const int n = __popc(__ballot_sync(0xffffffffu, ok));  // offsets ascend: the lanes that pass are a prefix
        lo += n * step;
        hi = hi < lo + step ? hi : lo + step;
    }
    return lo;
}

// First index in [0, count) of the ascending array v whose element is >= key (count if none), the same in every lane.
__device__ __forceinline__ int WarpLowerBound(const int *__restrict__ v, int count, long long key, int lane)
{
    int lo = 0, hi = count;  // the answer lies in [lo, hi]
    while (lo < hi) {
        const int step = (hi - lo + 31) / 32;
        const long long idx = (long long)lo + (long long)(lane + 1) * step - 1;
        const bool below = idx < hi && (long long)__ldg(v + idx) < key;
        const int n = __popc(__ballot_sync(0xffffffffu, below));
        const long long next = (long long)lo + (long long)(n + 1) * step - 1;  // the first probe that was not below
        lo += n * step;
        hi = next < hi ? (int)next : hi;
    }
    return lo;
}

// Row of every lane's entry p (32 ascending entries), given a row r0 with rowPtr[r0] - base <= every p: largest r
// with rowPtr[r] - base <= p.
__device__ __forceinline__ int RowOfLane(const int *__restrict__ rowPtr, int m, int r0, int p, int lane, int base = 0)
{
    const int last = 0x7fffffff;
    const int end = r0 + 1 + lane <= m - 1 ? __ldg(rowPtr + r0 + 1 + lane) - base : last;  // starts of the 32 rows after r0
    int n = 0;  // how many of them are <= p: they ascend
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
        const int at = __shfl_sync(0xffffffffu, end, n + step - 1);
        if (at <= p) n += step;
    }
    const int end31 = __shfl_sync(0xffffffffu, end, 31);
    if (n == 31 && end31 <= p) n = 32;
    int r = r0 + n;
    if (n == 32) {  // more than 32 rows within 32 entries: go on alone
        int hi = m - 1;
        while (r < hi) {
            const int mid = r + ((hi - r + 1) >> 1);
            if (__ldg(rowPtr + mid) - base <= p) r = mid;
            else hi = mid - 1;
        }
    }
    return r;
}

// out[i] = plus + (number of elements of the ascending array v that are < i + keyBase), for the calling CTA's 256
// values of i and i <= last.  Two warps bracket the CTA's range; the threads then search a few thousand elements.
__device__ __forceinline__ void OffsetsOfSorted(const int *__restrict__ v, int count, long long i0, long long last, int keyBase,
                                                int plus, int *__restrict__ out)
{
    __shared__ int sBound[2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < 2) {
        const long long i = warp == 0 ? i0 : (i0 + 255 < last ? i0 + 255 : last);
        const int b = WarpLowerBound(v, count, i + keyBase, lane);
        if (lane == 0) sBound[warp] = b;
    }
    __syncthreads();
    const long long i = i0 + threadIdx.x;
    if (i <= last) {
        int lo = sBound[0], hi = sBound[1];
        while (lo < hi) {
            const int mid = lo + ((hi - lo) >> 1);
            if ((long long)__ldg(v + mid) < i + keyBase) lo = mid + 1;
            else hi = mid;
        }
        out[i] = lo + plus;
    }
    __syncthreads();  // sBound may be written again
}

}  // namespace b200sp
