// Stable in-place sort of the columns of every CSR row, with the permutation P carried along, for aclsparseXcsrsort.
//
//   rows of up to 32 entries     a warp takes as many whole consecutive rows as fit into 32 entries; every lane counts
//                                the entries of its row that belong before its own (a shuffle up and one down per
//                                distance), which is its place: no network, and a thousand short rows are not a
//                                thousand warps' work;
//   up to 256                    a warp per row, 2, 4 or 8 keys per lane in registers, bitonic network over shuffles and
//                                register pairs; column and place share a 32-bit key below 2^24 columns;
//   up to kLargeMax = 16384      a CTA per row, in shared memory: the row's column range is cut into half as many buckets as
//                                it has entries, entries are dropped into their buckets and every entry counts those of
//                                its bucket that belong before it.  One pass instead of three or four radix passes; where
//                                the columns cluster so that buckets get long, radix passes after all;
//   longer                       radix passes by one CTA between two arrays in global memory.
// The first kernel sorts the short rows and lists the others by size class; the later kernels, one per class so that
// each has little code, take their rows from the lists, so nothing is read back.
// Measured on 31.2 M entries in 1 M power-law rows: a warp for every short row and global-memory passes from 2048
// entries on took 523 + 709 us; short rows 66, warp rows 43 and the three CTA kernels 112 to 117 us each now.
#pragma once

#include <atomic>
#include <cstdint>

#include <cuda_runtime.h>

#include "b200sp_kernels.h"
#include "common/chained.cuh"
#include "convert/radix.cuh"

namespace b200sp_rowsort {

constexpr int kWarpMax = 256;
constexpr int kMidMax = 2048, kBigMax = 8192, kLargeMax = 16384;
// The list: counters and cursors, then two arrays of m rows.  The first is filled from the front by rows of 33 to 256
// entries and from the back by those of up to kMidMax, the second from the front by those of up to kBigMax and from the
// back by longer ones (beyond kLargeMax as their complement).
enum { kCountWarp = 0, kCountMid = 1, kCountBig = 2, kCountLong = 3, kCountHuge = 4, kTake = 8 };  // a cursor per class
constexpr int kListHead = 16;

// Bitonic sort of 32 * E keys held by one warp, element i = r * 32 + lane in v[r]; ascending in i.
template <int E, typename Key>
__device__ __forceinline__ void WarpSort(Key (&v)[E], int lane)
{
#pragma unroll
    for (int k = 2; k <= 32 * E; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {  // partner in the same lane: registers r and r | (j / 32)
                const int jr = j >> 5;
#pragma unroll
                for (int r = 0; r < E; ++r) {
                    if ((r & jr) != 0) continue;
                    const bool up = ((r << 5) & k) == 0;  // k >= 64: decided by the register index alone
                    const Key lo = v[r] < v[r | jr] ? v[r] : v[r | jr], hi = v[r] < v[r | jr] ? v[r | jr] : v[r];
                    v[r] = up ? lo : hi;
                    v[r | jr] = up ? hi : lo;
                }
            } else {  // partner in lane ^ j, same register
#pragma unroll
                for (int r = 0; r < E; ++r) {
                    const Key other = __shfl_xor_sync(0xffffffffu, v[r], j);
                    const bool up = (((r << 5) | lane) & k) == 0;
                    const bool lower = (lane & j) == 0;
                    const bool takeMin = lower == up;
                    v[r] = takeMin ? (v[r] < other ? v[r] : other) : (v[r] > other ? v[r] : other);
                }
            }
        }
    }
}

// One row of up to 32 * E entries.  Key: column, then place in the row (unique, so any sort is the stable one).
template <int E, typename Key>
__device__ __forceinline__ void WarpRow(int *__restrict__ col, int *__restrict__ P, int len, int lane)
{
    constexpr int kShift = sizeof(Key) == 8 ? 32 : 8;
    Key v[E];
#pragma unroll
    for (int r = 0; r < E; ++r) {
        const int i = r * 32 + lane;
        v[r] = i < len ? ((Key)(unsigned)col[i] << kShift) | (unsigned)i : ~(Key)0;  // ~0 sorts after every real key
    }
    WarpSort<E, Key>(v, lane);
    int p[E];
#pragma unroll
    for (int r = 0; r < E; ++r) p[r] = r * 32 + lane < len ? P[(unsigned)v[r] & (kWarpMax - 1)] : 0;
    __syncwarp();  // every lane has fetched before any lane writes: the sort is in place
#pragma unroll
    for (int r = 0; r < E; ++r) {
        const int i = r * 32 + lane;
        if (i < len) {
            col[i] = (int)(v[r] >> kShift);
            P[i] = p[r];
        }
    }
}

// A warp per listed row of 33 to 256 entries; Key is 32 bits wide when every column is below 2^24 - 1.
template <typename Key>
static __global__ void __launch_bounds__(128) RowSortWarpKernel(const int *__restrict__ rowPtr, int base, int *colInd, int *P,
                                                                const int *__restrict__ list)
{
    b200sp::WaitForPrevious();
    const int lane = threadIdx.x & 31;
    const int count = list[kCountWarp];
    for (int i = blockIdx.x * 4 + (threadIdx.x >> 5); i < count; i += gridDim.x * 4) {
        const int row = __ldg(list + kListHead + i);
        const int s = __ldg(rowPtr + row) - base, n = __ldg(rowPtr + row + 1) - base - s;
        if (n <= 64) WarpRow<2, Key>(colInd + s, P + s, n, lane);
        else if (n <= 128) WarpRow<4, Key>(colInd + s, P + s, n, lane);
        else WarpRow<8, Key>(colInd + s, P + s, n, lane);
    }
}

// A warp per `rowsPerWarp` (<= 32) consecutive rows; lane r holds the bounds of row r.
static __global__ void __launch_bounds__(256) RowSortShortKernel(const int *__restrict__ rowPtr, int base, int m, int rowsPerWarp,
                                                                 int *colInd, int *P, int *__restrict__ list)
{
    b200sp::WaitForPrevious();
    const int lane = threadIdx.x & 31;
    const long long row0 = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * rowsPerWarp;
    if (row0 >= m) return;
    const int rows = m - row0 < rowsPerWarp ? (int)(m - row0) : rowsPerWarp;
    const int start = lane < rows ? rowPtr[row0 + lane] - base : 0x7fffffff;
    const int end = lane < rows ? rowPtr[row0 + lane + 1] - base : 0x7fffffff;
    const int len = end - start;
    const unsigned shortRows = __ballot_sync(0xffffffffu, lane < rows && len <= 32);
    if (lane < rows && len > 32) {
        const int r = (int)row0 + lane;
        int *first = list + kListHead, *second = first + m;
        if (len <= kWarpMax) {
            first[atomicAdd(list + kCountWarp, 1)] = r;
        } else if (len <= kMidMax) {
            first[m - 1 - atomicAdd(list + kCountMid, 1)] = r;
        } else if (len <= kBigMax) {
            second[atomicAdd(list + kCountBig, 1)] = r;
        } else {
            second[m - 1 - atomicAdd(list + kCountLong, 1)] = len <= kLargeMax ? r : ~r;
            if (len > kLargeMax) atomicAdd(list + kCountHuge, 1);
        }
    }
    int r = 0;  // next row of the warp
    while (r < rows) {
        if (!((shortRows >> r) & 1u)) {
            ++r;
            continue;
        }
        // Rows r .. last: short ones that end within 32 entries of where row r starts.
        const int s = __shfl_sync(0xffffffffu, start, r);
        const unsigned fits = __ballot_sync(0xffffffffu, lane >= r && ((shortRows >> lane) & 1u) && end - s <= 32);
        const unsigned run = fits >> r;                       // bit 0: row r itself
        const int count = run == 0xffffffffu ? 32 : __ffs(~run) - 1;
        const int last = r + count - 1;
        const int total = __shfl_sync(0xffffffffu, end, last) - s;
        if (total > 0) {
            // The row of entry s + lane: the last of the rows r .. last that starts at or before it.
            int at = r;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const int cand = at + step;
                const int cs = __shfl_sync(0xffffffffu, start, cand & 31);
                if (cand <= last && cs <= s + lane) at = cand;
            }
            const int rs = __shfl_sync(0xffffffffu, start, at) - s, re = __shfl_sync(0xffffffffu, end, at) - s;
            const bool in = lane < total;
            const int c = in ? colInd[s + lane] : 0, p = in ? P[s + lane] : 0;
            const int most = __reduce_max_sync(0xffffffffu, in ? re - rs : 0);
            int place = rs;
            for (int d = 1; d < most; ++d) {
                const int below = __shfl_up_sync(0xffffffffu, c, d), above = __shfl_down_sync(0xffffffffu, c, d);
                if (lane - d >= rs && (unsigned)below <= (unsigned)c) ++place;  // an equal column earlier in the row goes first
                if (lane + d < re && (unsigned)above < (unsigned)c) ++place;
            }
            __syncwarp();
            if (in) {
                colInd[s + place] = c;
                P[s + place] = p;
            }
            __syncwarp();
        }
        r = last + 1;
    }
}

constexpr int kDigitBits = 8;
constexpr int kBins = 1 << kDigitBits;

// The lanes whose digit equals this lane's, by one ballot per bit; lanes with `in` false only meet each other.
__device__ __forceinline__ unsigned PeersOf(int digit, int bits, bool in)
{
    const unsigned live = __ballot_sync(0xffffffffu, in);
    unsigned peers = in ? live : ~live;
    for (int b = 0; b < bits; ++b) {  // the same in every lane
        const bool bit = (digit >> b) & 1;
        const unsigned with = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? with : ~with;
    }
    return peers;
}

// A CTA's shared memory: column, value of P and place in the row of every entry, a second array of places for the
// radix passes, and 16-bit counters (of the buckets, or per warp and digit).
template <int kThreads, int kMax> struct CtaShape {
    static constexpr int kWarps = kThreads / 32;
    static constexpr int kMaxBuckets = kMax / 2;
    static constexpr int kCounters = kMaxBuckets > kWarps * kBins ? kMaxBuckets : kWarps * kBins;
    static constexpr int kSmem = kMax * 12 + kCounters * 2;
};

// The radix passes: columns and places between the two pairs of arrays, then P through the columns' second array.
template <int kThreads, int kMax>
__device__ void CtaRowRadix(int *__restrict__ col, int *__restrict__ P, int len, unsigned span, unsigned lowest, unsigned char *sRaw,
                            int *sWarp)
{
    using Shape = CtaShape<kThreads, kMax>;
    unsigned *c0 = reinterpret_cast<unsigned *>(sRaw), *c1 = c0 + kMax;
    uint16_t *i0 = reinterpret_cast<uint16_t *>(c1 + kMax), *i1 = i0 + kMax;
    uint16_t *sCount = i1 + kMax;  // [warp][digit]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < len; i += kThreads) {
        c0[i] = (unsigned)col[i] - lowest;
        i0[i] = (uint16_t)i;
    }
    const int bits = span <= 1 ? 1 : 32 - __clz(span - 1);
    const int passes = (bits + kDigitBits - 1) / kDigitBits, digit = (bits + passes - 1) / passes, bins = 1 << digit;
    const int steps = (len + kThreads - 1) / kThreads;
    const int w0 = warp * 32 * steps + lane;  // a warp's entries are consecutive
    uint16_t *mine = sCount + warp * kBins;
    for (int p = 0; p < passes; ++p) {
        const int shift = p * digit;
        for (int i = lane; i < bins; i += 32) mine[i] = 0;
        __syncthreads();
        for (int u = 0; u < steps; ++u) {
            const bool in = w0 + u * 32 < len;
            const int d = in ? (int)(c0[w0 + u * 32] >> shift) & (bins - 1) : 0;
            const unsigned peers = PeersOf(d, digit, in);
            if (in && (peers & ((1u << lane) - 1u)) == 0) mine[d] = (uint16_t)(mine[d] + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        int tot = 0;  // counts -> first place of (digit, warp)
        if (tid < bins)
            for (int w = 0; w < Shape::kWarps; ++w) {
                const int n = sCount[w * kBins + tid];
                sCount[w * kBins + tid] = (uint16_t)tot;
                tot += n;
            }
        const int start = b200sp_radix::CtaInclusiveScan<kThreads>(tot, sWarp) - tot;
        if (tid < bins)
            for (int w = 0; w < Shape::kWarps; ++w) sCount[w * kBins + tid] = (uint16_t)(sCount[w * kBins + tid] + start);
        __syncthreads();
        for (int u = 0; u < steps; ++u) {
            const bool in = w0 + u * 32 < len;
            const unsigned c = in ? c0[w0 + u * 32] : 0u;
            const int d = (int)(c >> shift) & (bins - 1);
            const unsigned peers = PeersOf(d, digit, in);
            const int rank = __popc(peers & ((1u << lane) - 1u));
            const int to = in ? mine[d] + rank : 0;
            __syncwarp();
            if (in) {
                c1[to] = c;
                i1[to] = i0[w0 + u * 32];
                if (rank == 0) mine[d] = (uint16_t)(mine[d] + __popc(peers));
            }
            __syncwarp();
        }
        __syncthreads();
        unsigned *tc = c0; c0 = c1; c1 = tc;
        uint16_t *ti = i0; i0 = i1; i1 = ti;
    }
    for (int i = tid; i < len; i += kThreads) c1[i] = (unsigned)P[i0[i]];
    __syncthreads();  // every fetch is done before any entry is written
    for (int i = tid; i < len; i += kThreads) {
        col[i] = (int)(c0[i] + lowest);
        P[i] = (int)c1[i];
    }
}

template <int kThreads, int kMax>
__device__ __forceinline__ void CtaRow(int *__restrict__ col, int *__restrict__ P, int len, unsigned char *sRaw, int *sWarp,
                                       unsigned *sRange, unsigned *sCost)
{
    using Shape = CtaShape<kThreads, kMax>;
    unsigned *sCol = reinterpret_cast<unsigned *>(sRaw);
    int *sP = reinterpret_cast<int *>(sCol + kMax);
    uint16_t *sIdx = reinterpret_cast<uint16_t *>(sP + kMax);
    uint16_t *sCount = sIdx + 2 * kMax;  // [bucket]
    uint32_t *sPair = reinterpret_cast<uint32_t *>(sCount);
    const int tid = threadIdx.x, lane = tid & 31;

    // The thread's entries tid, tid + kThreads, ... stay in registers: they are wanted three times, and everything there is to
    // fetch of a row is asked for at once (30.5 M power-law entries: the three classes 343 -> 309 us).
    constexpr int kEach = kMax / kThreads;
    unsigned c[kEach];
    int p[kEach];
    unsigned lowest = 0xffffffffu, highest = 0;
#pragma unroll
    for (int u = 0; u < kEach; ++u) {
        const int i = tid + u * kThreads;
        c[u] = i < len ? (unsigned)col[i] : 0u;
        p[u] = i < len ? P[i] : 0;
    }
#pragma unroll
    for (int u = 0; u < kEach; ++u) {
        if (tid + u * kThreads < len) {
            lowest = c[u] < lowest ? c[u] : lowest;
            highest = c[u] > highest ? c[u] : highest;
        }
    }
    if (tid == 0) {
        sRange[0] = 0xffffffffu;
        sRange[1] = 0;
        *sCost = 0;
    }
    int buckets = 64;  // a power of two, about half as many as entries
    while (buckets < Shape::kMaxBuckets && 2 * buckets < len) buckets *= 2;
    for (int i = tid; i < buckets / 2; i += kThreads) sPair[i] = 0;
    __syncthreads();
    lowest = __reduce_min_sync(0xffffffffu, lowest);
    highest = __reduce_max_sync(0xffffffffu, highest);
    if (lane == 0) {
        atomicMin(sRange, lowest);
        atomicMax(sRange + 1, highest);
    }
    __syncthreads();
    lowest = sRange[0];
    const unsigned span = sRange[1] - lowest + 1;  // column indices are below 2^31: no overflow
    // Bucket of a column: monotone, below `buckets`, and about evenly wide.
    const unsigned scale = span > (unsigned)buckets ? (unsigned)(((unsigned long long)buckets << 32) / span) : 0u;
    auto bucketOf = [&](unsigned c) {
        const unsigned b = scale ? __umulhi(c - lowest, scale) : c - lowest;
        return b < (unsigned)buckets ? b : (unsigned)buckets - 1;  // also for columns no matrix has
    };

#pragma unroll
    for (int u = 0; u < kEach; ++u) {
        if (tid + u * kThreads < len) {
            const unsigned b = bucketOf(c[u]);
            atomicAdd(sPair + (b >> 1), 1u << (16 * (b & 1)));
        }
    }
    __syncthreads();
    // Counts -> first place of every bucket; the cost of counting within buckets on the way.
    const int per = (buckets / 2 + kThreads - 1) / kThreads;  // pairs of a thread, consecutive
    int sum = 0;
    unsigned cost = 0;  // at most the square of the row length
    for (int k = 0; k < per; ++k) {
        const int i = tid * per + k;
        if (i < buckets / 2) {
            const unsigned lo = sPair[i] & 0xffffu, hi = sPair[i] >> 16;
            sum += (int)(lo + hi);
            cost += lo * lo + hi * hi;
        }
    }
    cost = __reduce_add_sync(0xffffffffu, cost);
    if (lane == 0) atomicAdd(sCost, cost);
    int run = b200sp_radix::CtaInclusiveScan<kThreads>(sum, sWarp) - sum;
    // 48 entries looked at per entry cost about as much as the radix passes (an even spread looks at three)
    if (*sCost > 48u * (unsigned)len) {
        __syncthreads();
        CtaRowRadix<kThreads, kMax>(col, P, len, span, lowest, sRaw, sWarp);
        return;
    }
    for (int k = 0; k < per; ++k) {
        const int i = tid * per + k;
        if (i < buckets / 2) {
            const unsigned lo = sPair[i] & 0xffffu, hi = sPair[i] >> 16;
            sPair[i] = (unsigned)run | ((unsigned)run + lo) << 16;
            run += (int)(lo + hi);
        }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kEach; ++u) {
        const int i = tid + u * kThreads;
        if (i < len) {
            const unsigned b = bucketOf(c[u]);
            const unsigned to = (atomicAdd(sPair + (b >> 1), 1u << (16 * (b & 1))) >> (16 * (b & 1))) & 0xffffu;
            sCol[to] = c[u];
            sP[to] = p[u];
            sIdx[to] = (uint16_t)i;
        }
    }
    __syncthreads();  // sCount[b] is the end of bucket b now
    for (int i = tid; i < len; i += kThreads) {
        const unsigned ci = sCol[i], idx = sIdx[i], b = bucketOf(ci);
        const int lo = b > 0 ? sCount[b - 1] : 0, hi = sCount[b];
        int place = lo;
        for (int j = lo; j < hi; ++j) {
            const unsigned cj = sCol[j];
            if (cj < ci || (cj == ci && sIdx[j] < idx)) ++place;
        }
        col[place] = (int)ci;
        P[place] = sP[i];
    }
}

template <int kThreads, int kMax, int kClass>
static __global__ void __launch_bounds__(kThreads, 2048 / kThreads > 227 * 1024 / CtaShape<kThreads, kMax>::kSmem
                                                       ? 227 * 1024 / CtaShape<kThreads, kMax>::kSmem
                                                       : 2048 / kThreads)
    RowSortCtaKernel(const int *__restrict__ rowPtr, int base, int m, int *colInd, int *P, int *list)
{
    extern __shared__ __align__(16) unsigned char sRaw[];
    __shared__ int sWarp[kThreads / 32];
    __shared__ unsigned sRange[2];
    __shared__ unsigned sCost;
    __shared__ int sTake;
    b200sp::WaitForPrevious();
    const int count = list[kClass];
    const int *rows = list + kListHead + (kClass == kCountMid ? 0 : m);
    int ahead = 0;  // of thread 0: the row taken next, asked for while the one before is sorted
    if (threadIdx.x == 0 && count > 0) ahead = atomicAdd(list + kTake + kClass, 1);
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) sTake = ahead;
        __syncthreads();
        const int li = sTake;
        if (li >= count) break;
        if (threadIdx.x == 0) ahead = atomicAdd(list + kTake + kClass, 1);
        const int row = kClass == kCountBig ? rows[li] : rows[m - 1 - li];
        if (row < 0) continue;  // longer than this kernel takes
        const int s = rowPtr[row] - base, len = rowPtr[row + 1] - base - s;
        CtaRow<kThreads, kMax>(colInd + s, P + s, len, sRaw, sWarp, sRange, &sCost);
    }
}

// Rows of more than kLargeMax entries: (column, place) keys between two arrays in global memory, by one CTA.
constexpr int kHugeThreads = 256;
constexpr int kHugeWarps = kHugeThreads / 32;
static __global__ void __launch_bounds__(kHugeThreads) RowSortHugeKernel(const int *__restrict__ rowPtr, int base, int m,
                                                                         int *colInd, int *P, unsigned long long *keysA,
                                                                         unsigned long long *keysB, int *list)
{
    __shared__ int sHist[kBins * kHugeWarps];
    __shared__ unsigned sMask[kBins * kHugeWarps];
    __shared__ int sWarp[kHugeWarps];
    __shared__ int sTake, sWord;
    b200sp::WaitForPrevious();
    if (list[kCountHuge] == 0) return;
    const int count = list[kCountLong];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (;;) {
        __syncthreads();
        if (tid == 0) sTake = atomicAdd(list + kTake + kCountHuge, 1);
        __syncthreads();
        if (sTake >= count) break;
        const int entry = list[kListHead + 2ll * m - 1 - sTake];
        if (entry >= 0) continue;
        const int row = ~entry;
        const int s = rowPtr[row] - base, len = rowPtr[row + 1] - base - s;
        unsigned long long *src = keysA + s, *dst = keysB + s;
        if (tid == 0) sWord = 0;
        __syncthreads();
        unsigned seen = 0;
        for (int i = tid; i < len; i += kHugeThreads) {
            const unsigned c = (unsigned)colInd[s + i];
            src[i] = ((unsigned long long)c << 32) | (unsigned)i;
            seen |= c;
        }
        seen = __reduce_or_sync(0xffffffffu, seen);
        if (lane == 0) atomicOr(&sWord, (int)seen);
        __syncthreads();
        const int bits = sWord == 0 ? 1 : 32 - __clz((unsigned)sWord);
        const int per = ((len + kHugeWarps - 1) / kHugeWarps + 31) & ~31;
        const int w0 = warp * per < len ? warp * per : len, w1 = w0 + per < len ? w0 + per : len;
        for (int shift = 32; shift < 32 + bits; shift += kDigitBits) {
            for (int i = tid; i < kBins * kHugeWarps; i += kHugeThreads) {
                sHist[i] = 0;
                sMask[i] = 0;
            }
            __syncthreads();
            for (int i = w0 + lane; i < w1; i += 4 * 32) {  // four loads in flight per lane
                unsigned long long k[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) k[u] = i + 32 * u < w1 ? src[i + 32 * u] : 0ull;
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (i + 32 * u < w1) atomicAdd(&sHist[warp * kBins + ((unsigned)(k[u] >> shift) & (kBins - 1))], 1);
            }
            __syncthreads();
            {
                int c[kHugeWarps], tot = 0;
#pragma unroll
                for (int w = 0; w < kHugeWarps; ++w) {
                    c[w] = sHist[w * kBins + tid];
                    tot += c[w];
                }
                int before = b200sp_radix::CtaInclusiveScan<kHugeThreads>(tot, sWarp) - tot;
#pragma unroll
                for (int w = 0; w < kHugeWarps; ++w) {
                    sHist[w * kBins + tid] = before;
                    before += c[w];
                }
            }
            __syncthreads();
            unsigned long long ahead = w0 + lane < w1 ? src[w0 + lane] : 0ull;  // the next step's key, a step early
            for (int i0 = w0; i0 < w1; i0 += 32) {
                const bool in = i0 + lane < w1;
                const unsigned long long key = ahead;
                ahead = i0 + lane + 32 < w1 ? src[i0 + lane + 32] : 0ull;
                const unsigned d = (unsigned)(key >> shift) & (kBins - 1);
                if (in) atomicOr(&sMask[warp * kBins + d], 1u << lane);
                __syncwarp();
                const unsigned peers = in ? *(volatile unsigned *)&sMask[warp * kBins + d] : 0u;
                const int rank = __popc(peers & ((1u << lane) - 1u));
                int pos = 0;
                if (in) pos = sHist[warp * kBins + d] + rank;
                __syncwarp();
                if (in && rank == 0) {
                    sHist[warp * kBins + d] += __popc(peers);
                    sMask[warp * kBins + d] = 0;
                }
                __syncwarp();
                if (in) dst[pos] = key;
            }
            __syncthreads();
            unsigned long long *t = src;
            src = dst;
            dst = t;
        }
        // P goes through the array the keys are not in: it is read at arbitrary places before any of it is written.
        unsigned *park = reinterpret_cast<unsigned *>(dst);
        for (int i = tid; i < len; i += kHugeThreads) park[i] = (unsigned)P[s + (int)(unsigned)src[i]];
        __syncthreads();
        for (int i = tid; i < len; i += kHugeThreads) {
            colInd[s + i] = (int)(src[i] >> 32);
            P[s + i] = (int)park[i];
        }
    }
}

inline size_t ListBytes(long long rows) { return (sizeof(int) * (size_t)(2 * rows + kListHead) + 255) / 256 * 256; }

// `shortest`: of the rows this kernel takes.  Not launched when nnz leaves no room for one.
template <int kThreads, int kMax, int kClass>
inline cudaError_t LaunchCta(const int *rowPtr, int base, int m, int nnz, int *colInd, int *P, int *list, int shortest, cudaStream_t stream)
{
    if (nnz < shortest) return cudaSuccess;
    constexpr int kSmem = CtaShape<kThreads, kMax>::kSmem;
    constexpr int kByThreads = 2048 / kThreads, kBySmem = 227 * 1024 / (kSmem + 1024);
    constexpr int kPerSm = kByThreads < kBySmem ? kByThreads : kBySmem;
    static std::atomic<bool> configured[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!configured[dev].load(std::memory_order_relaxed)) {
        const cudaError_t e = cudaFuncSetAttribute(RowSortCtaKernel<kThreads, kMax, kClass>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
        if (e != cudaSuccess) return e;
        configured[dev].store(true, std::memory_order_relaxed);
    }
    const long long most = nnz / shortest, fit = (long long)kPerSm * b200sp_sm_count();
    b200sp_note_launches(1);
    return b200sp::LaunchChained(RowSortCtaKernel<kThreads, kMax, kClass>, (unsigned)(most < fit ? most : fit), kThreads, kSmem, stream,
                                 rowPtr, base, m, colInd, P, list);
}

// `list` holds ListBytes(m) bytes; keysA / keysB a key per entry (touched only for rows of more than kLargeMax).
inline cudaError_t Sort(const int *rowPtr, int base, int m, int n, int nnz, int *colInd, int *P, unsigned long long *keysA,
                        unsigned long long *keysB, int *list, cudaStream_t stream)
{
    if (m <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(list, 0, sizeof(int) * kListHead, stream);
    if (e != cudaSuccess) return e;
    const int sms = b200sp_sm_count();
    int rowsPerWarp = 32;  // fewer when that leaves SMs without warps
    while (rowsPerWarp > 1 && m / rowsPerWarp < 16 * sms) rowsPerWarp /= 2;
    const long long warps = ((long long)m + rowsPerWarp - 1) / rowsPerWarp;
    b200sp_note_launches(1);
    e = b200sp::LaunchChained(RowSortShortKernel, (unsigned)((warps + 7) / 8), 256, 0, stream, rowPtr, base, m, rowsPerWarp, colInd,
                              P, list);
    if (e == cudaSuccess)
        e = LaunchCta<1024, kLargeMax, kCountLong>(rowPtr, base, m, nnz, colInd, P, list, kBigMax + 1, stream);
    if (e == cudaSuccess) e = LaunchCta<512, kBigMax, kCountBig>(rowPtr, base, m, nnz, colInd, P, list, kMidMax + 1, stream);
    if (e == cudaSuccess) e = LaunchCta<256, kMidMax, kCountMid>(rowPtr, base, m, nnz, colInd, P, list, kWarpMax + 1, stream);
    if (e == cudaSuccess && nnz > 32) {
        const long long most = (nnz / 33 + 3) / 4;
        const unsigned grid = (unsigned)(most < 64ll * sms ? most : 64ll * sms);
        b200sp_note_launches(1);
        e = b200sp::LaunchChained(n < (1 << 24) - 2 ? RowSortWarpKernel<unsigned> : RowSortWarpKernel<unsigned long long>, grid, 128,
                                  0, stream, rowPtr, base, colInd, P, (const int *)list);
    }
    if (e == cudaSuccess && nnz > kLargeMax) {
        const long long most = nnz / (kLargeMax + 1);
        b200sp_note_launches(1);
        e = b200sp::LaunchChained(RowSortHugeKernel, (unsigned)(most < 4 * sms ? most : 4 * sms), kHugeThreads, 0, stream, rowPtr,
                                  base, m, colInd, P, keysA, keysB, list);
    }
    return e;
}

}  // namespace b200sp_rowsort
