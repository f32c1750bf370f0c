// Stable least-significant-digit radix sort of (column, row, value) triples in global memory, for aclsparseCsr2cscEx2.
//
// One pass is four launches, none of which waits for another CTA: a histogram of the digit per tile; prefix sums of every
// digit's counts over chunks of tiles, then over chunks and digits; and the scatter, in which a tile ranks its entries
// (stable: by digit, then by their present order), reorders them in shared memory and writes every digit's run to its
// place with consecutive addresses.  Columns of b bits take ceil(b / 10) passes of equal digits, so a million columns
// take two.  The first pass reads the caller's columns and makes the rows from the row offsets; the last one leaves
// rows and values in the caller's arrays.
//
// What bounds a scatter pass is the number of 32-byte sectors it stores (a tile of 8192 entries meets 1024 digits eight
// times each, so a run is about a sector long, unaligned: 85 us per 4-byte array of 31 M entries).  So as few arrays
// as possible move: with up to two passes the first packs the row and the digit of the second into one word where
// they fit, and the column offsets come from the counts instead of from sorted columns.
#pragma once

#include <atomic>
#include <cstdint>

#include <cuda_runtime.h>

#include "common/chained.cuh"
#include "common/rows.cuh"

namespace b200sp_radix {

constexpr int kMaxDigitBits = 10;
constexpr int kMaxBins = 1 << kMaxDigitBits;
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kItemsLarge = 16, kItemsSmall = 4;  // entries per thread; tiles of 8192, or of 2048 while those fill the SMs better

inline int ItemsFor(long long nnz) { return nnz <= (1ll << 20) ? kItemsSmall : kItemsLarge; }
inline long long TilesFor(long long nnz)
{
    const long long tile = (long long)kThreads * ItemsFor(nnz);
    return (nnz + tile - 1) / tile;
}

// Rank of this lane's entry among its warp's entries with the same digit so far, in order (step, lane): `masks` and
// `counts` hold a word and a count per digit for this warp alone, masks zero before and after.  The lanes of a digit
// find each other through an atomic OR in shared memory: 31 M entries with 10-bit digits spend 43 us of a scatter pass
// here; a ballot per bit and, worse, match.any (a turn per distinct value) keep the pipe of the votes busy longer.
__device__ __forceinline__ int RankStep(uint32_t *masks, uint16_t *counts, int digit, bool in, int lane)
{
    if (in) atomicOr(masks + digit, 1u << lane);
    __syncwarp();
    uint32_t peers = 0;
    int before = 0;
    if (in) {
        peers = *static_cast<volatile uint32_t *>(masks + digit);
        before = *static_cast<volatile uint16_t *>(counts + digit);
    }
    const int rank = __popc(peers & ((1u << lane) - 1u));
    __syncwarp();
    if (in && rank == 0) {  // the lowest lane of every digit
        masks[digit] = 0;
        counts[digit] = (uint16_t)(before + __popc(peers));
    }
    __syncwarp();
    return before + rank;
}

// Which digit an entry has: (its word >> shift) & (bins - 1), where the word is a column minus the index base, or what an
// earlier pass left (a column, or (row << digit bits) | digit with shift 0).
__device__ __forceinline__ int DigitOf(int word, int base, int shift, int bins)
{
    return (int)((unsigned)(word - base) >> shift) & (bins - 1);
}

// counts[tile][digit]
template <int kItems>
static __global__ void __launch_bounds__(kThreads) HistogramKernel(const int *__restrict__ words, int nnz, int base, int shift,
                                                                   int bins, int *__restrict__ counts)
{
    __shared__ int sHist[kMaxBins];
    b200sp::WaitForPrevious();
    for (int i = threadIdx.x; i < bins; i += kThreads) sHist[i] = 0;
    __syncthreads();
    const long long first = (long long)blockIdx.x * kThreads * kItems;
    int k[kItems];
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
        const long long i = first + u * kThreads + threadIdx.x;
        k[u] = i < nnz ? __ldg(words + i) : 0;
    }
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
        const long long i = first + u * kThreads + threadIdx.x;
        if (i < nnz) atomicAdd(&sHist[DigitOf(k[u], base, shift, bins)], 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < bins; i += kThreads) counts[(long long)blockIdx.x * bins + i] = sHist[i];
}

// Inclusive scan of one value per thread over the CTA; sWarp holds one int per warp.
template <int kCtaThreads>
__device__ __forceinline__ int CtaInclusiveScan(int x, int *sWarp)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += t;
    }
    if (lane == 31) sWarp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < kCtaThreads / 32 ? sWarp[lane] : 0;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, w, d);
            if (lane >= d) w += t;
        }
        if (lane < kCtaThreads / 32) sWarp[lane] = w;
    }
    __syncthreads();
    const int before = warp > 0 ? sWarp[warp - 1] : 0;
    __syncthreads();
    return x + before;
}

// A thread per digit and chunk of kChunk tiles: counts[tile][digit] becomes the count in the chunk's tiles before it,
// chunks[chunk][digit] the chunk's sum.
constexpr int kChunk = 64;
inline int ChunksFor(long long tiles) { return (int)((tiles + kChunk - 1) / kChunk); }
static __global__ void __launch_bounds__(128) ScanTilesKernel(int *__restrict__ counts, int tiles, int bins, int *__restrict__ chunks)
{
    b200sp::WaitForPrevious();
    const int digitBlocks = (bins + 127) / 128;
    const int d = (int)(blockIdx.x % digitBlocks) * 128 + threadIdx.x, chunk = blockIdx.x / digitBlocks;
    if (d >= bins) return;
    const int t0 = chunk * kChunk, t1 = t0 + kChunk < tiles ? t0 + kChunk : tiles;
    int run = 0;
    for (int t = t0; t < t1; t += 16) {
        int v[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = t + u < t1 ? counts[(long long)(t + u) * bins + d] : 0;
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            if (t + u < t1) counts[(long long)(t + u) * bins + d] = run;
            run += v[u];
        }
    }
    chunks[(long long)chunk * bins + d] = run;
}

// One CTA, a thread per digit: chunks[chunk][digit] becomes the count in the chunks before it, starts[digit] the first
// place of the digit in the output (starts[bins] = all).
static __global__ void __launch_bounds__(kMaxBins) ScanChunksKernel(int *__restrict__ chunks, int count, int bins, int *__restrict__ starts)
{
    __shared__ int sWarp[32];
    b200sp::WaitForPrevious();
    const int d = threadIdx.x;
    int run = 0;
    if (d < bins) {
        for (int c = 0; c < count; c += 16) {
            int v[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) v[u] = c + u < count ? chunks[(long long)(c + u) * bins + d] : 0;
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                if (c + u < count) chunks[(long long)(c + u) * bins + d] = run;
                run += v[u];
            }
        }
    }
    const int incl = CtaInclusiveScan<kMaxBins>(run, sWarp);
    if (d < bins) starts[d] = incl - run;
    if (d == bins - 1) starts[bins] = incl;
}

template <int kBytes> struct Value { using Type = uint32_t; };  // 4, and a placeholder for 0
template <> struct Value<1> { using Type = uint8_t; };
template <> struct Value<2> { using Type = uint16_t; };

struct PassArgs {
    const int *words;     // present order: columns, or packed words
    const int *rows;      // kKeys and not kFirst: rows beside the columns
    const void *vals;
    int *outWords;        // columns (kKeys), packed words, or nothing
    int *outRows;         // kKeys or the last pass: rows
    void *outVals;
    const int *rowPtr;    // kFirst
    int m, nnz, base;
    int wordBase;         // subtracted from the words read: the index base in the first pass
    int rowPlus;          // added to the rows written: the index base in the last pass
    int shift, digitBits, bins, tiles;
    const int *prefix;    // counts, chunks and starts after the scans
    const int *chunks;
    const int *starts;
};

template <int kItems> constexpr int ScatterSmem()
{
    constexpr int kArrays = kThreads * kItems * 8, kMasks = kWarps * kMaxBins * 4;
    return (kArrays > kMasks ? kArrays : kMasks) + kWarps * kMaxBins * 2 + 2 * kMaxBins * 4;
}

// Rows of the tile's entries, from the row offsets: a bit per entry that starts a (non-empty) row, the rows in order of
// their starts, and a running count of bits; an entry's row is then three shared-memory reads away, whatever the
// lengths of the rows.  A tile that spans far more rows than it has entries (most of them empty) does not go through
// them all: every entry's row is searched for between those of the warp's first and last one.  The whole conversion, us with
// every tile walked through and so, at 8, 16, 20, 50, 500 and 50,000 rows an entry: 486 and 419 (5 M entries), 68 and 45
// (250,000), 415 and 236 (2 M), 119 and 45 (20,000), 1976 and 68 (100,000), 88,496 and 44 (1000); at four the walk is no dearer.
constexpr int kWalkRows = 8;  // per entry of the tile
template <int kItems>
__device__ __forceinline__ void RowsOfTile(const PassArgs &a, long long first, int live, unsigned char *sRaw, int *sWarp,
                                           int (&row)[kItems])
{
    constexpr int kTile = kThreads * kItems, kWords = kTile / 32;
    static_assert(kWords <= kThreads, "a thread per word of bits");
    uint32_t *sBits = reinterpret_cast<uint32_t *>(sRaw);
    int *sBefore = reinterpret_cast<int *>(sBits + kWords);  // rows that start in the words before
    int *sList = sBefore + kWords;                           // [kTile]
    int *sEnds = sWarp;                                      // {first row, last row} of the tile
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < kWords) sBits[tid] = 0;
    if (warp < 2) {
        const int r = b200sp::WarpRowOf(a.rowPtr, a.m, warp == 0 ? first : first + live - 1, lane, a.base);
        if (lane == 0) sEnds[warp] = r;
    }
    __syncthreads();
    const int r0 = sEnds[0], r1 = sEnds[1];
    if (r1 - r0 > kWalkRows * kTile) {
        const int w0 = warp * 32 * kItems, w1 = w0 + 32 * kItems < live ? w0 + 32 * kItems : live;  // the warp's entries
#pragma unroll
        for (int u = 0; u < kItems; ++u) row[u] = 0;
        if (w0 < w1) {
            const int from = r0 + b200sp::WarpRowOf(a.rowPtr + r0, r1 - r0 + 1, first + w0, lane, a.base);
            const int to = r0 + b200sp::WarpRowOf(a.rowPtr + r0, r1 - r0 + 1, first + w1 - 1, lane, a.base);
#pragma unroll
            for (int u = 0; u < kItems; ++u) row[u] = from;
            for (int step = to > from ? 1 << (31 - __clz(to - from)) : 0; step > 0; step >>= 1) {  // all entries of a lane at once
#pragma unroll
                for (int u = 0; u < kItems; ++u) {
                    const bool ok = step <= to - row[u] && w0 + u * 32 + lane < w1 &&
                                    (long long)__ldg(a.rowPtr + row[u] + step) - a.base <= first + w0 + u * 32 + lane;
                    if (ok) row[u] += step;
                }
            }
        }
        __syncthreads();  // the space serves the ranking next
        return;
    }
    for (int r = r0 + tid; r <= r1; r += kThreads) {
        const long long s = (long long)__ldg(a.rowPtr + r) - a.base - first, e = (long long)__ldg(a.rowPtr + r + 1) - a.base - first;
        if (e > s && e > 0) {
            const int at = s > 0 ? (int)s : 0;
            atomicOr(sBits + (at >> 5), 1u << (at & 31));
        }
    }
    __syncthreads();
    const int n = tid < kWords ? __popc(sBits[tid]) : 0;
    const int incl = CtaInclusiveScan<kThreads>(n, sWarp);
    if (tid < kWords) sBefore[tid] = incl - n;
    __syncthreads();
    for (int r = r0 + tid; r <= r1; r += kThreads) {
        const long long s = (long long)__ldg(a.rowPtr + r) - a.base - first, e = (long long)__ldg(a.rowPtr + r + 1) - a.base - first;
        if (e > s && e > 0) {
            const int at = s > 0 ? (int)s : 0;
            sList[sBefore[at >> 5] + __popc(sBits[at >> 5] & ((1u << (at & 31)) - 1u))] = r;
        }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
        const int w = warp * kItems + u;  // the word of this warp's step: 32 entries
        const int at = sBefore[w] + __popc(sBits[w] & (0xffffffffu >> (31 - lane))) - 1;
        row[u] = w * 32 + lane < live ? sList[at] : 0;
    }
    __syncthreads();  // the space serves the ranking next
}

// kKeys: columns travel in an array of their own, beside the rows.  Otherwise a pass that is not the last leaves
// (row << digitBits) | (column >> digitBits), and the last one leaves rows.
template <int kItems, int kBytes, bool kFirst, bool kLast, bool kKeys>
static __global__ void __launch_bounds__(kThreads, 2) ScatterKernel(const PassArgs a)
{
    using Val = typename Value<kBytes>::Type;
    constexpr int kTile = kThreads * kItems;
    constexpr int kPerWarp = 32 * kItems;
    extern __shared__ __align__(16) unsigned char sRaw[];
    int *sMove = reinterpret_cast<int *>(sRaw);                               // [kTile] an array in its new order
    int *sWord = sMove + kTile;                                               // [kTile] columns in their new order (kKeys)
    uint16_t *sDigit = reinterpret_cast<uint16_t *>(sWord);                   // [kTile] or just the digits
    uint32_t *sMask = reinterpret_cast<uint32_t *>(sRaw);                     // [warp][digit], before the space serves those
    uint16_t *sCount = reinterpret_cast<uint16_t *>(sRaw + ScatterSmem<kItems>() - kWarps * kMaxBins * 2 - 2 * kMaxBins * 4);
    int *sStart = reinterpret_cast<int *>(sCount + kWarps * kMaxBins);        // [digit] first place in the tile
    int *sDest = sStart + kMaxBins;                                           // [digit] global place minus place in the tile
    __shared__ int sWarp[kWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int bins = a.bins;
    b200sp::WaitForPrevious();
    const long long first = (long long)blockIdx.x * kTile;
    const int live = a.nnz - first < kTile ? (int)(a.nnz - first) : kTile;

    // A warp's entries are consecutive, lane by lane within a step: their order is (step, lane).
    const int w0 = warp * kPerWarp + lane;
    int word[kItems];
#pragma unroll
    for (int u = 0; u < kItems; ++u) word[u] = w0 + u * 32 < live ? __ldg(a.words + first + w0 + u * 32) : 0;
    int row[kItems];
    if constexpr (kFirst) RowsOfTile<kItems>(a, first, live, sRaw, sWarp, row);
    for (int i = tid; i < kWarps * kMaxBins / 2; i += kThreads) reinterpret_cast<uint32_t *>(sCount)[i] = 0;
    for (int i = tid; i < kWarps * bins; i += kThreads) sMask[i] = 0;
    __syncthreads();

    // Rank of every entry among its warp's entries with the same digit; digit in the upper half of `place`.
    uint32_t place[kItems];
    uint16_t *mine = sCount + warp * kMaxBins;
    uint32_t *masks = sMask + warp * bins;
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
        const int d = DigitOf(word[u], a.wordBase, a.shift, bins);
        place[u] = ((uint32_t)d << 16) | (uint32_t)RankStep(masks, mine, d, w0 + u * 32 < live, lane);
    }
    __syncthreads();

    // Counts -> first place of (digit, warp) in the tile, and of every digit in the output.
    {
        constexpr int kPer = kMaxBins / kThreads;  // digits of a thread, consecutive
        int tot[kPer], glob[kPer], sum = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int d = tid * kPer + k;
            tot[k] = glob[k] = 0;
            if (d < bins) {
                glob[k] = __ldg(a.starts + d) + __ldg(a.prefix + (long long)blockIdx.x * bins + d) +
                          __ldg(a.chunks + (long long)(blockIdx.x / kChunk) * bins + d);
#pragma unroll
                for (int w = 0; w < kWarps; ++w) {
                    const int c = sCount[w * kMaxBins + d];
                    sCount[w * kMaxBins + d] = (uint16_t)tot[k];
                    tot[k] += c;
                }
            }
            sum += tot[k];
        }
        int start = CtaInclusiveScan<kThreads>(sum, sWarp) - sum;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int d = tid * kPer + k;
            if (d < bins) {
                sStart[d] = start;
                sDest[d] = glob[k] - start;
            }
            start += tot[k];
        }
    }
    __syncthreads();

#pragma unroll
    for (int u = 0; u < kItems; ++u) {
        const int i = w0 + u * 32;
        if (i < live) {
            const int d = (int)(place[u] >> 16);
            const int to = (int)(place[u] & 0xffffu) + mine[d] + sStart[d];
            place[u] = (uint32_t)to;
            const int w = word[u] - a.wordBase;
            if constexpr (kKeys) {
                sWord[to] = w;
                sMove[to] = kFirst ? row[u] : __ldg(a.rows + first + i);
            } else {
                sDigit[to] = (uint16_t)d;
                if constexpr (kFirst && !kLast) sMove[to] = (int)((unsigned)row[u] << a.digitBits | (unsigned)w >> a.digitBits);
                else if constexpr (kFirst) sMove[to] = row[u];
                else sMove[to] = (int)((unsigned)w >> a.digitBits);
            }
        }
    }
    [[maybe_unused]] Val val[kItems];
    if constexpr (kBytes > 0) {  // requested here, used after the barriers
#pragma unroll
        for (int u = 0; u < kItems; ++u)
            val[u] = w0 + u * 32 < live ? __ldg(static_cast<const Val *>(a.vals) + first + w0 + u * 32) : Val(0);
    }
    __syncthreads();
    int to[kItems];  // where the entry that now lies at u * kThreads + tid goes
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
        const int i = u * kThreads + tid;
        if (i < live) {
            const int d = kKeys ? DigitOf(sWord[i], 0, a.shift, bins) : (int)sDigit[i];
            to[u] = sDest[d] + i;
            if constexpr (kKeys) a.outWords[to[u]] = sWord[i];
            if constexpr (kKeys || kLast) a.outRows[to[u]] = sMove[i] + a.rowPlus;
            else a.outWords[to[u]] = sMove[i];
        }
    }
    if constexpr (kBytes > 0) {
        __syncthreads();
        Val *sVal = reinterpret_cast<Val *>(sMove);
#pragma unroll
        for (int u = 0; u < kItems; ++u)
            if (w0 + u * 32 < live) sVal[place[u]] = val[u];
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kItems; ++u) {
            const int i = u * kThreads + tid;
            if (i < live) static_cast<Val *>(a.outVals)[to[u]] = sVal[i];
        }
    }
}

// Column offsets from the counts of the last of at most two passes.  With one pass the digits are the columns.  With two,
// column (hi, lo) starts where the entries with digit hi that lie before the first entry with low digit lo end: a CTA
// per lo counts, in the tile in which that entry lies, the digits before it.
template <int kItems>
static __global__ void __launch_bounds__(256) OffsetsFromCountsKernel(const int *__restrict__ words, int nnz, int n, int passes,
                                                                      int digitBits, const int *__restrict__ lowStarts,
                                                                      const int *__restrict__ prefix, const int *__restrict__ chunks,
                                                                      const int *__restrict__ starts, int base, int *__restrict__ colPtr)
{
    constexpr int kTile = kThreads * kItems;
    __shared__ int sHist[kMaxBins];
    b200sp::WaitForPrevious();
    const int bins = 1 << digitBits, lo = blockIdx.x;
    if (lo == 0 && threadIdx.x == 0) colPtr[n] = nnz + base;
    if (passes == 1) {
        for (int c = threadIdx.x; c < n; c += 256) colPtr[c] = __ldg(starts + c) + base;
        return;
    }
    for (int i = threadIdx.x; i < bins; i += 256) sHist[i] = 0;
    __syncthreads();
    const int q = __ldg(lowStarts + lo), tile = q / kTile;
    const bool end = q >= nnz;
    if (!end)
        for (int i = tile * kTile + threadIdx.x; i < q; i += 256) atomicAdd(&sHist[__ldg(words + i) & (bins - 1)], 1);
    __syncthreads();
    for (int hi = threadIdx.x; hi < bins; hi += 256) {
        const long long c = ((long long)hi << digitBits) | lo;
        if (c >= n) break;
        colPtr[c] = base + (end ? __ldg(starts + hi + 1)
                                : __ldg(starts + hi) + __ldg(prefix + (long long)tile * bins + hi) +
                                      __ldg(chunks + (long long)(tile / kChunk) * bins + hi) + sHist[hi]);
    }
}

template <int kItems, int kBytes, bool kFirst, bool kLast, bool kKeys>
inline cudaError_t LaunchScatter(const PassArgs &a, cudaStream_t stream)
{
    constexpr int kSmem = ScatterSmem<kItems>();
    static std::atomic<bool> configured[64] = {};  // per device: this instantiation may use kSmem bytes
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!configured[dev].load(std::memory_order_relaxed)) {
        const cudaError_t e = cudaFuncSetAttribute(ScatterKernel<kItems, kBytes, kFirst, kLast, kKeys>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
        if (e != cudaSuccess) return e;
        configured[dev].store(true, std::memory_order_relaxed);
    }
    b200sp_note_launches(1);
    return b200sp::LaunchChained(ScatterKernel<kItems, kBytes, kFirst, kLast, kKeys>, (unsigned)a.tiles, kThreads, kSmem, stream, a);
}

}  // namespace b200sp_radix
