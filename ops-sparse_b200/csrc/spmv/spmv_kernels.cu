// CSR SpMV kernels for sm_100a and their extern "C" launchers.
//
// The reference's device code for this operator (sparse/spmv/arch22/kernels/spmv_kernel.h:
// 27-310 non-transpose, 321-640 transpose) gives every core an equal count of rows and
// walks them one at a time.  Two designs replace it here, chosen by what the caller set up.
//
// Binned path (a buffer analysed once by aclsparseSpMVPreprocess / b200sp_spmv_analyze with
// plan_info).  The analysis lists the rows of 33..511 entries ("medium") and of >= 512
// entries ("long", ordered by descending length) as {row, start, end}; a product is then two
// launches over disjoint rows of y, the first forked onto a side stream so that they share
// the SMs:
//   SpmvLongBlockKernel     (enough long rows -- 48 per block of x --, ascending columns, at most 2 M columns)
//                           x is cut into blocks of 32768 columns; a CTA keeps one block in
//                           shared memory and sums the pieces of all long rows that fall into
//                           it, so the gathers of more than half of the non-zeros of a
//                           power-law matrix never leave the SM.  The last CTA to finish a group
//                           of rows adds their per-block partial sums in block order.
//   SpmvAllBinsKernel       (otherwise) one grid for all bins: a CTA per listed long row with 128-bit
//                           loads first, then the medium and short rows as below; no side stream.
//   SpmvMediumShortKernel   one grid: first a warp per listed medium row, then every row gets
//                           a group of G = 2 or 4 lanes (rows longer than 32 entries are
//                           skipped).  SpmvShortRowsKernel, or SpmvStagedRowsKernel for
//                           banded matrices, alone when no row is medium.
// Gathers of x from scattered columns cost one L2 sector request each, and an SM issues one
// request per clock: many light warps, each with a few independent gathers in flight, keep
// that port busy for the medium and short rows, and the long rows stay off it altogether.
//
// Rows path (no analysed buffer): SpmvRowsKernel, a group of lanes per row and the whole warp for longer ones, then
// SpmvListedKernel for the rows it listed as too long for a warp.
//
// Tile path (no analysed buffer and no room for that list; the entry point that allocates nothing: the tile table is
// rebuilt on every call, no host synchronisation).  The work is
// cut by *merge path*: the rows' end markers and the non-zeros form one merged sequence of
// rows + nnz items and every CTA takes an equal slice (a tile) of it, whatever the row
// lengths are.  A tile
//   1. gives every thread eight consecutive non-zeros at a time: 128-bit loads of col_ind / values, eight gathers of x
//      in flight, products in registers;
//   2. marks the last entry of every row that ends in it in a bitmap in shared memory; a thread adds up its products,
//      storing a row's sum at every mark, and what is left open is joined across threads with a segmented scan;
//   3. writes y with one coalesced pass (alpha * sum + beta * y).
// A row cut by a tile boundary is finished without a second kernel and without waiting:
// every tile that holds a piece stores its partial sum, then bumps an arrival counter owned
// by the tile in which the row ends; whichever tile arrives last adds the pieces in tile
// order (so the result does not depend on scheduling) and writes y.
//
// Numerics follow the reference golden SpmvCpu (test/spmv/arch22/spmv_test.cpp:156-173):
// values and x are widened to the compute type before the multiply, sums are kept in the
// compute type, the result is alpha*sum + beta*y rounded once to the output type.
// beta == 0 never reads y.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <type_traits>

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "b200sp_kernels.h"
#include "../common/chained.cuh"
#include "../common/rows.cuh"
#include "../common/side_stream.h"

namespace {

// Tuning knobs (compile-time; the defaults are the measured best on B200, see profiles/).
// Merge items (row ends + non-zeros) per tile: kTileThreads threads take eight non-zeros each per round.  Small products
// use smaller tiles, so that there are enough of them for the SMs.
constexpr int kPerThread = 8;
constexpr int TileThreads(int size) { return size == 0 ? 128 : 256; }
constexpr int TileRounds(int size) { return size == 2 ? 2 : 1; }
constexpr int TileItems(int size) { return TileThreads(size) * TileRounds(size) * 15 / 2; }  // 960, 1920, 3840: room for alignment
inline int TileSizeFor(int64_t rows, int64_t nnz)
{
    return rows + nnz <= (1ll << 18) ? 0 : rows + nnz <= (1ll << 23) ? 1 : 2;
}

inline size_t AlignUp(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Rows of at least kLongLen entries form the "long" bin of the binned path (see below).  Measured on the
// 1,048,576-row power-law matrix (us per product): 1024: 95.0, 768: 94.5, 512: 90.6, 384: 104.2.
#ifndef B200SP_SPMV_LONG_LEN
#define B200SP_SPMV_LONG_LEN 512
#endif
constexpr int kLongLen = B200SP_SPMV_LONG_LEN;

// Long rows that keep CTAs of their own (the list path) are cut into segments of kSegLen entries, a CTA each: a
// 16384-entry row is then eight CTAs working side by side instead of one CTA making eight round trips to memory,
// which is what bounded a product on a small shard.  A row of several segments is finished by whichever of its
// CTAs arrives last: it adds the segments' partial sums in segment order (no wait, fixed order).
// One eighth of the power-law matrix (131,081 rows, 978 long ones, 3.8 M entries), whole product: segments of
// 2048 / 4096 / 8192 entries 22.6 / 21.9 / 20.6 us; one sixteenth: 14.4 / 14.0 / 14.4.
#ifndef B200SP_SPMV_SEG_LEN
#define B200SP_SPMV_SEG_LEN 8192
#endif
constexpr int kSegLen = B200SP_SPMV_SEG_LEN;


struct PlanLayout {  // tile plan: what SpmvTileKernel needs
    int64_t ntiles;
    int size;  // which TileItems
    size_t offTileRow, offCounters, offHead, offTail, total;
};

inline PlanLayout LayoutFor(int64_t rows, int64_t nnz)
{
    PlanLayout L;
    L.size = TileSizeFor(rows, nnz);
    L.ntiles = (rows + nnz + TileItems(L.size) - 1) / TileItems(L.size);
    L.offTileRow = 0;
    L.offCounters = AlignUp(L.offTileRow + sizeof(int32_t) * (size_t)(L.ntiles + 1), 256);
    L.offHead = AlignUp(L.offCounters + sizeof(int32_t) * (size_t)L.ntiles, 256);
    L.offTail = AlignUp(L.offHead + 4 * (size_t)L.ntiles, 256);
    L.total = AlignUp(L.offTail + 4 * (size_t)L.ntiles, 256);
    if (L.total == 0) L.total = 256;
    return L;
}

// ---------------------------------------------------------------- element helpers

template <typename CompT, typename T>
__device__ __forceinline__ CompT Widen(T v);
template <> __device__ __forceinline__ float Widen<float, float>(float v) { return v; }
template <> __device__ __forceinline__ float Widen<float, __half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float Widen<float, __nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float Widen<float, int32_t>(int32_t v) { return static_cast<float>(v); }
template <> __device__ __forceinline__ int32_t Widen<int32_t, int32_t>(int32_t v) { return v; }

template <typename OutT, typename CompT>
__device__ __forceinline__ OutT Narrow(CompT v);
template <> __device__ __forceinline__ float Narrow<float, float>(float v) { return v; }
template <> __device__ __forceinline__ __half Narrow<__half, float>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 Narrow<__nv_bfloat16, float>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ int32_t Narrow<int32_t, int32_t>(int32_t v) { return v; }

template <typename CompT>
struct Scalars {
    CompT alpha, beta;
    const CompT *alphaDev, *betaDev;
    __device__ __forceinline__ CompT Alpha() const { return alphaDev ? *alphaDev : alpha; }
    __device__ __forceinline__ CompT Beta() const { return betaDev ? *betaDev : beta; }
};

// Four consecutive matrix values, streamed (evict-first) so they do not push x out of cache.
template <typename T>
struct Quad {
    T v[4];
};
__device__ __forceinline__ Quad<float> LoadQuad(const float *p)
{
    const float4 q = __ldcs(reinterpret_cast<const float4 *>(p));
    return {{q.x, q.y, q.z, q.w}};
}
__device__ __forceinline__ Quad<int32_t> LoadQuad(const int32_t *p)
{
    const int4 q = __ldcs(reinterpret_cast<const int4 *>(p));
    return {{q.x, q.y, q.z, q.w}};
}
__device__ __forceinline__ Quad<__half> LoadQuad(const __half *p)
{
    const uint2 q = __ldcs(reinterpret_cast<const uint2 *>(p));
    Quad<__half> r;
    *reinterpret_cast<uint2 *>(r.v) = q;
    return r;
}
__device__ __forceinline__ Quad<__nv_bfloat16> LoadQuad(const __nv_bfloat16 *p)
{
    const uint2 q = __ldcs(reinterpret_cast<const uint2 *>(p));
    Quad<__nv_bfloat16> r;
    *reinterpret_cast<uint2 *>(r.v) = q;
    return r;
}

template <typename CompT>
__device__ __forceinline__ CompT GroupSum(CompT v, int lanes)
{
    for (int off = lanes >> 1; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// ---------------------------------------------------------------- analysis

// One warp per tile boundary: search of diagonal t * items on the merge grid of (row end offsets, non-zero indices), 32
// probes per round.  tileRow[t] = number of rows that end before the tile.
__global__ void __launch_bounds__(256) SpmvTileSearchKernel(const int32_t *__restrict__ rowPtr, int rows, int nnz, int ntiles,
                                                            int items, int32_t *__restrict__ tileRow,
                                                            int32_t *__restrict__ counters)
{
    b200sp::WaitForPrevious();
    const int lane = threadIdx.x & 31;
    const int t = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (t > ntiles) return;
    const long long total = (long long)rows + nnz;
    long long d = (long long)t * items;
    if (d > total) d = total;
    long long lo = d - nnz > 0 ? d - nnz : 0;
    long long hi = d < rows ? d : rows;  // the answer lies in [lo, hi]; rows below it end before the diagonal
    while (lo < hi) {
        const long long step = (hi - lo + 31) / 32;
        const long long mid = lo + (lane + 1) * step - 1;
        const bool before = mid < hi && (long long)__ldg(rowPtr + mid + 1) <= d - mid - 1;
        const int n = __popc(__ballot_sync(0xffffffffu, before));
        const long long next = lo + (n + 1) * step - 1;  // the first probe that was not
        lo += n * step;
        hi = next < hi ? next : hi;
    }
    if (lane == 0) {
        tileRow[t] = (int32_t)lo;
        if (t < ntiles) counters[t] = 0;
    }
}

// ---------------------------------------------------------------- tile kernel

template <typename CompT, typename ValT, typename OutT>
struct TileArgs {
    const int32_t *rowPtr;
    const int32_t *colInd;
    const ValT *val;
    const ValT *x;
    OutT *y;
    int rows;
    int nnz;
    Scalars<CompT> sc;
    const int32_t *tileRow;
    int32_t *counters;
    CompT *partHead;
    CompT *partTail;
};

// Measured, bf16, 300,007 ragged rows with 7.2 M entries (search included): products parked in shared memory and walked
// from there 57 us, 51 us so; bound by the barriers and the chain table -> columns -> x (a persistent form with the next
// tile's entries requested ahead needs 64 registers and took 57).  SpmvRowsKernel, which has neither, is the first choice.
template <typename CompT, typename ValT, typename OutT, bool kVec, int kSize>
__global__ void __launch_bounds__(TileThreads(kSize)) SpmvTileKernel(const TileArgs<CompT, ValT, OutT> a)
{
    constexpr int kTileThreads = TileThreads(kSize), kRounds = TileRounds(kSize), kTileItems = TileItems(kSize);
    constexpr int kSpans = kTileThreads / 32 * kRounds;      // a span: 256 consecutive entries, one round of one warp
    constexpr int kWords = kTileThreads * kRounds * kPerThread / 32;
    __shared__ CompT sRowSum[kTileItems];                    // finished sum of every row that ends here
    __shared__ uint16_t sList[kTileItems];                   // rows that end at a non-zero of the tile, in order
    __shared__ uint32_t sBits[kWords];                       // bit: this entry is the last of its row
    __shared__ int sBefore[kWords];                          // marks in the words before
    __shared__ CompT sOpen[kSpans];                          // what a span leaves open at its end
    __shared__ int sClosed[kSpans];                          // whether it holds a mark

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int t = blockIdx.x;
    b200sp::WaitForPrevious();
    const int i0 = a.tileRow[t];
    const int i1 = a.tileRow[t + 1];
    const long long total = (long long)a.rows + a.nnz;
    const long long d0 = (long long)t * kTileItems;
    const long long d1 = d0 + kTileItems < total ? d0 + kTileItems : total;
    const int j0 = (int)(d0 - i0);
    const int j1 = (int)(d1 - i1);
    const int R = i1 - i0;       // rows whose end lies in this tile
    const int base = j0 & ~3;    // entry o of the tile's spans is entry base + o

    // ---- phase 1: this thread's entries; those outside [j0, j1) count as zero --------------------
    int c[kRounds][kPerThread];
    ValT v[kRounds][kPerThread];
#pragma unroll
    for (int h = 0; h < kRounds; ++h) {
        const int at = base + ((warp * kRounds + h) * 32 + lane) * kPerThread;
#pragma unroll
        for (int q = 0; q < kPerThread; q += 4) {
            if (kVec && at + q + 4 <= a.nnz && at + q < j1) {
                const int4 cc = __ldcs(reinterpret_cast<const int4 *>(a.colInd + at + q));
                const Quad<ValT> vv = LoadQuad(a.val + at + q);
                c[h][q] = cc.x; c[h][q + 1] = cc.y; c[h][q + 2] = cc.z; c[h][q + 3] = cc.w;
#pragma unroll
                for (int e = 0; e < 4; ++e) v[h][q + e] = vv.v[e];
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const bool in = at + q + e < j1 && at + q + e >= j0;
                    c[h][q + e] = in ? a.colInd[at + q + e] : 0;
                    v[h][q + e] = in ? a.val[at + q + e] : ValT(0);
                }
            }
        }
    }
    // y of the first rows that end here, fetched now so that the epilogue does not wait for it
    const CompT betaEarly = a.sc.Beta();
    CompT yEarly = CompT(0);
    if (betaEarly != CompT(0) && tid < R) yEarly = Widen<CompT>(a.y[i0 + tid]);

    for (int w = tid; w < kWords; w += kTileThreads) sBits[w] = 0;
    __syncthreads();
    for (int k = tid; k < R; k += kTileThreads) {
        const int s = __ldg(a.rowPtr + i0 + k), e = __ldg(a.rowPtr + i0 + k + 1);
        if (e > s && e > j0) atomicOr(sBits + ((e - 1 - base) >> 5), 1u << ((e - 1 - base) & 31));
        else sRowSum[k] = CompT(0);  // empty, or its last entry lies in the tile before
    }
    CompT p[kRounds][kPerThread];
#pragma unroll
    for (int h = 0; h < kRounds; ++h) {
        const int at = base + ((warp * kRounds + h) * 32 + lane) * kPerThread;
#pragma unroll
        for (int u = 0; u < kPerThread; ++u) {
            const bool in = at + u >= j0 && at + u < j1;
            const ValT xv = in ? __ldg(a.x + c[h][u]) : ValT(0);
            p[h][u] = in ? Widen<CompT>(v[h][u]) * Widen<CompT>(xv) : CompT(0);
        }
    }
    __syncthreads();
    if (warp == 0) {
        int n[(kWords + 31) / 32], sum = 0;
#pragma unroll
        for (int k = 0; k < (kWords + 31) / 32; ++k) {
            const int w = lane * ((kWords + 31) / 32) + k;
            n[k] = w < kWords ? __popc(sBits[w]) : 0;
            sum += n[k];
        }
        int incl = sum;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += o;
        }
        int run = incl - sum;
#pragma unroll
        for (int k = 0; k < (kWords + 31) / 32; ++k) {
            const int w = lane * ((kWords + 31) / 32) + k;
            if (w < kWords) sBefore[w] = run;
            run += n[k];
        }
    }
    __syncthreads();
    for (int k = tid; k < R; k += kTileThreads) {
        const int s = __ldg(a.rowPtr + i0 + k), e = __ldg(a.rowPtr + i0 + k + 1);
        if (e > s && e > j0) {
            const int o = e - 1 - base;
            sList[sBefore[o >> 5] + __popc(sBits[o >> 5] & ((1u << (o & 31)) - 1u))] = (uint16_t)k;
        }
    }
    __syncthreads();

    // ---- phase 2: sums between marks -----------------------------------------------------
    CompT open[kRounds];   // sum from the last mark at or before this thread's entries (within its span) to their end
    CompT into[kRounds];   // what the span's earlier threads leave open where this thread's entries begin
    int first[kRounds];    // first row this thread closes, or -1
    bool reaches[kRounds]; // no mark in the span before this thread's entries
#pragma unroll
    for (int h = 0; h < kRounds; ++h) {
        const int o = ((warp * kRounds + h) * 32 + lane) * kPerThread;
        const uint32_t word = sBits[o >> 5];
        const uint32_t marks = (word >> (o & 31)) & 0xffu;
        int k = sBefore[o >> 5] + __popc(word & ((1u << (o & 31)) - 1u));
        first[h] = marks != 0 ? sList[k] : -1;
        CompT run = CompT(0);
#pragma unroll
        for (int u = 0; u < kPerThread; ++u) {
            run += p[h][u];
            if (marks & (1u << u)) {
                sRowSum[sList[k]] = run;
                ++k;
                run = CompT(0);
            }
        }
        const uint32_t closers = __ballot_sync(0xffffffffu, marks != 0);
        const uint32_t upTo = closers & (0xffffffffu >> (31 - lane));
        const int head = upTo != 0 ? 31 - __clz(upTo) : 0;  // the sum reaches back to this lane
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const CompT o2 = __shfl_up_sync(0xffffffffu, run, off);
            if (lane - off >= head) run += o2;
        }
        open[h] = run;
        into[h] = __shfl_up_sync(0xffffffffu, run, 1);
        if (lane == 0) into[h] = CompT(0);
        reaches[h] = (closers & ((1u << lane) - 1u)) == 0;
        if (lane == 31) {
            sOpen[warp * kRounds + h] = run;
            sClosed[warp * kRounds + h] = closers != 0;
        }
    }
    __syncthreads();
    CompT tail = CompT(0);  // in the last thread: what the tile leaves open
#pragma unroll
    for (int h = 0; h < kRounds; ++h) {
        CompT carry = CompT(0);
        if (reaches[h]) {
            for (int w = warp * kRounds + h - 1; w >= 0; --w) {
                carry += sOpen[w];
                if (sClosed[w]) break;
            }
        }
        if (first[h] >= 0) sRowSum[first[h]] += into[h] + carry;
        tail = open[h] + (reaches[h] && first[h] < 0 ? carry : CompT(0));
    }
    __syncthreads();

    // ---- phase 3: coalesced epilogue ---------------------------------------------------
    const CompT alpha = a.sc.Alpha();
    const CompT beta = a.sc.Beta();
    auto storeRow = [&](int r, CompT sum) {
        CompT z = alpha * sum;
        if (beta != CompT(0)) z += beta * Widen<CompT>(a.y[r]);
        a.y[r] = Narrow<OutT>(z);
    };
    // Arrival protocol for a row r cut by tile boundaries; t1 is the tile where r ends.
    auto arrive = [&](int r, int t1) {
        __threadfence();
        const int tFirst = (int)(((long long)r + a.rowPtr[r]) / kTileItems);
        const int expected = t1 - tFirst;  // arrivals that precede the last one
        const int old = atomicAdd(a.counters + t1, 1);
        if (old == expected) {
            a.counters[t1] = 0;  // ready for the next launch
            __threadfence();
            CompT s = CompT(0);
            for (int u = tFirst; u < t1; ++u) s += __ldcg(a.partTail + u);
            s += __ldcg(a.partHead + t1);
            storeRow(r, s);
        }
    };
    const bool headContinues = R > 0 && __ldg(a.rowPtr + i0) < j0;  // row i0 began in an earlier tile
    for (int k = tid; k < R; k += kTileThreads) {
        if (k == 0 && headContinues) {
            a.partHead[t] = sRowSum[0];
            arrive(i0, t);
        } else if (k == tid) {  // y of this row was fetched at the start of the kernel
            CompT z = alpha * sRowSum[k];
            if (beta != CompT(0)) z += beta * yEarly;
            a.y[i0 + k] = Narrow<OutT>(z);
        } else {
            storeRow(i0 + k, sRowSum[k]);
        }
    }
    // Piece of the row after the last complete one, if this tile holds any of it.
    if (tid == kTileThreads - 1) {
        const int end = __ldg(a.rowPtr + i1);
        const int tailStart = end > j0 ? end : j0;
        if (i1 < a.rows && j1 > tailStart) {
            a.partTail[t] = tail;
            arrive(i1, (int)(((long long)i1 + a.rowPtr[i1 + 1]) / kTileItems));
        }
    }
}

// ---------------------------------------------------------------- binned path

// Rows are binned by length by the analysis pass and each bin has its own code:
//   short  (<= kShortMax entries)   ShortRowsBody : G = 2 or 4 lanes per row (8 compiles, for experiments), all rows scanned
//   medium (<  kLongLen entries)    MediumRowsBody: one warp per listed row
//   long   (>= kLongLen entries)    SpmvLongBlockKernel (x blocks in shared memory) or LongRowBody (a CTA per row)
// Short and medium rows share one grid; the long rows run beside it on a side stream.
#ifndef B200SP_SPMV_SHORT_MAX
#define B200SP_SPMV_SHORT_MAX 32
#endif
constexpr int kShortMax = B200SP_SPMV_SHORT_MAX;
#ifndef B200SP_SPMV_LONG_UNROLL
#define B200SP_SPMV_LONG_UNROLL 4
#endif
constexpr int kLongUnroll = B200SP_SPMV_LONG_UNROLL;  // quads in flight per thread of the long-row kernel

struct BinHeader {  // first 256 bytes of the binned plan
    int32_t medium;           // rows in the medium list
    int32_t longs;            // rows in the long list
    unsigned long long shortNnz;  // entries in short rows (picks the lane-group width)
    int32_t shortRows;
    int32_t unsorted;         // set when a long row has descending column indices
    int32_t segments;         // segments the long rows were cut into
    int32_t longestShort;     // entries of the longest short row
    int32_t pairs, nearPairs; // sampled neighbouring rows, and those whose first and last columns lie within kNear
    unsigned long long longNnz;   // entries in long rows
    int32_t longestLong;
};

// Long rows, second form: x is cut into blocks of kXBlockElems columns and every CTA of
// SpmvLongBlockKernel keeps one block in shared memory, so the gathers of the long rows never
// leave the SM (the other bins keep the L1 -> L2 request path to themselves).
#ifndef B200SP_SPMV_XBLOCK_ELEMS
#define B200SP_SPMV_XBLOCK_ELEMS 32768
#endif
#ifndef B200SP_SPMV_LONG_BLOCK_THREADS
#define B200SP_SPMV_LONG_BLOCK_THREADS 1024
#endif
#ifndef B200SP_SPMV_LONG_BLOCK_UNROLL
#define B200SP_SPMV_LONG_BLOCK_UNROLL 2
#endif
constexpr int kXBlockElems = B200SP_SPMV_XBLOCK_ELEMS;  // 128 KB of fp32 x, 64 KB of 16-bit x
constexpr int kMaxXBlocks = 64;      // wider matrices use SpmvLongListKernel
constexpr int kMaxLongGroups = 160;  // CTAs per column block
constexpr int kLongBlockThreads = B200SP_SPMV_LONG_BLOCK_THREADS;
#ifndef B200SP_SPMV_FUSE_LIST
#define B200SP_SPMV_FUSE_LIST 1      // long rows that keep a CTA each share one grid with the other bins
#endif
#ifndef B200SP_SPMV_MIN_LONG_BLOCKED
#define B200SP_SPMV_MIN_LONG_BLOCKED 64  // fewer long rows than this: not worth staging x
#endif

// Two neighbouring rows are near when they begin and end within this many columns of each other: the lanes that walk
// them in step then gather x from the same few cache lines.  Every kPairStride-th pair is looked at.
constexpr int kNear = 64, kPairStride = 32;
__global__ void SpmvBinRowsKernel(const int32_t *__restrict__ rowPtr, const int32_t *__restrict__ colInd, int rows, BinHeader *hdr,
                                  int4 *__restrict__ listM, int4 *__restrict__ listL)
{
    const int lane = threadIdx.x & 31;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long rowsPadded = ((long long)rows + stride - 1) / stride * stride;
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < rowsPadded; r += stride) {
        int shortLen = 0, isShort = 0, longest = 0;
        if (r < rows) {
            const int rs = rowPtr[r], re = rowPtr[r + 1];
            const int len = re - rs;
            // a list entry carries the row's bounds, so its kernel starts on col_ind / values at once
            if (len >= kLongLen) {
                listL[atomicAdd(&hdr->longs, 1)] = make_int4((int)r, rs, re, 0);
                atomicAdd(&hdr->longNnz, (unsigned long long)len);
                if (len > *const_cast<volatile int32_t *>(&hdr->longestLong)) atomicMax(&hdr->longestLong, len);
            } else if (len > kShortMax) listM[atomicAdd(&hdr->medium, 1)] = make_int4((int)r, rs, re, 0);
            else {
                shortLen = longest = len;
                isShort = 1;
                if (colInd != nullptr && r % kPairStride == 0 && r + 1 < rows && len > 0) {
                    const int ne = rowPtr[r + 2];
                    if (ne > re) {
                        atomicAdd(&hdr->pairs, 1);
                        if (abs(colInd[rs] - colInd[re]) <= kNear && abs(colInd[re - 1] - colInd[ne - 1]) <= kNear)
                            atomicAdd(&hdr->nearPairs, 1);
                    }
                }
            }
        }
        longest = __reduce_max_sync(0xffffffffu, longest);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            shortLen += __shfl_xor_sync(0xffffffffu, shortLen, off);
            isShort += __shfl_xor_sync(0xffffffffu, isShort, off);
        }
        if (lane == 0 && isShort) {
            atomicAdd(&hdr->shortNnz, (unsigned long long)shortLen);
            atomicAdd(&hdr->shortRows, isShort);
            if (longest > *const_cast<volatile int32_t *>(&hdr->longestShort)) atomicMax(&hdr->longestShort, longest);
        }
    }
}

// Orders a list of {row, start, end} entries by descending row length (in classes of an
// eighth of an octave; the order inside a class is arbitrary and no result depends on it), so
// that the longest rows start first and the rows that share a warp or a CTA are alike.
// One CTA: the lists hold thousands of rows, not millions.
__global__ void __launch_bounds__(1024) SpmvSortByLengthKernel(const int32_t *__restrict__ count,
                                                                const int4 *__restrict__ in, int4 *__restrict__ out)
{
    __shared__ int sHist[256];
    const int tid = threadIdx.x;
    const int n = *count;
    auto lengthClass = [](int4 ent) {
        const int len = ent.z - ent.y;             // >= 33 for every listed row
        const int k = 31 - __clz(len);             // floor(log2(len)) >= 5
        const int key = k * 8 + ((len >> (k - 3)) & 7);
        return 255 - key;                          // descending
    };
    if (tid < 256) sHist[tid] = 0;
    __syncthreads();
    for (int i = tid; i < n; i += 1024) atomicAdd(&sHist[lengthClass(in[i])], 1);
    __syncthreads();
    if (tid == 0) {
        int running = 0;
        for (int d = 0; d < 256; ++d) {
            const int c = sHist[d];
            sHist[d] = running;
            running += c;
        }
    }
    __syncthreads();
    for (int i = tid; i < n; i += 1024) {
        const int4 ent = in[i];
        out[atomicAdd(&sHist[lengthClass(ent)], 1)] = ent;
    }
}

// One CTA: segment table of the ordered long list.  Slot i (row r, entries [s, e)) gets ceil(len / kSegLen)
// consecutive entries {r, segment start, segment end, i} of `segs`, rowSeg[i] = {first partial slot, segments}, and
// a zeroed arrival counter; the order of `segs` is the order of the list (longest rows first).
__global__ void __launch_bounds__(1024) SpmvCutSegmentsKernel(BinHeader *hdr, const int4 *__restrict__ listL,
                                                               int4 *__restrict__ segs, int2 *__restrict__ rowSeg,
                                                               int32_t *__restrict__ counters)
{
    __shared__ int sWarp[32];
    __shared__ int sCarry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = hdr->longs;
    if (tid == 0) sCarry = 0;
    __syncthreads();
    for (int i0 = 0; i0 < n; i0 += 1024) {
        const int i = i0 + tid;
        int4 ent = make_int4(0, 0, 0, 0);
        int nseg = 0;
        if (i < n) {
            ent = listL[i];
            nseg = (ent.z - ent.y + kSegLen - 1) / kSegLen;
        }
        int incl = nseg;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += t;
        }
        if (lane == 31) sWarp[warp] = incl;
        __syncthreads();
        int before = sCarry;
        for (int w = 0; w < warp; ++w) before += sWarp[w];
        const int first = before + incl - nseg;
        if (i < n) {
            rowSeg[i] = make_int2(first, nseg);
            counters[i] = 0;
            for (int k = 0; k < nseg; ++k) {
                const int a = ent.y + k * kSegLen;
                segs[first + k] = make_int4(ent.x, a, a + kSegLen < ent.z ? a + kSegLen : ent.z, i);
            }
        }
        __syncthreads();
        if (tid == 1023) sCarry = before + incl;
        __syncthreads();
    }
    if (tid == 0) hdr->segments = sCarry;
}

// One warp per listed long row: checks that its column indices ascend, then cuts it at the x
// block boundaries by binary search: segStart[slot * (xBlocks + 1) + b] = first entry of the row
// whose column is >= b * kXBlockElems.
__global__ void SpmvLongSegmentsKernel(const int32_t *__restrict__ colInd, BinHeader *hdr,
                                       const int4 *__restrict__ listL, int32_t *__restrict__ segStart,
                                       int xBlocks)
{
    const int lane = threadIdx.x & 31;
    const int warpsTotal = gridDim.x * (blockDim.x >> 5);
    const int n = hdr->longs;
    for (int slot = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); slot < n; slot += warpsTotal) {
        const int4 ent = listL[slot];
        const int s = ent.y, e = ent.z;
        bool bad = false;
        for (int p = s + lane; p + 1 < e; p += 32) bad |= colInd[p] > colInd[p + 1];
        if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&hdr->unsorted, 1);
        for (int b = lane; b <= xBlocks; b += 32) {
            int lo = s, hi = e;
            if (b == xBlocks) lo = hi;
            const long long bound = (long long)b * kXBlockElems;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (colInd[mid] < bound) lo = mid + 1;
                else hi = mid;
            }
            segStart[(long long)slot * (xBlocks + 1) + b] = lo;
        }
    }
}

template <typename CompT, typename ValT, typename OutT>
struct LongBlockArgs {
    const int32_t *colInd;
    const ValT *val;
    const ValT *x;
    OutT *y;
    int cols;
    Scalars<CompT> sc;
    const int4 *list;          // {row, start, end, 0} per long row
    const int32_t *segStart;   // [slot][xBlocks + 1]
    int32_t *counters;         // [group], arrivals of the group's column-block CTAs
    CompT *partials;           // [slot][xBlocks]
    int nLong;
    int xBlocks;
    int groups;                // CTAs per column block
};

// CTA (b, g) keeps block b of x in shared memory and sums, for every long row of its group,
// the entries whose column falls in that block -- a contiguous piece of the row, because the
// column indices ascend.  kPieceLanes lanes share a piece (8, 32 or 256: see LongBlockLanes); x comes from shared memory, so the
// only global traffic is the col_ind / values stream.  The last CTA of a row group to finish
// adds each row's partial sums in block order (no wait, fixed order) and writes y.
// Registers are capped at 48 (not at the 64 a 1024-thread CTA could have): while this kernel holds an SM, the
// CTAs of the medium / short grid get what is left of the register file, and both grids are bound by latency x
// occupancy.  Timestamps taken inside the kernels on the power-law matrix: these CTAs run 30-43 us, all done 47 us
// after the first started; the medium rows beside them finish at 68 us instead of 35 alone, the short rows at
// 91.  Product time with 56 / 46 / 40 registers here: 90.2 / 86.4 / 89.2 us.
template <typename CompT, typename ValT, typename OutT, bool kVec, int kPieceLanes>
__global__ void __maxnreg__(48) SpmvLongBlockKernel(const LongBlockArgs<CompT, ValT, OutT> a)
{
    extern __shared__ __align__(16) unsigned char sRaw[];
    ValT *xs = reinterpret_cast<ValT *>(sRaw);
    const int tid = threadIdx.x;
    const int b = blockIdx.x % a.xBlocks;
    const int g = blockIdx.x / a.xBlocks;
    const int nLong = a.nLong;
    const int x0 = b * kXBlockElems;
    const int xn = a.cols - x0 < kXBlockElems ? a.cols - x0 : kXBlockElems;

    // stage the x block
    constexpr int kPer16 = 16 / (int)sizeof(ValT);
    if (reinterpret_cast<uintptr_t>(a.x) % 16 == 0) {
        const int nv = xn / kPer16;
        const int4 *src = reinterpret_cast<const int4 *>(a.x + x0);  // x0 * sizeof(ValT) is a multiple of 16
        int4 *dst = reinterpret_cast<int4 *>(xs);
        for (int i = tid; i < nv; i += kLongBlockThreads) dst[i] = __ldg(src + i);
        for (int i = nv * kPer16 + tid; i < xn; i += kLongBlockThreads) xs[i] = a.x[x0 + i];
    } else {
        for (int i = tid; i < xn; i += kLongBlockThreads) xs[i] = a.x[x0 + i];
    }
    __syncthreads();

    const ValT *xrel = xs - x0;  // xrel[col] is x[col] for the columns of this block
    constexpr int kUnroll = B200SP_SPMV_LONG_BLOCK_UNROLL;  // quads in flight per lane
    constexpr int kPiecesPerCta = kLongBlockThreads / kPieceLanes;
    const int pl = tid & (kPieceLanes - 1);
    const int piece = tid / kPieceLanes;
    const int stride = a.groups * kPiecesPerCta;
    const int first = g * kPiecesPerCta + piece;
    const int trips = nLong > g * kPiecesPerCta ? (nLong - g * kPiecesPerCta + stride - 1) / stride : 0;  // CTA-uniform
    // piece bounds are fetched one trip ahead so that a trip starts with its loads, not a wait
    auto loadBounds = [&](int slot, int &s, int &e) {
        s = 0;
        e = 0;
        if (slot < nLong) {
            const int32_t *seg = a.segStart + (long long)slot * (a.xBlocks + 1) + b;
            s = seg[0];
            e = seg[1];
        }
    };
    int sCur, eCur, sNext, eNext;
    loadBounds(first, sCur, eCur);
    for (int it = 0; it < trips; ++it) {
        const int slot = first + it * stride;
        loadBounds(slot + stride, sNext, eNext);
        const int s = sCur, e = eCur;
        CompT sum = CompT(0);
        if (e > s) {
            if (kVec) {
                // whole aligned quads [vs, ve) in the middle, up to three single entries at either end;
                // the single entries are requested first and used last
                const int vs = (s + 3) >> 2;
                const int ve = e >> 2;
                const int headEnd = 4 * vs < e ? 4 * vs : e;
                const int ph = s + pl;
                const int pt = 4 * ve + pl;
                const bool doHead = pl < 4 && ph < headEnd;
                const bool doTail = pl < 4 && ve >= vs && pt < e;
                const int ch = doHead ? a.colInd[ph] : x0, ct = doTail ? a.colInd[pt] : x0;
                const ValT vh = doHead ? a.val[ph] : ValT(0), vt = doTail ? a.val[pt] : ValT(0);
                for (int v = vs + pl; v < ve; v += kUnroll * kPieceLanes) {
                    int4 c[kUnroll];
                    Quad<ValT> q[kUnroll];
#pragma unroll
                    for (int u = 0; u < kUnroll; ++u) {
                        const int vv = v + kPieceLanes * u;
                        if (vv < ve) {
                            c[u] = __ldcs(reinterpret_cast<const int4 *>(a.colInd) + vv);
                            q[u] = LoadQuad(a.val + 4 * vv);
                        } else {
                            c[u] = make_int4(x0, x0, x0, x0);
#pragma unroll
                            for (int k = 0; k < 4; ++k) q[u].v[k] = ValT(0);
                        }
                    }
                    // Where a lane has no entry both factors are 0: x[x0] may be an infinity or a NaN.  (Selected, not
                    // branched over: the power-law product takes 1.3 % longer with branches.)
#pragma unroll
                    for (int u = 0; u < kUnroll; ++u) {
                        const bool in = v + kPieceLanes * u < ve;
                        const ValT xv[4] = {xrel[c[u].x], xrel[c[u].y], xrel[c[u].z], xrel[c[u].w]};
#pragma unroll
                        for (int k = 0; k < 4; ++k) sum += Widen<CompT>(q[u].v[k]) * Widen<CompT>(in ? xv[k] : ValT(0));
                    }
                }
                const ValT xh = xrel[ch], xt = xrel[ct];
                sum += Widen<CompT>(vh) * Widen<CompT>(doHead ? xh : ValT(0)) + Widen<CompT>(vt) * Widen<CompT>(doTail ? xt : ValT(0));
            } else {
                for (int p = s + pl; p < e; p += kPieceLanes)
                    sum += Widen<CompT>(a.val[p]) * Widen<CompT>(xrel[a.colInd[p]]);
            }
        }
        sCur = sNext;
        eCur = eNext;
        sum = GroupSum(sum, kPieceLanes < 32 ? kPieceLanes : 32);
        if constexpr (kPieceLanes > 32) {  // the piece's warps, in order
            __shared__ CompT sWarp[kLongBlockThreads / 32];
            if ((tid & 31) == 0) sWarp[tid >> 5] = sum;
            __syncthreads();
            if (pl == 0) {
#pragma unroll
                for (int w = 1; w < kPieceLanes / 32; ++w) sum += sWarp[(tid >> 5) + w];
            }
            __syncthreads();
        }
        if (pl == 0 && slot < nLong) a.partials[(long long)slot * a.xBlocks + b] = sum;
    }

    // The CTAs (0..xBlocks-1, g) share the rows of group g: the last of them to get here adds
    // each row's partial sums in block order and writes y.
    __shared__ int sLast;
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const int old = atomicAdd(a.counters + g, 1);
        sLast = (old == a.xBlocks - 1);
        if (sLast) a.counters[g] = 0;  // ready for the next launch
    }
    __syncthreads();
    if (!sLast) return;
    __threadfence();
    const CompT alpha = a.sc.Alpha();
    const CompT beta = a.sc.Beta();
    for (int i = tid; i < trips * kPiecesPerCta; i += kLongBlockThreads) {
        const int slot = g * kPiecesPerCta + (i % kPiecesPerCta) + (i / kPiecesPerCta) * stride;
        if (slot >= nLong) continue;
        CompT total = CompT(0);
        const CompT *part = a.partials + (long long)slot * a.xBlocks;
        for (int bb = 0; bb < a.xBlocks; bb += 8) {  // eight loads in flight, added in block order
            CompT pv[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) pv[k] = bb + k < a.xBlocks ? __ldcg(part + bb + k) : CompT(0);
#pragma unroll
            for (int k = 0; k < 8; ++k) total += pv[k];
        }
        const int r = a.list[slot].x;
        CompT z = alpha * total;
        if (beta != CompT(0)) z += beta * Widen<CompT>(a.y[r]);
        a.y[r] = Narrow<OutT>(z);
    }
}

// The three bins as device functions of a block index `bid`.  (One fused grid with a role per
// block range was measured: no faster than three kernels on forked streams on the power-law
// matrix, 6-12 % slower on the banded one, so each bin is a kernel of its own.)
template <typename CompT, typename ValT, typename OutT, int G>
__device__ __forceinline__ void ShortRowsBody(unsigned bid, const int32_t *__restrict__ rowPtr,
                                              const int32_t *__restrict__ colInd, const ValT *__restrict__ val,
                                              const ValT *__restrict__ x, OutT *__restrict__ y, int rows,
                                              const Scalars<CompT> &sc)
{
    const int lane = threadIdx.x & (G - 1);
    const long long r = ((long long)bid * blockDim.x + threadIdx.x) / G;
    int s = 0, e = 0;
    if (r < rows) {
        s = rowPtr[r];
        e = rowPtr[r + 1];
    }
    const bool mine = r < rows && e - s <= kShortMax;  // longer rows belong to the other kernels
    if (!mine) e = s;
    const CompT beta = sc.Beta();
    CompT yOld = CompT(0);
    if (mine && lane == 0 && beta != CompT(0)) yOld = Widen<CompT>(y[r]);  // requested now, used at the end
    CompT sum = CompT(0);
    // up to four entries per lane in flight
    for (int p = s + lane; p < e; p += 4 * G) {
        int c[4];
        ValT v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool in = p + u * G < e;
            c[u] = in ? __ldcs(colInd + p + u * G) : 0;
            v[u] = in ? __ldcs(val + p + u * G) : ValT(0);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const ValT xv = p + u * G < e ? __ldg(x + c[u]) : ValT(0);
            sum += Widen<CompT>(v[u]) * Widen<CompT>(xv);
        }
    }
    sum = GroupSum(sum, G);
    if (mine && lane == 0) {
        CompT z = sc.Alpha() * sum;
        if (beta != CompT(0)) z += beta * yOld;
        y[r] = Narrow<OutT>(z);
    }
}

template <typename CompT, typename ValT, typename OutT>
__device__ __forceinline__ void MediumRowsBody(unsigned bid, const int32_t *__restrict__ colInd,
                                               const ValT *__restrict__ val, const ValT *__restrict__ x,
                                               OutT *__restrict__ y, const int4 *__restrict__ list, int count,
                                               const Scalars<CompT> &sc)
{
    const int lane = threadIdx.x & 31;
    const int i = (int)bid * (int)(blockDim.x >> 5) + (threadIdx.x >> 5);
    if (i >= count) return;  // whole warps leave together
    const int4 ent = __ldg(list + i);
    const int r = ent.x, s = ent.y, e = ent.z;
    const CompT beta = sc.Beta();
    CompT yOld = CompT(0);
    if (lane == 0 && beta != CompT(0)) yOld = Widen<CompT>(y[r]);  // requested now, used at the end
    CompT sum = CompT(0);
    for (int p = s + lane; p < e; p += 4 * 32) {
        int c[4];
        ValT v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool in = p + u * 32 < e;
            c[u] = in ? __ldcs(colInd + p + u * 32) : 0;
            v[u] = in ? __ldcs(val + p + u * 32) : ValT(0);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const ValT xv = p + u * 32 < e ? __ldg(x + c[u]) : ValT(0);
            sum += Widen<CompT>(v[u]) * Widen<CompT>(xv);
        }
    }
    sum = GroupSum(sum, 32);
    if (lane == 0) {
        CompT z = sc.Alpha() * sum;
        if (beta != CompT(0)) z += beta * yOld;
        y[r] = Narrow<OutT>(z);
    }
}

// Rows of one length or nearly so, none above kShortMax (stencils, banded matrices, k-nearest-neighbour graphs): a CTA copies the
// col_ind and values of its 128 consecutive rows into shared memory (cp.async, 16 bytes at a time, whatever the
// rows' alignment) and gives every row a thread.  The lanes of a warp then walk neighbouring rows in step, so that their
// gathers of x fall into neighbouring elements, and an entry costs five instructions instead of a dozen.
// Measured on the 128^3 stencil (27 entries per row, fp16): 91 us with four lanes per row, 69 us so (5.1 TB/s).  Only for
// rows that lie near their neighbours (BinHeader::nearPairs): with random columns the few warps that this much shared
// memory leaves room for lose to the many of the lane groups (231,721 rows of 19: 40 against 23 us).
constexpr int kStageRows = 128;  // 64 and 256 take the same time
template <typename CompT, typename ValT, typename OutT>
__global__ void __launch_bounds__(kStageRows) SpmvStagedRowsKernel(const int32_t *__restrict__ rowPtr,
                                                                   const int32_t *__restrict__ colInd,
                                                                   const ValT *__restrict__ val, const ValT *__restrict__ x,
                                                                   OutT *__restrict__ y, int rows, int nnz, int stageBytes, Scalars<CompT> sc)
{
    extern __shared__ __align__(16) unsigned char sRaw[];
    const int tid = threadIdx.x;
    b200sp::WaitForPrevious();
    const long long r0 = (long long)blockIdx.x * kStageRows;
    const int last = rows - r0 < kStageRows ? (int)(rows - r0) : kStageRows;
    const int s0 = __ldg(rowPtr + r0), e0 = __ldg(rowPtr + r0 + last);
    constexpr int kPer16 = 16 / (int)sizeof(ValT);
    const int cBase = s0 & ~3, vBase = s0 & ~(kPer16 - 1);  // first entries of the copies
    int32_t *sCol = reinterpret_cast<int32_t *>(sRaw);
    ValT *sVal = reinterpret_cast<ValT *>(sRaw + stageBytes);
    auto copy16 = [](void *dst, const void *src, int bytes) {  // `bytes` of them are read
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes)
                     : "memory");
    };
    for (int i = cBase + 4 * tid; i < e0; i += 4 * kStageRows)
        copy16(sCol + (i - cBase), colInd + i, nnz - i < 4 ? 4 * (nnz - i) : 16);
    for (int i = vBase + kPer16 * tid; i < e0; i += kPer16 * kStageRows)
        copy16(sVal + (i - vBase), val + i, nnz - i < kPer16 ? (int)sizeof(ValT) * (nnz - i) : 16);
    const long long r = r0 + tid;
    int s = 0, e = 0;
    CompT yOld = CompT(0);
    const CompT beta = sc.Beta();
    if (r < rows) {
        s = __ldg(rowPtr + r);
        e = __ldg(rowPtr + r + 1);
        if (beta != CompT(0)) yOld = Widen<CompT>(y[r]);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    CompT sum = CompT(0);
    const int32_t *c = sCol + (s - cBase);
    const ValT *v = sVal + (s - vBase);
    const int len = e - s;
    int i = 0;
    for (; i + 8 <= len; i += 8) {
        ValT xv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) xv[u] = __ldg(x + c[i + u]);
#pragma unroll
        for (int u = 0; u < 8; ++u) sum += Widen<CompT>(v[i + u]) * Widen<CompT>(xv[u]);
    }
    for (; i < len; ++i) sum += Widen<CompT>(v[i]) * Widen<CompT>(__ldg(x + c[i]));
    if (r < rows) {
        CompT z = sc.Alpha() * sum;
        if (beta != CompT(0)) z += beta * yOld;
        y[r] = Narrow<OutT>(z);
    }
}

struct LongSegs {             // the long rows cut into segments (see SpmvCutSegmentsKernel)
    const int4 *segs;         // {row, start, end, slot}
    const int4 *list;         // {row, row start, row end, 0} per slot
    const int2 *rowSeg;       // {first partial slot, segments} per slot
    int32_t *counters;        // arrivals per slot
    void *partials;           // one compute-type value per segment
};

template <typename CompT, typename ValT, typename OutT, bool kVec, int kUnrollQ = kLongUnroll>
__device__ __forceinline__ void LongRowBody(unsigned bid, const int32_t *__restrict__ colInd,
                                            const ValT *__restrict__ val, const ValT *__restrict__ x,
                                            OutT *__restrict__ y, const LongSegs &ls, const Scalars<CompT> &sc,
                                            CompT *sWarp)
{
    const int tid = threadIdx.x;
    const int4 ent = __ldg(ls.segs + bid);
    const int r = ent.x, s = ent.y, e = ent.z, slot = ent.w;
    const int2 rs = __ldg(ls.rowSeg + slot);  // {first partial slot, segments of this row}
    const CompT beta = sc.Beta();
    CompT yOld = CompT(0);
    if (tid == 0 && rs.y == 1 && beta != CompT(0)) yOld = Widen<CompT>(y[r]);  // requested now, used at the end
    CompT sum = CompT(0);
    if (kVec) {
        // whole aligned quads [vs, ve); up to three single entries before and after them
        const int vs = (s + 3) >> 2, ve = e >> 2;
        const int headEnd = 4 * vs < e ? 4 * vs : e;
        const int ph = s + tid, pt = 4 * ve + (tid - 4);
        const bool doHead = tid < 4 && ph < headEnd;
        const bool doTail = tid >= 4 && tid < 8 && ve >= vs && pt < e;
        const int pe = doHead ? ph : pt;
        const int ce = (doHead || doTail) ? colInd[pe] : 0;
        const ValT vE = (doHead || doTail) ? val[pe] : ValT(0);
        for (int v = vs + tid; v < ve; v += kUnrollQ * 256) {
            int4 c[kUnrollQ];
            Quad<ValT> q[kUnrollQ];
#pragma unroll
            for (int u = 0; u < kUnrollQ; ++u) {
                const int vv = v + 256 * u;
                if (vv < ve) {
                    c[u] = __ldcs(reinterpret_cast<const int4 *>(colInd) + vv);
                    q[u] = LoadQuad(val + 4 * vv);
                } else {
                    c[u] = make_int4(0, 0, 0, 0);
#pragma unroll
                    for (int k = 0; k < 4; ++k) q[u].v[k] = ValT(0);
                }
            }
#pragma unroll
            for (int u = 0; u < kUnrollQ; ++u) {
                if (v + 256 * u < ve) {
                    sum += Widen<CompT>(q[u].v[0]) * Widen<CompT>(__ldg(x + c[u].x));
                    sum += Widen<CompT>(q[u].v[1]) * Widen<CompT>(__ldg(x + c[u].y));
                    sum += Widen<CompT>(q[u].v[2]) * Widen<CompT>(__ldg(x + c[u].z));
                    sum += Widen<CompT>(q[u].v[3]) * Widen<CompT>(__ldg(x + c[u].w));
                }
            }
        }
        if (doHead || doTail) sum += Widen<CompT>(vE) * Widen<CompT>(__ldg(x + ce));
    } else {
        for (int p = s + tid; p < e; p += 256) sum += Widen<CompT>(val[p]) * Widen<CompT>(__ldg(x + colInd[p]));
    }
    sum = GroupSum(sum, 32);
    if ((tid & 31) == 0) sWarp[tid >> 5] = sum;
    __syncthreads();
    if (tid == 0) {
        CompT tot = CompT(0);
#pragma unroll
        for (int w = 0; w < 8; ++w) tot += sWarp[w];
        if (rs.y > 1) {
            // one of several segments: leave the partial sum, and finish the row if this CTA is the last to arrive
            CompT *part = static_cast<CompT *>(ls.partials) + rs.x;
            const int rowStart = __ldg(ls.list + slot).y;
            part[(s - rowStart) / kSegLen] = tot;
            __threadfence();
            const int old = atomicAdd(ls.counters + slot, 1);
            if (old != rs.y - 1) return;
            ls.counters[slot] = 0;  // ready for the next launch
            __threadfence();
            tot = CompT(0);
            for (int k = 0; k < rs.y; ++k) tot += __ldcg(part + k);  // segment order: the sum does not depend on timing
            if (beta != CompT(0)) yOld = Widen<CompT>(y[r]);
        }
        CompT z = sc.Alpha() * tot;
        if (beta != CompT(0)) z += beta * yOld;
        y[r] = Narrow<OutT>(z);
    }
}

template <typename CompT, typename ValT, typename OutT, int G>
__global__ void __launch_bounds__(256) SpmvShortRowsKernel(const int32_t *__restrict__ rowPtr,
                                                            const int32_t *__restrict__ colInd,
                                                            const ValT *__restrict__ val,
                                                            const ValT *__restrict__ x, OutT *__restrict__ y,
                                                            int rows, Scalars<CompT> sc)
{
    b200sp::WaitForPrevious();
    ShortRowsBody<CompT, ValT, OutT, G>(blockIdx.x, rowPtr, colInd, val, x, y, rows, sc);
}

// Medium and short rows in one grid: blocks [0, ceil(nM / 8)) take eight listed medium rows
// each (the longer pieces of work start first), the rest sweep all rows for the short ones.
// One launch instead of two streams: whether two large grids on different streams really
// overlap depends on how the driver maps streams to hardware queues, which a library cannot see.
template <typename CompT, typename ValT, typename OutT, int G>
__global__ void __launch_bounds__(256) SpmvMediumShortKernel(const int32_t *__restrict__ rowPtr,
                                                              const int32_t *__restrict__ colInd,
                                                              const ValT *__restrict__ val,
                                                              const ValT *__restrict__ x, OutT *__restrict__ y,
                                                              const int4 *__restrict__ listM, int nM, int rows,
                                                              Scalars<CompT> sc)
{
    b200sp::WaitForPrevious();
    const unsigned wpc = blockDim.x >> 5;
    const unsigned mediumBlocks = ((unsigned)nM + wpc - 1u) / wpc;
    if (blockIdx.x < mediumBlocks) MediumRowsBody<CompT, ValT, OutT>(blockIdx.x, colInd, val, x, y, listM, nM, sc);
    else ShortRowsBody<CompT, ValT, OutT, G>(blockIdx.x - mediumBlocks, rowPtr, colInd, val, x, y, rows, sc);
}

template <typename CompT, typename ValT, typename OutT, bool kVec>
__global__ void __launch_bounds__(256) SpmvLongListKernel(const int32_t *__restrict__ colInd,
                                                           const ValT *__restrict__ val,
                                                           const ValT *__restrict__ x, OutT *__restrict__ y,
                                                           LongSegs ls, Scalars<CompT> sc)
{
    __shared__ CompT sWarp[8];
    LongRowBody<CompT, ValT, OutT, kVec>(blockIdx.x, colInd, val, x, y, ls, sc, sWarp);
}

// All three bins in one grid, for matrices whose long rows keep a CTA each: blocks [0, nL) take one long
// row, the next ceil(nM / 8) eight medium rows, the rest sweep the short rows.  Blocks are handed out in
// index order, so the longest pieces of work start first.  One launch and no fork / join: on a
// 131,000-row shard the two-stream form spent more time between its kernels than in them.
template <typename CompT, typename ValT, typename OutT, int G, bool kVec>
__global__ void __launch_bounds__(256, 6) SpmvAllBinsKernel(const int32_t *__restrict__ rowPtr,
                                                             const int32_t *__restrict__ colInd,
                                                             const ValT *__restrict__ val, const ValT *__restrict__ x,
                                                             OutT *__restrict__ y, const int4 *__restrict__ listM,
                                                             LongSegs ls, int nM, int nL, int rows,
                                                             Scalars<CompT> sc)
{
    __shared__ CompT sWarp[8];
    b200sp::WaitForPrevious();
    unsigned b = blockIdx.x;
    if (b < (unsigned)nL) {  // nL counts segments here
        LongRowBody<CompT, ValT, OutT, kVec, 2>(b, colInd, val, x, y, ls, sc, sWarp);
        return;
    }
    b -= (unsigned)nL;
    const unsigned mediumBlocks = ((unsigned)nM + 7u) >> 3;
    if (b < mediumBlocks) MediumRowsBody<CompT, ValT, OutT>(b, colInd, val, x, y, listM, nM, sc);
    else ShortRowsBody<CompT, ValT, OutT, G>(b - mediumBlocks, rowPtr, colInd, val, x, y, rows, sc);
}

// ---------------------------------------------------------------- rows without a plan

// A product without an analysed plan: a light kernel over the rows -- no shared memory, no barrier, 64 warps per SM,
// which is what keeps the gathers of x near the one sector per clock and SM that L2 delivers -- and a second one for the
// rows that would hold up a warp, which the first lists.
//   rows of up to kGroupTrips * 4 * G entries   G lanes each, four entries per lane in flight (as ShortRowsBody)
//   up to kListedRow                            the row's whole warp, after its groups are done
//   longer                                      listed in segments of kSegLen entries; a CTA of the second kernel each,
//                                               rows of several segments finished by the last CTA to arrive
// Measured, bf16, 300,007 ragged rows with 7.2 M entries: 36 us (the tile kernel with its table: 57); 33,000 rows: 7 us for
// two launches.  7.2 M gathers at one per clock and SM are 26 us.
constexpr int kGroupTrips = 4;
constexpr int kListedRow = 1024;
// A listed row writes its segments into the slots of the multiples of kListedRow among its entry numbers: it has one at
// least, and enough for its segments, and no other row has them.  So there is no counter that a product would have to find
// at zero, and whatever an earlier product (one cut short, or of another matrix) left in the slots is harmless: the second
// kernel takes an item only if the row offsets bear it out, and then it is what the first kernel wrote there.
struct RowList {              // what the first kernel leaves for the second
    int2 *items;              // {row, segment}; a row's segments are consecutive
    int32_t *counters;        // arrivals, at the first segment of a row
    void *partials;           // one compute-type value per segment
    int slots;
};
inline int64_t RowListItems(int64_t nnz) { return nnz / kListedRow + 1; }
__device__ __forceinline__ int RowListSlot(int start) { return (int)(((unsigned)start + (kListedRow - 1)) / kListedRow); }
inline size_t RowListBytes(int64_t nnz) { return (size_t)RowListItems(nnz) * 16 + 512; }
inline RowList RowListIn(void *scratch, int64_t nnz)
{
    const size_t n = AlignUp((size_t)RowListItems(nnz) * 8, 256);
    char *p = reinterpret_cast<char *>(AlignUp(reinterpret_cast<size_t>(scratch), 8));  // the caller's may start on any word
    return {reinterpret_cast<int2 *>(p), reinterpret_cast<int32_t *>(p + n), p + n + (size_t)RowListItems(nnz) * 4,
            (int)RowListItems(nnz)};
}

// kList false: rows of kLongLen entries and more are somebody else's and not listed.
template <typename CompT, typename ValT, typename OutT, int G, bool kList>
__global__ void __launch_bounds__(128, 16) SpmvRowsKernel(const int32_t *__restrict__ rowPtr, const int32_t *__restrict__ colInd,
                                                          const ValT *__restrict__ val, const ValT *__restrict__ x,
                                                          OutT *__restrict__ y, int rows, Scalars<CompT> sc, RowList list)
{
    constexpr int kGroupMax = kGroupTrips * 4 * G;
    const int lane = threadIdx.x & 31, li = lane & (G - 1);
    b200sp::WaitForPrevious();
    const long long r = ((long long)blockIdx.x * 128 + threadIdx.x) / G;
    int s = 0, e = 0;
    if (r < rows) {
        s = rowPtr[r];
        e = rowPtr[r + 1];
    }
    const CompT beta = sc.Beta();
    const int len = e - s;
    if (kList && len > kListedRow && li == 0) {
        const int n = (len + kSegLen - 1) / kSegLen;
        const int at = RowListSlot(s);
        list.counters[at] = 0;
        for (int k = 0; k < n; ++k) list.items[at + k] = make_int2((int)r, k);
    }
    const bool mine = r < rows && (kList ? len <= kListedRow : len < kLongLen);
    if (!mine) e = s;
    CompT yOld = CompT(0);
    if (mine && li == 0 && beta != CompT(0)) yOld = Widen<CompT>(y[r]);  // requested now, used at the end
    CompT sum = CompT(0);
    if (len <= kGroupMax) {
        for (int p = s + li; p < e; p += 4 * G) {
            int c[4];
            ValT v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool in = p + u * G < e;
                c[u] = in ? __ldcs(colInd + p + u * G) : 0;
                v[u] = in ? __ldcs(val + p + u * G) : ValT(0);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const ValT xv = p + u * G < e ? __ldg(x + c[u]) : ValT(0);
                sum += Widen<CompT>(v[u]) * Widen<CompT>(xv);
            }
        }
    }
    sum = GroupSum(sum, G);
    unsigned wide = __ballot_sync(0xffffffffu, mine && len > kGroupMax && li == 0);
    while (wide != 0) {
        const int owner = __ffs(wide) - 1;
        wide &= wide - 1;
        const int ws = __shfl_sync(0xffffffffu, s, owner), we = __shfl_sync(0xffffffffu, e, owner);
        CompT part = CompT(0);
        for (int p = ws + lane; p < we; p += 4 * 32) {
            int c[4];
            ValT v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool in = p + u * 32 < we;
                c[u] = in ? __ldcs(colInd + p + u * 32) : 0;
                v[u] = in ? __ldcs(val + p + u * 32) : ValT(0);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const ValT xv = p + u * 32 < we ? __ldg(x + c[u]) : ValT(0);
                part += Widen<CompT>(v[u]) * Widen<CompT>(xv);
            }
        }
        part = GroupSum(part, 32);
        if (lane == owner) sum = part;
    }
    if (mine && li == 0) {
        CompT z = sc.Alpha() * sum;
        if (beta != CompT(0)) z += beta * yOld;
        y[r] = Narrow<OutT>(z);
    }
}

// The listed segments.  Every CTA looks through its share of the slots, 256 at a time and strided, so that the segments of
// one row go to different CTAs, and sums what it finds.
template <typename CompT, typename ValT, typename OutT>
__global__ void __launch_bounds__(256) SpmvListedKernel(const int32_t *__restrict__ rowPtr, const int32_t *__restrict__ colInd,
                                                        const ValT *__restrict__ val, const ValT *__restrict__ x,
                                                        OutT *__restrict__ y, int rows, Scalars<CompT> sc, RowList list)
{
    __shared__ CompT sWarp[8];
    __shared__ int2 sItem[256];
    __shared__ int sFound;
    const int tid = threadIdx.x;
    b200sp::WaitForPrevious();
    const CompT beta = sc.Beta();
    for (long long slot0 = blockIdx.x; slot0 < list.slots; slot0 += 256ll * gridDim.x) {
        const long long slot = slot0 + (long long)tid * gridDim.x;
        int2 found = make_int2(0, 0);
        bool mine = false;
        if (slot < list.slots) {
            found = list.items[slot];
            if (found.x >= 0 && found.x < rows && found.y >= 0) {
                const int rowStart = __ldg(rowPtr + found.x), len = __ldg(rowPtr + found.x + 1) - rowStart;
                mine = len > kListedRow && found.y < (len + kSegLen - 1) / kSegLen && RowListSlot(rowStart) + found.y == slot;
            }
        }
        if (tid == 0) sFound = 0;
        if (__syncthreads_or(mine) == 0) continue;
        if (mine) sItem[atomicAdd(&sFound, 1)] = found;
        __syncthreads();
        for (int i = 0; i < sFound; ++i) {
            const int2 item = sItem[i];
            const int rowStart = __ldg(rowPtr + item.x), rowEnd = __ldg(rowPtr + item.x + 1);
            const int s = rowStart + item.y * kSegLen, e = rowEnd - s > kSegLen ? s + kSegLen : rowEnd;
            const int segments = (rowEnd - rowStart + kSegLen - 1) / kSegLen;
            CompT sum = CompT(0);
            for (int p = s + tid; p < e; p += 8 * 256) {
                int c[8];
                ValT v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const bool in = p + u * 256 < e;
                    c[u] = in ? __ldcs(colInd + p + u * 256) : 0;
                    v[u] = in ? __ldcs(val + p + u * 256) : ValT(0);
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const ValT xv = p + u * 256 < e ? __ldg(x + c[u]) : ValT(0);
                    sum += Widen<CompT>(v[u]) * Widen<CompT>(xv);
                }
            }
            sum = GroupSum(sum, 32);
            __syncthreads();  // sWarp may still be read for the segment before
            if ((tid & 31) == 0) sWarp[tid >> 5] = sum;
            __syncthreads();
            if (tid == 0) {
                CompT tot = CompT(0);
#pragma unroll
                for (int w = 0; w < 8; ++w) tot += sWarp[w];
                bool last = true;
                if (segments > 1) {
                    const int first = RowListSlot(rowStart);
                    CompT *part = static_cast<CompT *>(list.partials) + first;
                    part[item.y] = tot;
                    __threadfence();
                    last = atomicAdd(list.counters + first, 1) == segments - 1;
                    if (last) {
                        __threadfence();
                        tot = CompT(0);
                        for (int k = 0; k < segments; ++k) tot += __ldcg(part + k);  // segment order: the sum does not depend on timing
                    }
                }
                if (last) {
                    CompT z = sc.Alpha() * tot;
                    if (beta != CompT(0)) z += beta * Widen<CompT>(y[item.x]);
                    y[item.x] = Narrow<OutT>(z);
                }
            }
        }
        __syncthreads();  // sItem and sFound may be written again
    }
}

// ---------------------------------------------------------------- workspace-free kernel

// G lanes per row (G a power of two <= 32 chosen from nnz / rows), grid-stride over rows.
template <typename CompT, typename ValT, typename OutT>
__global__ void __launch_bounds__(256) SpmvRowGroupKernel(const int32_t *__restrict__ rowPtr,
                                                           const int32_t *__restrict__ colInd,
                                                           const ValT *__restrict__ val,
                                                           const ValT *__restrict__ x, OutT *__restrict__ y,
                                                           int rows, Scalars<CompT> sc, int G)
{
    const CompT alpha = sc.Alpha();
    const CompT beta = sc.Beta();
    const int lane = threadIdx.x & (G - 1);
    const long long groupsTotal = (long long)gridDim.x * blockDim.x / G;
    const long long first = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / G;
    const long long rowsPadded = ((long long)rows + groupsTotal - 1) / groupsTotal * groupsTotal;
    for (long long r = first; r < rowsPadded; r += groupsTotal) {
        CompT sum = CompT(0);
        if (r < rows) {
            const int s = rowPtr[r];
            const int e = rowPtr[r + 1];
            for (int p = s + lane; p < e; p += G)
                sum += Widen<CompT>(__ldcs(val + p)) * Widen<CompT>(__ldg(x + __ldcs(colInd + p)));
        }
        sum = GroupSum(sum, G);
        if (r < rows && lane == 0) {
            CompT z = alpha * sum;
            if (beta != CompT(0)) z += beta * Widen<CompT>(y[r]);
            y[r] = Narrow<OutT>(z);
        }
    }
}

// ---------------------------------------------------------------- transpose kernels

// acc[j] = beta * y[j]  (AccT is the output type itself, or float for 16-bit outputs)
template <typename CompT, typename OutT, typename AccT>
__global__ void SpmvTransScaleKernel(const OutT *y, AccT *acc, int n, Scalars<CompT> sc)  // y may alias acc
{
    b200sp::WaitForPrevious();
    const CompT beta = sc.Beta();
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x)
        acc[j] = (beta == CompT(0)) ? AccT(0) : static_cast<AccT>(beta * Widen<CompT>(y[j]));
}

__global__ void SpmvMaxRowLengthKernel(const int32_t *__restrict__ rowPtr, int rows, int32_t *__restrict__ out)
{
    int best = 0;
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < rows;
         r += (long long)gridDim.x * blockDim.x) {
        const int len = rowPtr[r + 1] - rowPtr[r];
        best = len > best ? len : best;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const int o = __shfl_xor_sync(0xffffffffu, best, off);
        best = o > best ? o : best;
    }
    if ((threadIdx.x & 31) == 0 && best > 0) atomicMax(out, best);
}

// acc[col] += (alpha * x[row]) * a_ij, cut by non-zeros: a warp takes chunks of kTransChunk consecutive entries, whatever
// rows they belong to (a scatter needs no per-row reduction, so a row of 16384 entries is simply spread over 64 warps).  All
// columns and values of a chunk are requested at once.  The rows it touches are read side by side, a lane each: every
// non-empty one marks its first entry in a bitmap in shared memory and leaves alpha * x there, and an entry finds its row
// at the last mark at or before it.  A chunk that spans more than kTransSpan rows (stretches of empty ones) searches the
// offsets for its entries instead, eight of a lane at a time.  Bound by the additions: one request per entry on the
// path from the SM to L2 and one operation there.
// Measured, fp32: 11.5 M entries in 500,009 power-law rows: 72 us with a search of the row offsets per entry, 67 with the rows
// held by the lanes and found by shuffles, 65 so (0.65 of them per clock and SM); 4 M entries in 100,000 rows after 400,000
// rows of one entry: 37 with a lane group per row, 49 held by the lanes, 31 so; a million empty rows inside a chunk: 12 us
// with a search per entry, 8.1 ms when the lanes walked through them, 15 so.
constexpr int kTransChunk = 256;
constexpr int kTransSpan = 1024;
constexpr int kTransWarps = 8;
// The chunks of one warp, from entry c0 on; put(column, term) adds a term.  bits, factor: shared memory of the warp.
template <typename CompT, typename ValT, typename AccT, int kChunk, typename Put>
__device__ __forceinline__ void TransChunks(const int32_t *__restrict__ rowPtr, const int32_t *__restrict__ colInd,
                                            const ValT *__restrict__ val, const ValT *__restrict__ x, int rows, int nnz, long long c0,
                                            int chunksPerWarp, CompT alpha, uint32_t *bits, CompT *factor, Put put)
{
    constexpr int kSteps = kChunk / 32;
    const int lane = threadIdx.x & 31;
    if (c0 >= nnz) return;
    int r0 = b200sp::WarpRowOf(rowPtr, rows, c0, lane);  // a row that starts at or before the chunk's first entry
    for (int chunk = 0; chunk < chunksPerWarp && c0 < nnz; ++chunk, c0 += kChunk) {
        int c[kSteps];
        ValT v[kSteps];
#pragma unroll
        for (int u = 0; u < kSteps; ++u) {
            const long long p = c0 + u * 32 + lane;
            c[u] = p < nnz ? __ldcs(colInd + p) : -1;
            v[u] = p < nnz ? __ldcs(val + p) : ValT(0);
        }
        const int first = (int)c0, last = (int)(c0 + kChunk < nnz ? c0 + kChunk - 1 : nnz - 1);
        auto add = [&](int u, CompT f) {
            if (c[u] >= 0 && f != CompT(0)) put(c[u], static_cast<AccT>(f * Widen<CompT>(v[u])));
        };
        // Bounds of the rows r0 + 32 k + lane; beyond the last row both lie behind every entry.
        int s[4], e[4];
        auto load = [&](int k) {
            const unsigned r = (unsigned)r0 + 32 * k + lane;
            s[k] = r < (unsigned)rows ? __ldg(rowPtr + r) : 0x7fffffff;
            e[k] = r < (unsigned)rows ? __ldg(rowPtr + r + 1) : 0x7fffffff;
        };
        load(0);
        if (r0 < rows - kTransSpan && __ldg(rowPtr + r0 + kTransSpan) <= last) {  // the same in every lane
            const int rEnd = r0 + b200sp::WarpRowOf(rowPtr + r0, rows - r0, last, lane);
            int at[kSteps];  // each entry's row lies in [at, at + left]
#pragma unroll
            for (int u = 0; u < kSteps; ++u) at[u] = r0;
            for (int left = rEnd - r0; left > 0;) {
                const int step = (left + 3) / 4;  // three probes at once: half as many round trips as with one
#pragma unroll
                for (int u = 0; u < kSteps; ++u) {
                    const int entry = u * 32 + lane < last - first ? first + u * 32 + lane : last;
                    int below = 0;
#pragma unroll
                    for (int k = 1; k <= 3; ++k) below += k * step <= rEnd - at[u] && __ldg(rowPtr + at[u] + k * step) <= entry;
                    at[u] += below * step;
                }
                left = step - 1 > left - 3 * step ? step - 1 : left - 3 * step;
            }
#pragma unroll
            for (int u = 0; u < kSteps; ++u) add(u, alpha * Widen<CompT>(__ldg(x + at[u])));
            r0 = rEnd;
            continue;
        }
        if (lane < kSteps) bits[lane] = 0;
        __syncwarp();
        // Returns how many of the 32 rows start at or before the chunk's last entry: a prefix, as starts ascend.
        auto mark = [&](int k) {
            const int from = s[k] > first ? s[k] : first;
            if (s[k] <= last && e[k] > from) {  // holds entries of the chunk
                factor[from - first] = alpha * Widen<CompT>(__ldg(x + r0 + 32 * k + lane));
                atomicOr(bits + ((from - first) >> 5), 1u << ((from - first) & 31));
            }
            return __popc(__ballot_sync(0xffffffffu, s[k] <= last));
        };
        int n = mark(0);
        int end = __shfl_sync(0xffffffffu, e[0], 31);
        for (int rowsRead = 32; end <= last; rowsRead = 128) {  // more rows: four times 32 at a time
            r0 += rowsRead;
#pragma unroll
            for (int k = 0; k < 4; ++k) load(k);
            n = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) n += mark(k);
            end = __shfl_sync(0xffffffffu, e[3], 31);
        }
        r0 += n - 1;  // the last row that starts within the chunk, or before it
        __syncwarp();
        int before = 0;  // the last mark in the words before
#pragma unroll
        for (int u = 0; u < kSteps; ++u) {
            const uint32_t word = bits[u], upTo = word & (0xffffffffu >> (31 - lane));
            add(u, factor[upTo != 0 ? u * 32 + 31 - __clz(upTo) : before]);
            if (word != 0) before = u * 32 + 31 - __clz(word);
        }
        __syncwarp();  // bits and factors may be written again
    }
}

template <typename CompT, typename ValT, typename AccT, int kChunk>
__global__ void __launch_bounds__(32 * kTransWarps, 5) SpmvTransScatterKernel(const int32_t *__restrict__ rowPtr,
                                                                           const int32_t *__restrict__ colInd,
                                                                           const ValT *__restrict__ val, const ValT *__restrict__ x,
                                                                           AccT *__restrict__ acc, int rows, int nnz, int chunksPerWarp,
                                                                           Scalars<CompT> sc)
{
    __shared__ uint32_t sBits[kTransWarps][kChunk / 32];
    __shared__ CompT sFactor[kTransWarps][kChunk];
    b200sp::WaitForPrevious();
    const int warp = threadIdx.x >> 5;
    const long long c0 = ((long long)blockIdx.x * kTransWarps + warp) * chunksPerWarp * kChunk;
    TransChunks<CompT, ValT, AccT, kChunk>(rowPtr, colInd, val, x, rows, nnz, c0, chunksPerWarp, sc.Alpha(), sBits[warp],
                                           sFactor[warp], [&](int c, AccT term) { atomicAdd(acc + c, term); });
}

// Few columns: the additions of all SMs meet at the few lines of y and wait for one another in L2 (15 M entries, fp32, 1000 columns: 1084 us;
// 0.05 of them per clock and SM).  A CTA per SM adds up a y of its own in shared memory instead, and that to y: 49 us, 1.1 per
// clock and SM; 4000 columns 331 and 46, 16,000 193 and 46, 48,000 129 and 52.  (Adding up the parts of 2, 4 or 8 CTAs of a cluster before
// they go to y: the same for 2, 2 to 18 % slower for more, as not all SMs are in a cluster.)
constexpr int kTransBlockWarps = 32;
// Few entries are spread over more CTAs than they would fill, as long as these have no more than so many columns between them to add to y: an address of
// shared memory takes an addition per 26 ns.  85,000 entries, half of them in one column, us straight to y, with full CTAs, spread by 16 K and 64 K
// columns: 30 columns 73, 108, 19 and 19, 395 69, 105, 38 and 20; evenly drawn 21, 14, 7.8 and 7.5, and 17.6, 8.4, 6.9 and 7.1; 30,000 on 30
// columns 28, 107, 12 and 12, evenly 9.8, 15, 7.2 and 7.0; 200,000 on 1000 158, 107, 106 and 43, evenly 19, 8.5, 8.4 and 7.2.
constexpr long long kTransSpread = 64 << 10;
constexpr int kTransBlockCols = 48 << 10;  // what fits beside the warps' marks and factors
template <typename CompT, typename ValT, typename AccT>
__global__ void __launch_bounds__(32 * kTransBlockWarps, 1) SpmvTransBlockKernel(const int32_t *__restrict__ rowPtr,
                                                                                const int32_t *__restrict__ colInd,
                                                                                const ValT *__restrict__ val, const ValT *__restrict__ x,
                                                                                AccT *__restrict__ acc, int rows, int cols, int nnz,
                                                                                int chunksPerWarp, Scalars<CompT> sc)
{
    extern __shared__ __align__(16) unsigned char sRaw[];
    AccT *sY = reinterpret_cast<AccT *>(sRaw);
    __shared__ uint32_t sBits[kTransBlockWarps][kTransChunk / 32];
    __shared__ CompT sFactor[kTransBlockWarps][kTransChunk];
    for (int j = threadIdx.x; j < cols; j += blockDim.x) sY[j] = AccT(0);
    __syncthreads();
    b200sp::WaitForPrevious();
    const int warp = threadIdx.x >> 5;
    const long long c0 = ((long long)warp * gridDim.x + blockIdx.x) * chunksPerWarp * kTransChunk;
    TransChunks<CompT, ValT, AccT, kTransChunk>(rowPtr, colInd, val, x, rows, nnz, c0, chunksPerWarp, sc.Alpha(), sBits[warp],
                                                sFactor[warp], [&](int c, AccT term) {
                                                    if (c < cols) atomicAdd(sY + c, term);
                                                });
    __syncthreads();
    for (int j = threadIdx.x; j < cols; j += blockDim.x) {
        const AccT sum = sY[j];
        if (sum != AccT(0)) atomicAdd(acc + j, sum);
    }
}

template <typename OutT>
__global__ void SpmvTransNarrowKernel(const float *__restrict__ acc, OutT *__restrict__ y, int n)
{
    b200sp::WaitForPrevious();
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x)
        y[j] = Narrow<OutT>(acc[j]);
}

// ---------------------------------------------------------------- host dispatch

template <typename CompT>
Scalars<CompT> MakeScalars(const b200spScalars *s);
template <>
Scalars<float> MakeScalars<float>(const b200spScalars *s)
{
    return {s->alpha_f, s->beta_f, static_cast<const float *>(s->alpha_dev), static_cast<const float *>(s->beta_dev)};
}
template <>
Scalars<int32_t> MakeScalars<int32_t>(const b200spScalars *s)
{
    return {s->alpha_i, s->beta_i, static_cast<const int32_t *>(s->alpha_dev),
            static_cast<const int32_t *>(s->beta_dev)};
}

int GroupWidthFor(int64_t rows, int64_t nnz)
{
#ifdef B200SP_SPMV_FORCE_G
    return B200SP_SPMV_FORCE_G;
#endif
    const int64_t avg = rows > 0 ? nnz / rows : 0;
    int G = 1;
    while (G < 32 && G < avg) G <<= 1;
    return G;
}

// Lanes per row of SpmvRowsKernel, which gives a row of up to 16 times as many entries to them.
int RowsGroup(int64_t rows, int64_t nnz)
{
    const int64_t avg = rows > 0 ? nnz / rows : 0;
    return avg <= 6 ? 2 : avg <= 28 ? 4 : avg <= 64 ? 8 : avg <= 128 ? 16 : 32;
}

// Binned plan in the caller's buffer: header, list of medium rows, list of long rows and, when
// the matrix is narrow enough for the blocked long-row kernel, that kernel's tables.
struct BinLayout {
    int64_t capM, capL, capS;
    int32_t xBlocks;  // column blocks of x; 0 = the blocked long-row kernel is not available
    size_t offHeader, offListM, offListL, offTmpL, offSegStart, offLongCounters, offPartials, offSegs, offRowSeg,
        offSegCounters, offSegPartials, total;
};

inline BinLayout BinLayoutFor(int64_t rows, int64_t cols, int64_t nnz)
{
    BinLayout L;
    const int64_t byNnz = nnz / (kShortMax + 1);
    L.capM = (byNnz < rows ? byNnz : rows) + 1;
    L.capL = nnz / kLongLen + 1;
    const int64_t xb = (cols + kXBlockElems - 1) / kXBlockElems;
    L.xBlocks = (xb >= 1 && xb <= kMaxXBlocks && nnz / kLongLen >= B200SP_SPMV_MIN_LONG_BLOCKED) ? (int32_t)xb : 0;
    L.offHeader = 0;
    L.offListM = 256;
    L.offListL = AlignUp(L.offListM + sizeof(int4) * (size_t)L.capM, 256);
    L.offTmpL = AlignUp(L.offListL + sizeof(int4) * (size_t)L.capL, 256);  // long rows as found, before ordering
    L.offSegStart = AlignUp(L.offTmpL + sizeof(int4) * (size_t)L.capL, 256);
    L.offLongCounters = AlignUp(L.offSegStart + sizeof(int32_t) * (size_t)L.capL * (L.xBlocks > 0 ? L.xBlocks + 1 : 0), 256);
    L.offPartials = AlignUp(L.offLongCounters + sizeof(int32_t) * kMaxLongGroups, 256);
    L.capS = nnz / kSegLen + L.capL;  // a row of len entries has at most len / kSegLen + 1 segments
    L.offSegs = AlignUp(L.offPartials + 4 * (size_t)L.capL * L.xBlocks, 256);
    L.offRowSeg = AlignUp(L.offSegs + sizeof(int4) * (size_t)L.capS, 256);
    L.offSegCounters = AlignUp(L.offRowSeg + sizeof(int2) * (size_t)L.capL, 256);
    L.offSegPartials = AlignUp(L.offSegCounters + sizeof(int32_t) * (size_t)L.capL, 256);
    L.total = AlignUp(L.offSegPartials + 4 * (size_t)L.capS, 256);
    return L;
}

// plan_info layout shared with the host layer (see b200sp_kernels.h)
enum { kInfoKind = 0, kInfoMedium = 1, kInfoLong = 2, kInfoGroup = 3, kInfoXBlocks = 4, kInfoBlockElems = 5, kInfoLongLen = 6,
       kInfoSegments = 7 };
enum { kPlanTiles = 0, kPlanBinned = 1, kPlanBinnedBlocked = 2 };  // blocked: long rows go to SpmvLongBlockKernel

// How SpmvLongBlockKernel shares out the long rows: groups of them, a CTA for each on every block of x (one CTA per SM at
// most: it holds half of the SM's threads and a block of x), and lanes per piece.  With many blocks the groups are
// few and large, and eight lanes per piece keep 128 pieces going; with few blocks a group is a handful of rows, whose pieces are
// long, and more lanes share a piece.  Estimated in us per trip: a fixed part, more where its warps meet, and a round trip to memory per eight entries of
// a lane, for the longest rows in the first trip (they are ordered) and the average in the others.  All that is done before the other rows are,
// which run beside, is early enough: then the fewest lanes, whose CTAs are the fewest.  600,000 power-law rows, us with 8 and 32 lanes: 100,000 columns (4
// blocks) 87 and 55, 250,000 (8) 51 and 53, 1 M (32) 55 and 74; 86,660 rows, 137,378 columns (5), 433 long rows of up to 68,689, 8, 32 and 256 lanes 109, 36
// and 21; 583,532 rows of 38 on 29,971 columns (1), 780 long rows, 173, 65 and 82; 25,544 rows of mean 26, one block: 40 with 8, 10 with 32.  Of 250
// power-law matrices the choice is within 3 % of the best for 238, and at worst 5 % slower than by the number of blocks alone (3.1 times as fast at best).
int LongBlockGroups(int xBlocks, int nLong, int lanes)
{
    int groups = b200sp_sm_count() / xBlocks;
    groups = groups < 1 ? 1 : groups > kMaxLongGroups ? kMaxLongGroups : groups;
    const int slots = kLongBlockThreads / lanes, useful = (nLong + slots - 1) / slots;
    return groups < useful ? groups : useful;
}
int LongBlockLanes(int xBlocks, int nLong, long long nnz, long long longNnz, int longest)
{
    int best = 8;
    double least = 1e30;
    const double others = 4e-6 * (double)(nnz - longNnz);
    for (int lanes : {8, 32, 256}) {
        const int slots = kLongBlockThreads / lanes, groups = LongBlockGroups(xBlocks, nLong, lanes);
        const int trips = ((nLong + groups - 1) / groups + slots - 1) / slots;
        auto trip = [&](double entries) { return (lanes > 32 ? 3.0 : 1.0) + 0.7 * ceil(entries / xBlocks / (8.0 * lanes)); };
        const double cost = std::max(others, trip(longest) + (trips - 1) * trip((double)longNnz / nLong));
        if (cost < least) {
            least = cost;
            best = lanes;
        }
    }
    return best;
}

template <typename CompT, typename ValT, typename OutT, bool kVec, int kPieceLanes>
int LaunchLongBlock(const LongBlockArgs<CompT, ValT, OutT> &la, int blocks, cudaStream_t stream)
{
    constexpr int kSmem = kXBlockElems * (int)sizeof(ValT);
    static bool configured[b200sp::kMaxDevices] = {};  // per device: this instantiation may use kSmem bytes
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= b200sp::kMaxDevices) return (int)cudaErrorInvalidDevice;
    if (!configured[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(SpmvLongBlockKernel<CompT, ValT, OutT, kVec, kPieceLanes>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
        if (e != cudaSuccess) return (int)e;
        configured[dev] = true;
    }
    SpmvLongBlockKernel<CompT, ValT, OutT, kVec, kPieceLanes><<<(unsigned)blocks, kLongBlockThreads, kSmem, stream>>>(la);
    b200sp_note_launches(1);
    return (int)cudaGetLastError();
}

template <typename CompT, typename ValT, typename OutT>
int LaunchBinned(const int32_t *rowPtr, const int32_t *colInd, const ValT *val, const ValT *x, OutT *y, int64_t rows,
                 int64_t cols, int64_t nnz, const Scalars<CompT> &sc, void *plan, const int32_t *info,
                 cudaStream_t stream)
{
    const BinLayout L = BinLayoutFor(rows, cols, nnz);
    char *p = static_cast<char *>(plan);
    const int4 *listM = reinterpret_cast<const int4 *>(p + L.offListM);
    const int4 *listL = reinterpret_cast<const int4 *>(p + L.offListL);
    const int nM = info[kInfoMedium], nL = info[kInfoLong], G = info[kInfoGroup], nS = info[kInfoSegments];
    LongSegs ls;
    ls.segs = reinterpret_cast<const int4 *>(p + L.offSegs);
    ls.list = listL;
    ls.rowSeg = reinterpret_cast<const int2 *>(p + L.offRowSeg);
    ls.counters = reinterpret_cast<int32_t *>(p + L.offSegCounters);
    ls.partials = p + L.offSegPartials;
    const bool vec = (reinterpret_cast<uintptr_t>(colInd) % 16 == 0) &&
                     (reinterpret_cast<uintptr_t>(val) % (4 * sizeof(ValT)) == 0);
#if B200SP_SPMV_FUSE_LIST
    // Only for small products (up to 4 M entries): there the fork / join costs more than it buys.  Larger ones
    // keep two kernels on forked streams -- equal in isolation (36.9 us either way on 7.6 M entries), but four
    // such products pipelined on three streams with their host copies took 329 us fused against 287 us forked.
    if (nL > 0 && nnz <= (4ll << 20) && !(info[kInfoKind] == kPlanBinnedBlocked && L.xBlocks > 0)) {
        const unsigned blocks = (unsigned)nS + (unsigned)((nM + 7) / 8) + (unsigned)((rows * G + 255) / 256);
        b200sp_note_launches(1);
        auto launch = [&]<int GG>() {
            return b200sp::LaunchChained(vec ? SpmvAllBinsKernel<CompT, ValT, OutT, GG, true>
                                             : SpmvAllBinsKernel<CompT, ValT, OutT, GG, false>,
                                         blocks, 256, 0, stream, rowPtr, colInd, val, x, y, listM, ls, nM, nS, (int)rows, sc);
        };
        switch (G) {
            case 2: return (int)launch.template operator()<2>();
            case 8: return (int)launch.template operator()<8>();
            default: return (int)launch.template operator()<4>();
        }
    }
#endif
    // The kernels write disjoint rows of y.  The long rows go first, to a side stream forked from
    // and joined back into the caller's stream; medium and short rows follow in one grid.
    b200sp::SideLanes *lanes = nL > 0 ? b200sp::GetSideLanes() : nullptr;
    cudaStream_t sL = stream;
    if (lanes != nullptr) {
        cudaError_t e = cudaEventRecord(lanes->fork, stream);
        if (e != cudaSuccess) return (int)e;
        sL = lanes->stream[0];
    }
    if (nL > 0) {
        if (lanes != nullptr && cudaStreamWaitEvent(sL, lanes->fork, 0) != cudaSuccess) return (int)cudaGetLastError();
        if (info[kInfoKind] == kPlanBinnedBlocked && L.xBlocks > 0) {
            LongBlockArgs<CompT, ValT, OutT> la;
            la.colInd = colInd;
            la.val = val;
            la.x = x;
            la.y = y;
            la.cols = (int)cols;
            la.sc = sc;
            la.list = listL;
            la.segStart = reinterpret_cast<const int32_t *>(p + L.offSegStart);
            la.counters = reinterpret_cast<int32_t *>(p + L.offLongCounters);
            la.partials = reinterpret_cast<CompT *>(p + L.offPartials);
            la.nLong = nL;
            la.xBlocks = L.xBlocks;
            const int pieceLanes = info[kInfoSegments];
            la.groups = LongBlockGroups(L.xBlocks, nL, pieceLanes);
            auto launchLong = [&]<int kPieceLanes>() {
                return vec ? LaunchLongBlock<CompT, ValT, OutT, true, kPieceLanes>(la, L.xBlocks * la.groups, sL)
                           : LaunchLongBlock<CompT, ValT, OutT, false, kPieceLanes>(la, L.xBlocks * la.groups, sL);
            };
            const int rcL = pieceLanes == 8 ? launchLong.template operator()<8>()
                          : pieceLanes == 32 ? launchLong.template operator()<32>() : launchLong.template operator()<256>();
            if (rcL != 0) return rcL;
        } else {
            if (vec) SpmvLongListKernel<CompT, ValT, OutT, true><<<(unsigned)nS, 256, 0, sL>>>(colInd, val, x, y, ls, sc);
            else SpmvLongListKernel<CompT, ValT, OutT, false><<<(unsigned)nS, 256, 0, sL>>>(colInd, val, x, y, ls, sc);
            b200sp_note_launches(1);
        }
        if (lanes != nullptr) cudaEventRecord(lanes->join[0], sL);
    }
    if (rows > 0) {
        // CTAs of kMsThreads threads: a CTA's slot is recycled when its slowest warp is done, and rows of one
        // CTA differ in length (128 threads: 90.4 us on the power-law matrix, 256: 91.3, 64: 91.8).
        constexpr int kMsThreads = 128;
        constexpr int kWpc = kMsThreads / 32;
        const unsigned shortBlocks = (unsigned)((rows * G + kMsThreads - 1) / kMsThreads);
        auto launch = [&]<int GG>() {
            // Where many rows are medium, a lane group that takes them too beats a warp each (fixed rows of 53 entries,
            // 169,574 of them: 47 us with a warp, 38 with 8 lanes); where they are few (power-law rows, one in seventeen to eight),
            // they start first and the lane groups stay narrow.
            if (nM >= rows / 4)
                return b200sp::LaunchChained(SpmvRowsKernel<CompT, ValT, OutT, GG, false>, (unsigned)((rows * GG + 127) / 128), 128, 0,
                                             stream, rowPtr, colInd, val, x, y, (int)rows, sc, RowList{});
            // every row short and near its neighbours, and enough entries per row for the copies to pay
            if (nM == 0 && nL == 0 && info[kInfoBlockElems] > 0 && vec && reinterpret_cast<uintptr_t>(val) % 16 == 0 && nnz >= 6 * rows) {
                const int entries = kStageRows * info[kInfoBlockElems] + 16;  // and room for the alignment at both ends
                const int stage = 4 * entries;
                const int smem = stage + (int)sizeof(ValT) * entries;
                return b200sp::LaunchChained(SpmvStagedRowsKernel<CompT, ValT, OutT>, (unsigned)((rows + kStageRows - 1) / kStageRows),
                                             kStageRows, smem, stream, rowPtr, colInd, val, x, y, (int)rows, (int)nnz, stage, sc);
            }
            if (nM > 0)
                return b200sp::LaunchChained(SpmvMediumShortKernel<CompT, ValT, OutT, GG>,
                                             (unsigned)((nM + kWpc - 1) / kWpc) + shortBlocks, kMsThreads, 0, stream, rowPtr,
                                             colInd, val, x, y, listM, nM, (int)rows, sc);
            return b200sp::LaunchChained(SpmvShortRowsKernel<CompT, ValT, OutT, GG>, shortBlocks, kMsThreads, 0, stream,
                                         rowPtr, colInd, val, x, y, (int)rows, sc);
        };
        cudaError_t rc = cudaSuccess;
        switch (nM >= rows / 4 ? RowsGroup(rows, nnz) : G) {
            case 16: rc = launch.template operator()<16>(); break;
            case 32: rc = launch.template operator()<32>(); break;
            case 2: rc = launch.template operator()<2>(); break;
            case 8: rc = launch.template operator()<8>(); break;
            default: rc = launch.template operator()<4>(); break;
        }
        if (rc != cudaSuccess) return (int)rc;
        b200sp_note_launches(1);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    if (lanes != nullptr) e = cudaStreamWaitEvent(stream, lanes->join[0], 0);
    return (int)e;
}

template <typename CompT, typename ValT, typename OutT>
int LaunchTyped(const int32_t *rowPtr, const int32_t *colInd, const void *val, const void *x, void *y, int64_t rows,
                int64_t cols, int64_t nnz, const b200spScalars *s, void *plan, const int32_t *info,
                cudaStream_t stream)
{
    const Scalars<CompT> sc = MakeScalars<CompT>(s);
    if (plan != nullptr && info != nullptr && info[kInfoKind] != kPlanTiles)
        return LaunchBinned<CompT, ValT, OutT>(rowPtr, colInd, static_cast<const ValT *>(val),
                                               static_cast<const ValT *>(x), static_cast<OutT *>(y), rows, cols, nnz,
                                               sc, plan, info, stream);
    if (plan != nullptr) {
        const PlanLayout L = LayoutFor(rows, nnz);
        if (L.ntiles == 0) return 0;
        char *p = static_cast<char *>(plan);
        TileArgs<CompT, ValT, OutT> a;
        a.rowPtr = rowPtr;
        a.colInd = colInd;
        a.val = static_cast<const ValT *>(val);
        a.x = static_cast<const ValT *>(x);
        a.y = static_cast<OutT *>(y);
        a.rows = (int)rows;
        a.nnz = (int)nnz;
        a.sc = sc;
        a.tileRow = reinterpret_cast<const int32_t *>(p + L.offTileRow);
        a.counters = reinterpret_cast<int32_t *>(p + L.offCounters);
        a.partHead = reinterpret_cast<CompT *>(p + L.offHead);
        a.partTail = reinterpret_cast<CompT *>(p + L.offTail);
        const bool vec = (reinterpret_cast<uintptr_t>(colInd) % 16 == 0) &&
                         (reinterpret_cast<uintptr_t>(val) % (4 * sizeof(ValT)) == 0);
        b200sp_note_launches(1);
        auto launch = [&]<int kSize>() {
            return (int)b200sp::LaunchChained(vec ? SpmvTileKernel<CompT, ValT, OutT, true, kSize>
                                                  : SpmvTileKernel<CompT, ValT, OutT, false, kSize>,
                                              (unsigned)L.ntiles, TileThreads(kSize), 0, stream, a);
        };
        switch (L.size) {
            case 0: return launch.template operator()<0>();
            case 1: return launch.template operator()<1>();
            default: return launch.template operator()<2>();
        }
    }
    if (rows == 0) return 0;
    const int G = GroupWidthFor(rows, nnz);
    const int64_t wantBlocks = (rows * G + 255) / 256;
    const int64_t maxBlocks = (int64_t)b200sp_sm_count() * 32;
    const unsigned blocks = (unsigned)(wantBlocks < maxBlocks ? wantBlocks : maxBlocks);
    SpmvRowGroupKernel<CompT, ValT, OutT><<<blocks, 256, 0, stream>>>(
        rowPtr, colInd, static_cast<const ValT *>(val), static_cast<const ValT *>(x), static_cast<OutT *>(y),
        (int)rows, sc, G);
    b200sp_note_launches(1);
    return (int)cudaGetLastError();
}

// Whether a y per SM pays: estimates of both times in us, from 49 products of 6000 to 15 M entries on 1000 to 48,000 columns.  Additions to y run
// at some 600 sqrt(columns) per us and all SMs, those to shared memory at 320,000, after the block is cleared and before it is
// added to y.  600,000 entries on 48,000 columns: 9 us and 16 with a y per SM, 3 M 28 and 23; 150,000 on 1000: 14 and 9.
bool TransByBlocks(int64_t cols, int64_t nnz)
{
    if (cols > kTransBlockCols) return false;
    const double direct = 3.5 + (double)nnz / (600.0 * sqrt((double)cols));
    const double blocks = 7.5 + 1.1e-4 * (double)cols + (double)nnz / 320000.0;
    return direct > 1.1 * blocks;
}

template <typename CompT, typename ValT, typename AccT>
cudaError_t LaunchTransBlock(const int32_t *rowPtr, const int32_t *colInd, const ValT *val, const ValT *x, AccT *acc, int rows,
                             int cols, int nnz, const Scalars<CompT> &sc, cudaStream_t stream)
{
    static std::atomic<bool> configured[b200sp::kMaxDevices] = {};  // per device: this instantiation may use a block of shared memory
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= b200sp::kMaxDevices) return cudaErrorInvalidDevice;
    if (!configured[dev].load(std::memory_order_relaxed)) {
        const cudaError_t e = cudaFuncSetAttribute(SpmvTransBlockKernel<CompT, ValT, AccT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   kTransBlockCols * (int)sizeof(AccT));
        if (e != cudaSuccess) return e;
        configured[dev].store(true, std::memory_order_relaxed);
    }
    const long long chunks = ((long long)nnz + kTransChunk - 1) / kTransChunk;
    const long long full = (chunks + kTransBlockWarps - 1) / kTransBlockWarps, apart = kTransSpread / cols;
    const long long ctas = std::min<long long>(b200sp_sm_count(), std::max(full, std::min(chunks, apart)));
    const long long perWarp = (chunks + kTransBlockWarps * ctas - 1) / (kTransBlockWarps * ctas);
    return b200sp::LaunchChained(SpmvTransBlockKernel<CompT, ValT, AccT>, (unsigned)ctas, 32 * kTransBlockWarps,
                                 (size_t)cols * sizeof(AccT), stream, rowPtr, colInd, val, x, acc, rows, cols, nnz, (int)perWarp, sc);
}

template <typename CompT, typename ValT, typename OutT>
int LaunchTransTyped(const int32_t *rowPtr, const int32_t *colInd, const void *val, const void *x, void *y,
                     int64_t rows, int64_t cols, int64_t nnz, const b200spScalars *s, void *scratch,
                     size_t scratchBytes, cudaStream_t stream)
{
    const Scalars<CompT> sc = MakeScalars<CompT>(s);
    if (cols == 0) return 0;
    const int sms = b200sp_sm_count();
    const unsigned eltBlocks = (unsigned)((cols + 255) / 256 < (int64_t)sms * 16 ? (cols + 255) / 256 : sms * 16);
    // Consecutive chunks share a warp (and its first search), as long as every SM gets its 64 warps twice.  Few entries are
    // shared by as many warps as the SMs hold, which then wait for one step's searches and loads instead of eight (2 M rows
    // with 20,000 entries: 40 us with chunks of 256, 8 so).
    const bool small = nnz <= 32ll * 5 * kTransWarps * sms;
    const int chunkLen = small ? 32 : kTransChunk;
    const int64_t chunks = (nnz + chunkLen - 1) / chunkLen;
    const int perWarp = small ? 1 : chunks >= 4 * 128ll * sms ? 4 : chunks >= 2 * 128ll * sms ? 2 : 1;
    const unsigned blocks = (unsigned)((chunks + kTransWarps * perWarp - 1) / (kTransWarps * perWarp));
    const auto *v = static_cast<const ValT *>(val), *xv = static_cast<const ValT *>(x);
    // A 16-bit y accumulates in scratch and is rounded once.
    constexpr bool kNarrowOut = sizeof(OutT) == 2;
    using AccT = std::conditional_t<kNarrowOut, float, OutT>;
    if (kNarrowOut && (scratch == nullptr || scratchBytes < sizeof(float) * (size_t)cols)) return (int)cudaErrorInvalidValue;
    auto *yv = static_cast<OutT *>(y);
    AccT *acc = kNarrowOut ? static_cast<AccT *>(scratch) : reinterpret_cast<AccT *>(yv);
    b200sp_note_launches(1);
    cudaError_t e = b200sp::LaunchChained(SpmvTransScaleKernel<CompT, OutT, AccT>, eltBlocks, 256, 0, stream, (const OutT *)yv, acc,
                                          (int)cols, sc);
    if (e == cudaSuccess && rows > 0 && nnz > 0) {
        b200sp_note_launches(1);
        if (TransByBlocks(cols, nnz))
            e = LaunchTransBlock<CompT, ValT, AccT>(rowPtr, colInd, v, xv, acc, (int)rows, (int)cols, (int)nnz, sc, stream);
        else
            e = b200sp::LaunchChained(small ? SpmvTransScatterKernel<CompT, ValT, AccT, 32> : SpmvTransScatterKernel<CompT, ValT, AccT, kTransChunk>,
                                      blocks, 32 * kTransWarps, 0, stream, rowPtr, colInd, v, xv, acc, (int)rows, (int)nnz, perWarp, sc);
    }
    if constexpr (kNarrowOut) {
        if (e == cudaSuccess) {
            b200sp_note_launches(1);
            e = b200sp::LaunchChained(SpmvTransNarrowKernel<OutT>, eltBlocks, 256, 0, stream, (const float *)acc, yv, (int)cols);
        }
    }
    return (int)e;
}

template <typename CompT, typename ValT, typename OutT>
int LaunchRows(const int32_t *rowPtr, const int32_t *colInd, const void *val, const void *x, void *y, int64_t rows, int64_t nnz,
               const b200spScalars *s, void *scratch, cudaStream_t stream)
{
    const Scalars<CompT> sc = MakeScalars<CompT>(s);
    const RowList list = RowListIn(scratch, nnz);
    const auto *v = static_cast<const ValT *>(val), *xv = static_cast<const ValT *>(x);
    auto *yv = static_cast<OutT *>(y);
    if (rows == 0) return 0;
    auto launch = [&]<int G>() {
        b200sp_note_launches(1);
        return b200sp::LaunchChained(SpmvRowsKernel<CompT, ValT, OutT, G, true>, (unsigned)((rows * G + 127) / 128), 128, 0, stream, rowPtr,
                                     colInd, v, xv, yv, (int)rows, sc, list);
    };
    cudaError_t e;
    switch (RowsGroup(rows, nnz)) {
        case 2: e = launch.template operator()<2>(); break;
        case 4: e = launch.template operator()<4>(); break;
        case 8: e = launch.template operator()<8>(); break;
        case 16: e = launch.template operator()<16>(); break;
        default: e = launch.template operator()<32>(); break;
    }
    if (e != cudaSuccess || nnz <= kListedRow) return (int)e;
    const int64_t most = nnz / (kListedRow + 1), cap = (int64_t)b200sp_sm_count() * 4;
    b200sp_note_launches(1);
    return (int)b200sp::LaunchChained(SpmvListedKernel<CompT, ValT, OutT>, (unsigned)(most < 1 ? 1 : most < cap ? most : cap), 256, 0,
                                      stream, rowPtr, colInd, v, xv, yv, (int)rows, sc, list);
}

// Calls f.template operator()<CompT, ValT, OutT>() for a supported type triple, or returns -1.
template <typename F>
int DispatchTypes(int comp, int val, int out, F &&f)
{
    if (comp == B200SP_I32) {
        if (val == B200SP_I32 && out == B200SP_I32) return f.template operator()<int32_t, int32_t, int32_t>();
        return -1;
    }
    if (comp != B200SP_F32) return -1;
    if (val == B200SP_F32 && out == B200SP_F32) return f.template operator()<float, float, float>();
    if (val == B200SP_F16 && out == B200SP_F32) return f.template operator()<float, __half, float>();
    if (val == B200SP_F16 && out == B200SP_F16) return f.template operator()<float, __half, __half>();
    if (val == B200SP_BF16 && out == B200SP_F32) return f.template operator()<float, __nv_bfloat16, float>();
    if (val == B200SP_BF16 && out == B200SP_BF16) return f.template operator()<float, __nv_bfloat16, __nv_bfloat16>();
    if (val == B200SP_I32 && out == B200SP_F32) return f.template operator()<float, int32_t, float>();
    return -1;
}

}  // namespace

extern "C" {

int b200sp_sm_count(void)
{
    // one cached value per device ordinal: the GPUs of a process need not be alike
    static std::atomic<int> cached[b200sp::kMaxDevices] = {};
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    const bool slot = dev >= 0 && dev < b200sp::kMaxDevices;
    if (slot) {
        n = cached[dev].load(std::memory_order_relaxed);
        if (n > 0) return n;
    }
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
    if (slot) cached[dev].store(n, std::memory_order_relaxed);
    return n;
}

size_t b200sp_spmv_tile_plan_bytes(int64_t rows, int64_t nnz) { return LayoutFor(rows, nnz).total; }

size_t b200sp_spmv_plan_bytes(int64_t rows, int64_t cols, int64_t nnz)
{
    const size_t tiles = LayoutFor(rows, nnz).total;
    const size_t bins = BinLayoutFor(rows, cols, nnz).total;
    return tiles > bins ? tiles : bins;  // one buffer serves either plan
}

int b200sp_spmv_analyze(const int32_t *row_ptr, const int32_t *col_ind, int64_t rows, int64_t cols, int64_t nnz,
                        void *plan, size_t plan_bytes, int32_t *plan_info, void *stream)
{
    const size_t need = plan_info == nullptr ? LayoutFor(rows, nnz).total : BinLayoutFor(rows, cols, nnz).total;
    if (plan == nullptr || plan_bytes < need) return (int)cudaErrorInvalidValue;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    char *p = static_cast<char *>(plan);
    if (plan_info == nullptr) {
        // Tile plan: nothing to read back, so nothing synchronises.
        const PlanLayout L = LayoutFor(rows, nnz);
        if (L.ntiles == 0) return 0;
        const unsigned blocks = (unsigned)((L.ntiles + 1 + 7) / 8);
        b200sp_note_launches(1);
        return (int)b200sp::LaunchChained(SpmvTileSearchKernel, blocks, 256, 0, st, row_ptr, (int)rows, (int)nnz,
                                          (int)L.ntiles, TileItems(L.size), reinterpret_cast<int32_t *>(p + L.offTileRow),
                                          reinterpret_cast<int32_t *>(p + L.offCounters));
    }
    // Binned plan: list the medium and the long rows, then read the counts back (one sync).
    const BinLayout L = BinLayoutFor(rows, cols, nnz);
    auto *hdr = reinterpret_cast<BinHeader *>(p + L.offHeader);
    cudaError_t e = cudaMemsetAsync(hdr, 0, 256, st);
    if (e != cudaSuccess) return (int)e;
    const bool blocked = L.xBlocks > 0 && col_ind != nullptr;
    if (blocked) {
        e = cudaMemsetAsync(p + L.offLongCounters, 0, sizeof(int32_t) * kMaxLongGroups, st);
        if (e != cudaSuccess) return (int)e;
    }
    if (rows > 0) {
        const long long want = (rows + 255) / 256;
        const long long cap = (long long)b200sp_sm_count() * 16;
        SpmvBinRowsKernel<<<(unsigned)(want < cap ? want : cap), 256, 0, st>>>(
            row_ptr, col_ind, (int)rows, hdr, reinterpret_cast<int4 *>(p + L.offListM),
            reinterpret_cast<int4 *>(p + L.offTmpL));
        SpmvSortByLengthKernel<<<1, 1024, 0, st>>>(&hdr->longs, reinterpret_cast<const int4 *>(p + L.offTmpL),
                                                   reinterpret_cast<int4 *>(p + L.offListL));
        SpmvCutSegmentsKernel<<<1, 1024, 0, st>>>(hdr, reinterpret_cast<const int4 *>(p + L.offListL),
                                                  reinterpret_cast<int4 *>(p + L.offSegs),
                                                  reinterpret_cast<int2 *>(p + L.offRowSeg),
                                                  reinterpret_cast<int32_t *>(p + L.offSegCounters));
        b200sp_note_launches(3);
        e = cudaGetLastError();
        if (e != cudaSuccess) return (int)e;
    }
    if (blocked && rows > 0) {
        // Cut every long row at the x block boundaries (the count of long rows is still on the device).
        SpmvLongSegmentsKernel<<<(unsigned)(b200sp_sm_count() * 4), 256, 0, st>>>(
            col_ind, hdr, reinterpret_cast<const int4 *>(p + L.offListL),
            reinterpret_cast<int32_t *>(p + L.offSegStart), L.xBlocks);
        b200sp_note_launches(1);
        e = cudaGetLastError();
        if (e != cudaSuccess) return (int)e;
    }
    BinHeader host{};
    e = cudaMemcpyAsync(&host, hdr, sizeof(host), cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess) return (int)e;
    e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return (int)e;
    const double avgShort = host.shortRows > 0 ? (double)host.shortNnz / host.shortRows : 0.0;
    // Staging x costs every one of the xBlocks x groups CTAs the same whatever the number of long rows:
    // on shards of the power-law matrix the blocked kernel won with 2155 long rows (51 vs 70 us) and 4299
    // (95 vs 133 us), lost with 1070 (44 vs 37 us), tied with 517 -- 32 column blocks each time.
    const int minLong = B200SP_SPMV_MIN_LONG_BLOCKED > 48 * L.xBlocks ? B200SP_SPMV_MIN_LONG_BLOCKED : 48 * L.xBlocks;
    const bool useBlocked = blocked && host.unsorted == 0 && host.longs >= minLong;
    plan_info[kInfoKind] = useBlocked ? kPlanBinnedBlocked : kPlanBinned;
    plan_info[kInfoXBlocks] = useBlocked ? L.xBlocks : 0;
    plan_info[kInfoBlockElems] = useBlocked ? kXBlockElems : host.nearPairs * 4ll > host.pairs * 3ll ? host.longestShort : 0;
    plan_info[kInfoLongLen] = kLongLen;
    plan_info[kInfoSegments] = useBlocked ? LongBlockLanes(L.xBlocks, host.longs, nnz, (long long)host.longNnz, host.longestLong) : host.segments;
    plan_info[kInfoMedium] = host.medium;
    plan_info[kInfoLong] = host.longs;
#ifdef B200SP_SPMV_FORCE_SHORT_G
    plan_info[kInfoGroup] = B200SP_SPMV_FORCE_SHORT_G;
#else
    // measured: 27-entry stencil rows run 92 us with 2 or 4 lanes per row, 107 us with 8, 141 us with 16;
    // power-law rows (3.3 entries on average) 96 us with 2 lanes, 115 us with 4
    plan_info[kInfoGroup] = avgShort < 6.0 ? 2 : 4;
#endif
    return 0;
}

int b200sp_spmv_launch(const int32_t *row_ptr, const int32_t *col_ind, const void *val, const void *x, void *y,
                       int64_t rows, int64_t cols, int64_t nnz, const b200spScalars *scalars, int comp_type,
                       int val_type, int out_type, void *plan, const int32_t *plan_info, void *stream)
{
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int rc = DispatchTypes(comp_type, val_type, out_type, [&]<typename C, typename V, typename O>() {
        return LaunchTyped<C, V, O>(row_ptr, col_ind, val, x, y, rows, cols, nnz, scalars, plan, plan_info, st);
    });
    return rc < 0 ? (int)cudaErrorInvalidValue : rc;
}

size_t b200sp_spmv_rows_bytes(int64_t nnz) { return RowListBytes(nnz); }

int b200sp_spmv_rows_launch(const int32_t *row_ptr, const int32_t *col_ind, const void *val, const void *x, void *y, int64_t rows,
                            int64_t nnz, const b200spScalars *scalars, int comp_type, int val_type, int out_type, void *scratch,
                            int32_t *state, void *stream)
{
    (void)state;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int rc = DispatchTypes(comp_type, val_type, out_type, [&]<typename C, typename V, typename O>() {
        return LaunchRows<C, V, O>(row_ptr, col_ind, val, x, y, rows, nnz, scalars, scratch, st);
    });
    return rc < 0 ? (int)cudaErrorInvalidValue : rc;
}

int b200sp_spmv_max_row_length(const int32_t *row_ptr, int64_t rows, void *scratch4, int32_t *max_len, void *stream)
{
    if (max_len == nullptr || scratch4 == nullptr) return (int)cudaErrorInvalidValue;
    *max_len = 0;
    if (rows <= 0) return 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaMemsetAsync(scratch4, 0, sizeof(int32_t), st);
    if (e != cudaSuccess) return (int)e;
    const long long want = (rows + 255) / 256;
    const long long cap = (long long)b200sp_sm_count() * 16;
    SpmvMaxRowLengthKernel<<<(unsigned)(want < cap ? want : cap), 256, 0, st>>>(row_ptr, (int)rows,
                                                                             static_cast<int32_t *>(scratch4));
    b200sp_note_launches(1);
    e = cudaMemcpyAsync(max_len, scratch4, sizeof(int32_t), cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess) return (int)e;
    return (int)cudaStreamSynchronize(st);
}

int b200sp_spmv_trans_launch(const int32_t *row_ptr, const int32_t *col_ind, const void *val, const void *x,
                             void *y, int64_t rows, int64_t cols, int64_t nnz, const b200spScalars *scalars,
                             int comp_type, int val_type, int out_type, void *scratch, size_t scratch_bytes,
                             int by_nnz, void *stream)
{
    (void)by_nnz;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int rc = DispatchTypes(comp_type, val_type, out_type, [&]<typename C, typename V, typename O>() {
        return LaunchTransTyped<C, V, O>(row_ptr, col_ind, val, x, y, rows, cols, nnz, scalars, scratch, scratch_bytes, st);
    });
    return rc < 0 ? (int)cudaErrorInvalidValue : rc;
}

}  // extern "C"

// ---------------------------------------------------------------- entry point without allocation

namespace {

// Scratch for b200sp_spmv_f32_noalloc: the tile table, arrival counters and partial sums that
// b200sp_spmv_analyze would otherwise write into a caller-allocated workspace.  Every GPU that
// loads the library carries this array until the process exits.
constexpr int64_t kNoAllocMaxItems = B200SP_NOALLOC_MAX_ITEMS;
constexpr size_t kNoAllocBytes = 16 * ((size_t)(kNoAllocMaxItems / TileItems(2)) + 2) + 4 * 256;
static __device__ __align__(256) unsigned char gNoAllocScratch[kNoAllocBytes];

constexpr int kMaxDevices = 64;
// Device address of gNoAllocScratch, per device ordinal.  Host threads may race to fill a slot; they all
// store the same address, and the atomic keeps that race defined.
std::atomic<void *> gNoAllocAddr[kMaxDevices] = {};

// In host code `gNoAllocScratch` is only a handle for the runtime, not an address a kernel can
// use; the device address has to be asked for, once per device, with that device current.
int NoAllocScratchAddress(void **out)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= kMaxDevices) return (int)cudaErrorInvalidDevice;
    void *p = gNoAllocAddr[dev].load(std::memory_order_relaxed);
    if (p == nullptr) {
        e = cudaGetSymbolAddress(&p, gNoAllocScratch);
        if (e != cudaSuccess) return (int)e;
        gNoAllocAddr[dev].store(p, std::memory_order_relaxed);
    }
    *out = p;
    return 0;
}

}  // namespace

extern "C" int b200sp_spmv_f32_noalloc(const int32_t *row_ptr, const int32_t *col_ind, const float *val,
                                       const float *x, float *y, int64_t rows, int64_t cols, int64_t nnz,
                                       float alpha, float beta, void *stream)
{
    if (rows < 0 || nnz < 0 || rows > INT32_MAX || nnz > INT32_MAX) return (int)cudaErrorInvalidValue;
    const PlanLayout L = LayoutFor(rows, nnz);
    if (rows + nnz > kNoAllocMaxItems || L.total > kNoAllocBytes) {
        std::fprintf(stderr,
                     "b200sp_spmv_f32_noalloc: rows + nnz = %lld exceeds B200SP_NOALLOC_MAX_ITEMS = %lld; "
                     "use aclsparseSpMV with a caller-provided buffer for a matrix of this size\n",
                     (long long)(rows + nnz), (long long)kNoAllocMaxItems);
        return (int)cudaErrorInvalidValue;
    }
    void *scratch = nullptr;
    const int rc = NoAllocScratchAddress(&scratch);
    if (rc != 0) return rc;
    if (L.ntiles == 0) return 0;
    // The analysis rewrites the tile table and zeroes the arrival counters, so nothing a previous
    // call left in the array is read.
    const int an = b200sp_spmv_analyze(row_ptr, nullptr, rows, cols, nnz, scratch, kNoAllocBytes, nullptr, stream);
    if (an != 0) return an;
    b200spScalars sc{};
    sc.alpha_f = alpha;
    sc.beta_f = beta;
    return LaunchTyped<float, float, float>(row_ptr, col_ind, val, x, y, rows, cols, nnz, &sc, scratch, nullptr,
                                            static_cast<cudaStream_t>(stream));
}
