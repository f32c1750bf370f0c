// CSR SpMM kernels for sm_100a and their extern "C" launchers.
//
// The reference computes one (row, 8-column chunk) per SIMT thread and re-reads the row's
// col_ind / values once per chunk (sparse/spmm/arch35/spmm_kernel.cpp:88-268).  Here a group
// of lanes owns a row: the lanes sit side by side on a row of B, 16 bytes each (so every B
// row is fetched with 128-bit coalesced loads), the row's col_ind / values are read once,
// one per lane, and handed round the group by shuffle.  A group is as wide as a B row needs
// (N * sizeof / 16 lanes, a power of two up to 32), so one warp carries 1 to 32 rows of A.
// Each output keeps one fp32 accumulator that takes its products in CSR order with separate
// multiply and add, exactly as the golden does: for rows of up to 1024 entries the result is
// bit-identical to the golden.
//
// Row-length routing (the analysis pass fills the workspace):
//     ordinary rows                     -> one lane group per row;
//     longer ones (MidRowLimit)         -> a unit each, rows above 1024 non-zeros one per 1024 of them.  The fp kernels
//                                          give a unit a warp per 64 bytes of a B row, which keeps some fifty
//                                          entries in flight and sums them in CSR order all the same (UnitSum); int8
//                                          a CTA.  A row of several units is completed by whichever comes last: it
//                                          adds the stored partial rows in order, so nobody ever waits and the sum
//                                          order is fixed.
// The kernels want contiguous, 16-byte aligned rows of B.  A B in any other layout (column-major, odd N or
// ldb) is first repacked into such rows in the caller's buffer (SpmmRepack*Kernel); a C that is column-major
// or unaligned is written through a shared-memory tile, with the index formulas of the reference
// (spmm_kernel.cpp:156-168, 215-219).  Products whose buffer was not analysed for the layout, or whose B is hardly
// reused, go through a generic one-thread-per-output kernel.
//
// Numerics follow the golden SpmmCpuFp32 / SpmmCpuInt8 (test/spmm/arch35/spmm_test.cpp:
// 125-200): inputs widened to fp32 (int32), products accumulated in fp32 (int32),
// C = alpha*acc + beta*C with C not read when beta == 0; fp16 output is clamped to
// +-65504 before rounding; int32 output is computed in int64 and saturated.
#include <atomic>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include <cuda.h>  // tensor maps: types only
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "b200sp_kernels.h"
#include "../common/chained.cuh"
#include "../common/side_stream.h"

namespace {

#ifndef B200SP_SPMM_THREADS
#define B200SP_SPMM_THREADS 128
#endif
constexpr int kThreads = B200SP_SPMM_THREADS;  // warps of a CTA: one lane-group set each, or one long-row segment
constexpr int kWarps = kThreads / 32;
constexpr int kLongRow = 1024;          // rows longer than this are cut
constexpr int kSegNnz = 1024;           // non-zeros per unit of theirs

inline size_t AlignUp(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct SegEntry {
    int32_t row;
    int32_t seg;      // index of this unit inside its row
    int32_t longIdx;  // index into the long-row table, -1: the unit is the whole row
    int32_t pad;
};
struct LongRow {
    int32_t row;
    int32_t segBase;   // first entry of this row in the segment table
    int32_t nseg;
    int32_t partBase;  // first partial-row slot (rows of two or more segments only)
};

// Column blocking of the long rows (see SpmmLongBlockKernel): B is cut into at most kMaxBlocks blocks of
// consecutive rows, each small enough to stay in L2 while every long row of A sums its entries that fall into it.
constexpr int kMaxBlocks = 64;
#ifndef B200SP_SPMM_BLOCK_MB
#define B200SP_SPMM_BLOCK_MB 32
#endif
constexpr long long kBlockBytes = (long long)B200SP_SPMM_BLOCK_MB << 20;  // target size of one block of B rows
constexpr long long kBlockMinB = 96ll << 20;      // a B smaller than this is left to L2 as a whole
constexpr int kBlockMinRowBytes = 512;            // B rows narrower than a warp of 16-byte pieces keep the segment CTAs
#ifndef B200SP_SPMM_UNIT_NNZ
#define B200SP_SPMM_UNIT_NNZ 256
#endif
constexpr int kUnitNnz = B200SP_SPMM_UNIT_NNZ;   // a (row, block) piece longer than this is cut into several units

// Rows longer than this are summed apart from their neighbours: a lane group has four entries in flight and lets the
// other groups of its warp wait.  Four times the mean leaves rows of like lengths together; where the rows do not fill
// the SMs anyway every row of more than a few entries is better off as a unit.
// 2,759 power-law rows of up to 4,245 entries, bf16, N = 12: 216 us with the limit at 1024, 19 us so; 597,812 rows of
// up to 16,384, N = 16: 694 and 362 us.
inline int MidRowLimit(int64_t rows, int64_t nnz, int64_t n)
{
    if (rows * (n < 16 ? 16 : n) < 148ll * 512) return 16;  // all units (a warp per 16 to 32 columns) resident at once
    const int64_t four = 4 * (nnz / (rows > 0 ? rows : 1));
    return (int)(four < 64 ? 64 : four > kLongRow ? kLongRow : four);
}

struct PlanLayout {
    int64_t capLong, capSegs, capBlockSlots;
    size_t offCounts, offLong, offSegs, offCounters, offPartials;
    size_t offCuts, offRowSlots, offBlockMeta, offUnits, offBlockPartials, total;
};

inline int64_t ArrivalsPerRow(int64_t n) { return (n + 15) / 16; }  // slices of 64 bytes in a B row, at most

inline PlanLayout LayoutFor(int64_t rows, int64_t nnz, int64_t n)
{
    PlanLayout L;
    L.capLong = nnz / (kLongRow + 1) + 1;
    L.capSegs = nnz / kSegNnz + L.capLong + nnz / (MidRowLimit(rows, nnz, n) + 1) + 1;
    L.offCounts = 0;
    L.offLong = 256;
    L.offSegs = AlignUp(L.offLong + sizeof(LongRow) * (size_t)L.capLong, 256);
    L.offCounters = AlignUp(L.offSegs + sizeof(SegEntry) * (size_t)L.capSegs, 256);
    L.offPartials = AlignUp(L.offCounters + sizeof(int32_t) * (size_t)(L.capLong * ArrivalsPerRow(n)), 256);
    // Only rows of two or more segments store partial rows; those have > kSegNnz entries.
    const int64_t capPartialSegs = 2 * (nnz / kSegNnz) + 1;
    L.offCuts = AlignUp(L.offPartials + sizeof(float) * (size_t)capPartialSegs * (size_t)n, 256);
    // Column blocks: a cut table and a {first slot, slots} pair per long row, the unit table and one partial row
    // per unit, up to a budget of one unit per 128 non-zeros (rows of C at least 128 wide only: narrower ones
    // never take that path).
    L.capBlockSlots = n >= 128 ? nnz / 128 + kMaxBlocks : 0;
    const bool on = L.capBlockSlots > 0;
    L.offRowSlots = AlignUp(L.offCuts + (on ? sizeof(int32_t) * (size_t)L.capLong * (kMaxBlocks + 1) : 0), 256);
    L.offBlockMeta = AlignUp(L.offRowSlots + (on ? sizeof(int2) * (size_t)L.capLong : 0), 256);
    L.offUnits = AlignUp(L.offBlockMeta + (on ? sizeof(int32_t) * 3 * kMaxBlocks : 0), 256);
    L.offBlockPartials = AlignUp(L.offUnits + (on ? sizeof(int4) * (size_t)L.capBlockSlots : 0), 256);
    L.total = AlignUp(L.offBlockPartials + sizeof(float) * (size_t)L.capBlockSlots * (size_t)n, 256);
    return L;
}

// ---------------------------------------------------------------- element helpers

template <typename T> __device__ __forceinline__ float ToF32(T v);
template <> __device__ __forceinline__ float ToF32<float>(float v) { return v; }
template <> __device__ __forceinline__ float ToF32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float ToF32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T FromF32(float v);
template <> __device__ __forceinline__ float FromF32<float>(float v) { return v; }
template <> __device__ __forceinline__ __half FromF32<__half>(float v)
{
    // Saturate instead of producing inf (reference spmm_kernel.cpp:232-236).
    v = fminf(fmaxf(v, -65504.0f), 65504.0f);
    return __float2half_rn(v);
}
template <> __device__ __forceinline__ __nv_bfloat16 FromF32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

struct ScalarsF {
    float alpha, beta;
    const float *alphaDev, *betaDev;
    __device__ __forceinline__ float Alpha() const { return alphaDev ? *alphaDev : alpha; }
    __device__ __forceinline__ float Beta() const { return betaDev ? *betaDev : beta; }
};
struct ScalarsI {
    int32_t alpha, beta;
    const int32_t *alphaDev, *betaDev;
    __device__ __forceinline__ int32_t Alpha() const { return alphaDev ? *alphaDev : alpha; }
    __device__ __forceinline__ int32_t Beta() const { return betaDev ? *betaDev : beta; }
};

// How the rows of B are fetched.  B is the operand every row of A gathers from: when it fits in L2 (67 MB at
// 262,144 x 64 fp32) it should stay there while col_ind / values / C stream past it, so its loads carry an
// L2 evict-last policy (per instruction; nothing outlives the launch) and the streams are evict-first.
//   0: plain read-only loads   1: read-only loads with L2::evict_last   2: the same without allocating in L1
#ifndef B200SP_SPMM_B_POLICY
#define B200SP_SPMM_B_POLICY 1
#endif
__device__ __forceinline__ uint4 LoadB16(const void *p)
{
#if B200SP_SPMM_B_POLICY == 0
    return __ldg(reinterpret_cast<const uint4 *>(p));
#else
    uint64_t pol;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));  // hoisted out of loops by the compiler
    uint4 q;
#if B200SP_SPMM_B_POLICY == 1
    asm volatile("ld.global.nc.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w)
                 : "l"(p), "l"(pol));
#else
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w)
                 : "l"(p), "l"(pol));
#endif
    return q;
#endif
}

__device__ __forceinline__ uint32_t LoadB4(const void *p)
{
    uint64_t pol;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    uint32_t q;
    asm volatile("ld.global.nc.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(q) : "l"(p), "l"(pol));
    return q;
}

// What a lane reads of a row of B: 16 bytes side by side, or (kWords: rows that do not start on 16-byte boundaries) four
// words a lane group apart, so that a group still reads consecutive words.  first[] in elements from the row's start.
template <typename ValT, bool kWords> struct Slice {
    static constexpr int kCols = 4 / (int)sizeof(ValT);  // columns of a word (fp types)
    int first[kWords ? 4 : 1];
    __device__ __forceinline__ uint4 Load(const ValT *row) const
    {
        if constexpr (kWords) return make_uint4(LoadB4(row + first[0]), LoadB4(row + first[1]), LoadB4(row + first[2]), LoadB4(row + first[3]));
        else return LoadB16(row + first[0]);
    }
};

// 16 bytes of a B row as fp32 values: 4 floats, or 8 half / bf16.
template <typename T> struct Pack;
template <> struct Pack<float> {
    static constexpr int kElems = 4;
    static __device__ __forceinline__ void Convert(const uint4 &q, float (&out)[4])
    {
        out[0] = __uint_as_float(q.x); out[1] = __uint_as_float(q.y);
        out[2] = __uint_as_float(q.z); out[3] = __uint_as_float(q.w);
    }
};
template <> struct Pack<__half> {
    static constexpr int kElems = 8;
    static __device__ __forceinline__ void Convert(const uint4 &q, float (&out)[8])
    {
        const __half2 *h = reinterpret_cast<const __half2 *>(&q);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(h[i]);
            out[2 * i] = f.x;
            out[2 * i + 1] = f.y;
        }
    }
};
template <> struct Pack<__nv_bfloat16> {
    static constexpr int kElems = 8;
    static __device__ __forceinline__ void Convert(const uint4 &q, float (&out)[8])
    {
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // bf16 -> fp32 is a 16-bit shift
            out[2 * i] = __uint_as_float(w[i] << 16);
            out[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
};

template <> struct Pack<int8_t> {
    static constexpr int kElems = 16;
};

// What a product of ValT operands accumulates in, and the scalars that go with it.
template <typename ValT> struct Arith {
    using Acc = float;
    using Scalars = ScalarsF;
};
template <> struct Arith<int8_t> {
    using Acc = int32_t;
    using Scalars = ScalarsI;
};

// alpha * acc + beta * old, rounded (or saturated: int64 epilogue, reference spmm_kernel.cpp:251-266) to OutT.
template <typename OutT>
__device__ __forceinline__ OutT Finish(float acc, float alpha, float beta, const OutT *old)
{
    float z = __fmul_rn(alpha, acc);
    if (beta != 0.0f) z = __fadd_rn(z, __fmul_rn(beta, ToF32(*old)));
    return FromF32<OutT>(z);
}
template <typename OutT>
__device__ __forceinline__ OutT Finish(int32_t acc, int32_t alpha, int32_t beta, const OutT *old)
{
    long long wide = (long long)alpha * (long long)acc;
    if (beta != 0) wide += (long long)beta * (long long)*old;
    if (wide > 2147483647LL) wide = 2147483647LL;
    if (wide < -2147483648LL) wide = -2147483648LL;
    return (OutT)wide;
}

// ---------------------------------------------------------------- analysis

__global__ void SpmmFindLongRowsKernel(const int32_t *__restrict__ rowPtr, int rows, int limit, int arrivals, int capSegs, int32_t *counts,
                                       LongRow *longRows, SegEntry *segs, int32_t *counters)
{
    int longest = 0;  // of the ordinary rows
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < rows;
         r += (long long)gridDim.x * blockDim.x) {
        const int len = rowPtr[r + 1] - rowPtr[r];
        if (len <= limit) {
            longest = len > longest ? len : longest;
            continue;
        }
        if (len <= kLongRow) {
            segs[capSegs - 1 - atomicAdd(&counts[5], 1)] = {(int32_t)r, 0, -1, 0};
            continue;
        }
        const int nseg = (len + kSegNnz - 1) / kSegNnz;
        const int li = atomicAdd(&counts[0], 1);
        const int sb = atomicAdd(&counts[1], nseg);
        const int pb = atomicAdd(&counts[2], nseg);
        longRows[li] = {(int32_t)r, sb, nseg, pb};
        for (int s = 0; s < arrivals; ++s) counters[(long long)li * arrivals + s] = 0;
        for (int s = 0; s < nseg; ++s) segs[sb + s] = {(int32_t)r, s, li, 0};
    }
    __syncwarp();
    longest = __reduce_max_sync(0xffffffffu, longest);
    if ((threadIdx.x & 31) == 0 && longest > 0) atomicMax(&counts[7], longest);
}

// A warp per long row: checks that its columns ascend, finds where it crosses the boundaries of the column
// blocks (cut[b] = first entry whose column is >= b * blockCols; cut[blocks] = the row's end) and counts the
// units (pieces of at most kUnitNnz entries inside one block) of the row and of every block.
__global__ void __launch_bounds__(256) SpmmCutBlocksKernel(const int32_t *__restrict__ rowPtr,
                                                           const int32_t *__restrict__ colInd,
                                                           const LongRow *__restrict__ longRows, int nLong,
                                                           long long blockCols, int blocks, int32_t *__restrict__ cuts,
                                                           int2 *__restrict__ rowSlots, int32_t *__restrict__ blockUnits,
                                                           int32_t *unsorted)
{
    const int lane = threadIdx.x & 31;
    const int li = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (li >= nLong) return;
    const int row = longRows[li].row;
    const int s = rowPtr[row], e = rowPtr[row + 1];
    bool bad = false;
    for (int p = s + lane; p + 1 < e; p += 32) bad |= colInd[p] > colInd[p + 1];
    if (__any_sync(0xffffffffu, bad)) {
        if (lane == 0) atomicExch(unsorted, 1);
    }
    int32_t *cut = cuts + (long long)li * (kMaxBlocks + 1);
    for (int b = lane; b <= blocks; b += 32) {
        int lo = s, hi = e;
        if (b == blocks) lo = e;
        const long long target = (long long)b * blockCols;
        while (lo < hi) {
            const int mid = lo + ((hi - lo) >> 1);
            if ((long long)colInd[mid] < target) lo = mid + 1;
            else hi = mid;
        }
        cut[b] = lo;
    }
    __syncwarp();
    int units = 0;
    for (int b = lane; b < blocks; b += 32) {
        const int len = cut[b + 1] - cut[b];
        const int u = len > 0 ? (len + kUnitNnz - 1) / kUnitNnz : 0;  // garbage-in (unsorted) can make len negative
        if (u > 0) atomicAdd(blockUnits + b, u);
        units += u;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) units += __shfl_xor_sync(0xffffffffu, units, off);
    if (lane == 0) rowSlots[li] = make_int2(0, units);
}

// One CTA: first slot of every long row (exclusive scan of the rows' unit counts, in list order) and first unit
// of every block; the total goes to *total.
__global__ void __launch_bounds__(1024) SpmmBlockScanKernel(int2 *__restrict__ rowSlots, int nLong,
                                                            int32_t *__restrict__ blockMeta, int blocks, int32_t *total)
{
    __shared__ int sWarp[32];
    __shared__ int sCarry;
    if (threadIdx.x == 0) sCarry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int base = 0; base < nLong; base += 1024) {
        const int i = base + threadIdx.x;
        const int n = i < nLong ? rowSlots[i].y : 0;
        int incl = n;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += t;
        }
        if (lane == 31) sWarp[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            int w = sWarp[lane];
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, w, off);
                if (lane >= off) w += t;
            }
            sWarp[lane] = w;  // inclusive over warps
        }
        __syncthreads();
        const int before = sCarry + (warp > 0 ? sWarp[warp - 1] : 0) + incl - n;
        if (i < nLong) rowSlots[i].x = before;
        __syncthreads();
        if (threadIdx.x == 1023) sCarry = before + n;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        int run = 0;
        for (int b = 0; b < blocks; ++b) {  // blockMeta: [0..64) units of the block, [64..128) first unit, [128..192) filled
            blockMeta[kMaxBlocks + b] = run;
            blockMeta[2 * kMaxBlocks + b] = 0;
            run += blockMeta[b];
        }
        *total = sCarry;
    }
}

struct BlockUnit {
    int32_t start, end;  // entries of the row inside one column block
    int32_t longIdx;
    int32_t slot;        // partial row this unit writes
};

// A warp per long row: writes the row's units into the table, block by block (the table is ordered by block; the
// order inside a block is whatever the atomics give, the slot of a unit is fixed by its place in the row).
__global__ void __launch_bounds__(256) SpmmFillUnitsKernel(const int32_t *__restrict__ cuts, const int2 *__restrict__ rowSlots,
                                                           int nLong, int blocks, int32_t *__restrict__ blockMeta,
                                                           BlockUnit *__restrict__ units, int capUnits)
{
    const int lane = threadIdx.x & 31;
    const int li = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (li >= nLong) return;
    const int32_t *cut = cuts + (long long)li * (kMaxBlocks + 1);
    int slot = rowSlots[li].x;
    for (int b = 0; b < blocks; ++b) {
        const int s = cut[b], e = cut[b + 1];
        const int n = e > s ? (e - s + kUnitNnz - 1) / kUnitNnz : 0;
        if (n == 0) continue;
        int pos = 0;
        if (lane == 0) pos = blockMeta[kMaxBlocks + b] + atomicAdd(blockMeta + 2 * kMaxBlocks + b, n);
        pos = __shfl_sync(0xffffffffu, pos, 0);
        for (int i = lane; i < n; i += 32) {
            const int us = s + i * kUnitNnz;
            if (pos + i < capUnits)
                units[pos + i] = {us, us + kUnitNnz < e ? us + kUnitNnz : e, li, slot + i};
        }
        slot += n;
    }
}

// ---------------------------------------------------------------- fast path

template <typename ValT, typename OutT>
struct FastArgs {
    const int32_t *rowPtr;
    const int32_t *colInd;
    const ValT *val;
    const ValT *B;
    OutT *C;
    int m;
    int n;
    int nB;               // columns of a row of B as laid out: n, padded to whole 16-byte pieces when repacked
    long long ldb;
    long long ldc;        // element (r, j) of C lies at r * ldc + j, or (kGenC) at r * cRow + j * cCol
    long long cRow, cCol;
    unsigned long long negZeros;
    typename Arith<ValT>::Scalars sc;
    int rowLimit;         // longer rows are units
    int longUnits;        // units of rows above kLongRow, from the front of the table, ...
    int nUnits;           // ... then those of one row each, from its end
    int unitCtas;         // CTAs at the front of the grid that work on them
    int slices;           // fp: warps a unit takes, 64 bytes of a B row each
    int splitRows;        // int8 only: a CTA per row
    int genRows;          // rows of a CTA: column-major C, and int8 as a loop
    const LongRow *longRows;
    const SegEntry *segs, *segsEnd;
    int32_t *counters;    // [long row][ArrivalsPerRow]
    int arrivals;
    void *partials;       // [partial slot][n] of the accumulator's type
};

// Accumulation in the golden's arithmetic: the product is rounded, then added (no fused multiply-add), so a row
// summed in CSR order reproduces the golden bit for bit.  Two of a lane's outputs share an instruction (packed fp32
// of sm_100): 8 instead of 16 per 16-byte piece of a half-precision B row.  The product is an fma with -0, which rounds
// it and keeps its sign, and the -0 comes from the launch (kNegZeros), out of the assembler's sight: it fuses a
// packed mul.rn, or an fma with a constant -0, with the addition that follows.
constexpr unsigned long long kNegZeros = 0x8000000080000000ull;
__device__ __forceinline__ void MulAdd2(float &a0, float &a1, float b0, float b1, float v,
                                        unsigned long long negZeros)
{
    asm("{\n\t.reg .b64 x, y, z;\n\t"
        "mov.b64 x, {%2, %3};\n\t"
        "mov.b64 y, {%4, %4};\n\t"
        "mov.b64 z, {%0, %1};\n\t"
        "fma.rn.f32x2 x, x, y, %5;\n\t"
        "add.rn.f32x2 z, z, x;\n\t"
        "mov.b64 {%0, %1}, z;\n\t}"
        : "+f"(a0), "+f"(a1)
        : "f"(b0), "f"(b1), "f"(v), "l"(negZeros));
}
template <int E>
__device__ __forceinline__ void Accumulate(float v, const float (&b)[E], float (&acc)[E], unsigned long long negZeros)
{
#pragma unroll
    for (int i = 0; i < E; i += 2) MulAdd2(acc[i], acc[i + 1], b[i], b[i + 1], v, negZeros);
}
// Compensated summation, the reference's high-precision algorithm.
__device__ __forceinline__ void AccumulateKahan(float v, float b, float &acc, float &comp)
{
    const float y = __fsub_rn(__fmul_rn(v, b), comp);
    const float t = __fadd_rn(acc, y);
    comp = __fsub_rn(__fsub_rn(t, acc), y);
    acc = t;
}

// Adds sum_{p in [s, e)} val[p] * B[col[p], slice] to acc, p ascending.  The kLanes lanes of a
// group call it together with the same s, e (groups of one warp may differ); `trips` is the
// warp-uniform number of kChunk-wide chunks to walk (>= this group's own need).
#ifndef B200SP_SPMM_BATCH
#define B200SP_SPMM_BATCH 4
#endif
template <int kLanes> struct Chunk {
    static constexpr int kHold = kLanes >= 8 ? 1 : 8 / kLanes;  // entries a lane holds, so that narrow groups have work in flight
    static constexpr int kChunk = kLanes * kHold;
};

template <typename ValT, bool kKahan, int kLanes, bool kWords, bool kOrdered>
__device__ __forceinline__ void RowDot(const int32_t *__restrict__ colInd, const ValT *__restrict__ val,
                                       const ValT *__restrict__ B, const Slice<ValT, kWords> &slice, long long ldb, int s, int e, int trips,
                                       unsigned long long negZeros, float (&acc)[Pack<ValT>::kElems],
                                       float (&comp)[Pack<ValT>::kElems])
{
    constexpr int E = Pack<ValT>::kElems;
    constexpr int kHold = Chunk<kLanes>::kHold;
    constexpr int kChunk = Chunk<kLanes>::kChunk;
    constexpr int kBatch = kChunk < B200SP_SPMM_BATCH ? kChunk : B200SP_SPMM_BATCH;  // B rows in flight per lane
    const int li = threadIdx.x & (kLanes - 1);
    [[maybe_unused]] int nextCol[kHold];
    [[maybe_unused]] ValT nextVal[kHold];
    // rem: entries of the row from p on, <= 0 past its end; p itself may then be past what an int counts
    [[maybe_unused]] auto request = [&](int p, int rem) {
#pragma unroll
        for (int h = 0; h < kHold; ++h) {
            nextCol[h] = 0;
            nextVal[h] = FromF32<ValT>(0.0f);
            if (h * kLanes + li < rem) {
                nextCol[h] = __ldcs(colInd + p + h * kLanes + li);
                nextVal[h] = __ldcs(val + p + h * kLanes + li);
            }
        }
    };
    // The entries of the next chunk are asked for before this one's rows of B.  us without and with: f32, 64 entries a row, N = 64, 262 and 252;
    // f32, N = 16, power-law rows of 100, 172 and 157, ragged rows of 16, 6.6 and 5.9; N = 32, 3000 rows of 60, 9.0 and 8.1.  Not for
    // fp32 rows of eight lanes and more that are taken by length (N = 64, ragged rows of 12, 52 and 56), nor for other widths (f16, N = 8: 53 and
    // 70; bf16, N = 128: 127 and 133; f16 and bf16, N = 32: 52 and 54, 88 and 91).
    constexpr bool kWide = sizeof(ValT) == 4;
    constexpr bool kEarly = (kLanes == 4 && kWide) || (kLanes == 8 && !(kWide && kOrdered)) || (kLanes == 16 && kWide && !kOrdered);
    if constexpr (kEarly)
        if (trips > 0) request(s, e - s);
    for (int chunk = 0; chunk < trips; ++chunk) {
        const int p0 = (int)((unsigned)s + chunk * kChunk);
        const int rem = e - s - chunk * kChunk;  // entries of this group's row left; <= 0 once the row is done
        int myCol[kHold];
        float myVal[kHold];
        if constexpr (kEarly) {
#pragma unroll
            for (int h = 0; h < kHold; ++h) {
                myCol[h] = nextCol[h];
                myVal[h] = ToF32(nextVal[h]);
            }
            if (chunk + 1 < trips) request((int)((unsigned)p0 + kChunk), rem - kChunk);
        } else {
#pragma unroll
            for (int h = 0; h < kHold; ++h) {
                myCol[h] = 0;
                myVal[h] = 0.0f;
                if (h * kLanes + li < rem) {
                    myCol[h] = __ldcs(colInd + p0 + h * kLanes + li);
                    myVal[h] = ToF32(__ldcs(val + p0 + h * kLanes + li));
                }
            }
        }
        // Whole warp on full chunks: straight-line code, no predicate per entry.
        if (__all_sync(0xffffffffu, rem >= kChunk)) {
#pragma unroll
            for (int q0 = 0; q0 < kChunk; q0 += kBatch) {
                uint4 q[kBatch];
                float v[kBatch];
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const int c = __shfl_sync(0xffffffffu, myCol[(q0 + u) / kLanes], (q0 + u) % kLanes, kLanes);
                    v[u] = __shfl_sync(0xffffffffu, myVal[(q0 + u) / kLanes], (q0 + u) % kLanes, kLanes);
                    q[u] = slice.Load(B + (long long)c * ldb);
                }
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    float b[E];
                    Pack<ValT>::Convert(q[u], b);
                    if constexpr (kKahan) {
#pragma unroll
                        for (int i = 0; i < E; ++i) AccumulateKahan(v[u], b[i], acc[i], comp[i]);
                    } else {
                        Accumulate<E>(v[u], b, acc, negZeros);
                    }
                }
            }
            continue;
        }
        // Entries past the end of this group's row count as 0 * 0: adding +0 to a sum that began at +0 changes no
        // bit of it.  (The compensated sum is not indifferent to zeros and skips them.)
#pragma unroll
        for (int q0 = 0; q0 < kChunk; q0 += kBatch) {
            if (!__any_sync(0xffffffffu, q0 < rem)) break;
            uint4 q[kBatch];
            float v[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                const int c = __shfl_sync(0xffffffffu, myCol[(q0 + u) / kLanes], (q0 + u) % kLanes, kLanes);
                v[u] = __shfl_sync(0xffffffffu, myVal[(q0 + u) / kLanes], (q0 + u) % kLanes, kLanes);
                q[u] = make_uint4(0, 0, 0, 0);
                if (q0 + u < rem) q[u] = slice.Load(B + (long long)c * ldb);
            }
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                float b[E];
                Pack<ValT>::Convert(q[u], b);
                if constexpr (kKahan) {
                    if (q0 + u < rem) {
#pragma unroll
                        for (int i = 0; i < E; ++i) AccumulateKahan(v[u], b[i], acc[i], comp[i]);
                    }
                } else {
                    Accumulate<E>(v[u], b, acc, negZeros);
                }
            }
        }
    }
}

// The int8 form: four entries at a time.  A lane holds 16 columns of four rows of B; each 4 x 4 block of bytes is
// transposed (eight byte permutes) so that one __dp4a adds four products: 12 instructions for 16 products instead
// of 32 (16 extractions and 16 multiply-adds).  Entries past a row's end carry value 0 and column 0, which adds
// nothing.  int32 addition wraps the same in any order, so the result is the golden's whatever the grouping.
// Up to four lanes side by side are too few for a row of their own: eight lanes share one, kShare sets of kLanes lanes
// that take every kShare-th entry; their sums are added when the row ends.
template <int kLanes> struct Group8 {
    static constexpr int kLanesOfRow = kLanes < 8 ? 8 : kLanes;
    static constexpr int kShare = kLanesOfRow / kLanes;
    static constexpr int kChunk = kShare > 1 ? 8 * kShare : kLanes;
};

__device__ __forceinline__ void DotQuad(const uint32_t (&x)[4], const uint32_t (&y)[4], const uint32_t (&z)[4], const uint32_t (&t)[4],
                                        int v, int32_t (&acc)[16])
{
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t lo01 = __byte_perm(x[j], y[j], 0x5140), lo23 = __byte_perm(z[j], t[j], 0x5140);
        const uint32_t hi01 = __byte_perm(x[j], y[j], 0x7362), hi23 = __byte_perm(z[j], t[j], 0x7362);
        acc[4 * j] = __dp4a((int)__byte_perm(lo01, lo23, 0x5410), v, acc[4 * j]);
        acc[4 * j + 1] = __dp4a((int)__byte_perm(lo01, lo23, 0x7632), v, acc[4 * j + 1]);
        acc[4 * j + 2] = __dp4a((int)__byte_perm(hi01, hi23, 0x5410), v, acc[4 * j + 2]);
        acc[4 * j + 3] = __dp4a((int)__byte_perm(hi01, hi23, 0x7632), v, acc[4 * j + 3]);
    }
}

template <int kLanes>
__device__ __forceinline__ void RowDot8(const int32_t *__restrict__ colInd, const int8_t *__restrict__ val,
                                        const int8_t *__restrict__ Bslice, long long ldb, int s, int e, int trips,
                                        int32_t (&acc)[16])
{
    using Shape = Group8<kLanes>;
    const int li = threadIdx.x & (Shape::kLanesOfRow - 1);
    for (int chunk = 0; chunk < trips; ++chunk) {
        const int p0 = s + chunk * Shape::kChunk;
        const int rem = e - p0;
        if constexpr (Shape::kShare > 1) {
            auto quadOf = [&](int first, int(&c)[4]) {  // columns and values of four entries of this lane
                int quad = 0;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int i = (first + u) * Shape::kShare + li / kLanes;
                    c[u] = i < rem ? __ldcs(colInd + p0 + i) : 0;
                    if (i < rem) quad |= (int)(unsigned char)__ldcs(reinterpret_cast<const signed char *>(val) + p0 + i) << (8 * u);
                }
                return quad;
            };
            auto rowsOf = [&](const int(&c)[4], uint32_t(&w)[4][4]) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint4 q = LoadB16(Bslice + (long long)c[u] * ldb);
                    w[u][0] = q.x; w[u][1] = q.y; w[u][2] = q.z; w[u][3] = q.w;
                }
            };
            int c0[4], c1[4];
            uint32_t w0[4][4], w1[4][4];
            const int v0 = quadOf(0, c0);
            if (__any_sync(0xffffffffu, rem > 4 * Shape::kShare)) {
                const int v1 = quadOf(4, c1);
                rowsOf(c0, w0);
                rowsOf(c1, w1);
                DotQuad(w0[0], w0[1], w0[2], w0[3], v0, acc);
                DotQuad(w1[0], w1[1], w1[2], w1[3], v1, acc);
            } else {
                rowsOf(c0, w0);
                DotQuad(w0[0], w0[1], w0[2], w0[3], v0, acc);
            }
        } else {
            int myCol = 0, quad = 0;
            if (li < rem) {
                myCol = __ldcs(colInd + p0 + li);
                quad = (int)(unsigned char)__ldcs(reinterpret_cast<const signed char *>(val) + p0 + li);
            }
            quad |= __shfl_down_sync(0xffffffffu, quad, 1, kLanes) << 8;
            quad = (quad & 0xffff) | (__shfl_down_sync(0xffffffffu, quad, 2, kLanes) << 16);  // lanes 0, 4, 8, ...: four values
#pragma unroll
            for (int q0 = 0; q0 < kLanes; q0 += 8) {  // two quads of B rows in flight per lane
                if (!__any_sync(0xffffffffu, q0 < rem)) break;
                uint32_t w[8][4];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int c = __shfl_sync(0xffffffffu, myCol, q0 + u, kLanes);
                    const uint4 q = LoadB16(Bslice + (long long)c * ldb);
                    w[u][0] = q.x; w[u][1] = q.y; w[u][2] = q.z; w[u][3] = q.w;
                }
                DotQuad(w[0], w[1], w[2], w[3], __shfl_sync(0xffffffffu, quad, q0, kLanes), acc);
                DotQuad(w[4], w[5], w[6], w[7], __shfl_sync(0xffffffffu, quad, q0 + 4, kLanes), acc);
            }
        }
    }
}

#ifndef B200SP_SPMM_C_STREAMED
#define B200SP_SPMM_C_STREAMED 1
#endif
#if B200SP_SPMM_C_STREAMED
#define B200SP_SPMM_C_LOAD(p) __ldcs(p)
#define B200SP_SPMM_C_STORE(p, v) __stcs(p, v)
#else
#define B200SP_SPMM_C_LOAD(p) (*(p))
#define B200SP_SPMM_C_STORE(p, v) (*(p) = (v))
#endif
template <typename OutT, int E>
__device__ __forceinline__ void StoreRowSlice(OutT *dst, const float (&acc)[E], float alpha, float beta)
{
    // C is read at most once and written once per product: streamed, so that it does not displace B in L2.
    float z[E];
    if (beta != 0.0f) {
        constexpr int kVecs = E * (int)sizeof(OutT) / 16;
        alignas(16) OutT old[E];
#pragma unroll
        for (int i = 0; i < kVecs; ++i)
            reinterpret_cast<uint4 *>(old)[i] = B200SP_SPMM_C_LOAD(reinterpret_cast<const uint4 *>(dst) + i);
#pragma unroll
        for (int i = 0; i < E; ++i) z[i] = __fadd_rn(__fmul_rn(alpha, acc[i]), __fmul_rn(beta, ToF32(old[i])));
    } else {
#pragma unroll
        for (int i = 0; i < E; ++i) z[i] = __fmul_rn(alpha, acc[i]);
    }
    if constexpr (sizeof(OutT) == 4) {
#pragma unroll
        for (int i = 0; i < E; i += 4)
            B200SP_SPMM_C_STORE(reinterpret_cast<float4 *>(dst + i), make_float4(z[i], z[i + 1], z[i + 2], z[i + 3]));
    } else {
        static_assert(E == 8, "16-bit output slices are 8 wide");
        alignas(16) OutT o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = FromF32<OutT>(z[i]);
        B200SP_SPMM_C_STORE(reinterpret_cast<uint4 *>(dst), *reinterpret_cast<const uint4 *>(o));
    }
}

template <typename OutT>
__device__ __forceinline__ void StoreRowSlice(OutT *dst, const int32_t (&acc)[16], int32_t alpha, int32_t beta)
{
    static_assert(sizeof(OutT) == 4, "int8 products are stored as int32");
#pragma unroll
    for (int i = 0; i < 16; i += 4) {
        alignas(16) int32_t old[4] = {0, 0, 0, 0}, z[4];
        if (beta != 0) *reinterpret_cast<int4 *>(old) = __ldcs(reinterpret_cast<const int4 *>(dst + i));
#pragma unroll
        for (int k = 0; k < 4; ++k) z[k] = Finish<int32_t>(acc[i + k], alpha, beta, old + k);
        __stcs(reinterpret_cast<int4 *>(dst + i), *reinterpret_cast<const int4 *>(z));
    }
}

template <int kBytes> __device__ __forceinline__ void CopyAsync(void *dst, const void *src, bool on)  // zeros where not `on`
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (kBytes == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(on ? 16 : 0) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(on ? 4 : 0) : "memory");
}

// A unit: a row of up to kLongRow entries, or that many of a longer one.  A warp sums kPieces * 16 bytes of the B rows of
// its entries, in CSR order.  What bounds it is the latency of the gathers: they come through shared memory by cp.async,
// kStages rounds in flight, requested by all lanes whatever the number of columns; the columns and values of a round are
// loaded kStages rounds before its request.  Then lane l adds up word l of the B rows, one entry after the other.
// 64 bytes per warp at most: wide rows are shared by more warps, and the shared memory (some 18 KB a CTA) leaves the
// ordinary rows of the same grid their occupancy.
template <int kLanes> struct UnitShape {
    static constexpr int kPieces = kLanes < 4 ? kLanes : 4;
    static constexpr int kRound = kPieces == 4 ? 16 : 32;            // entries per round
    static constexpr int kStages = 4;
    static constexpr int kStageBytes = kRound * kPieces * 16;
    static constexpr int kWarpBytes = kStages * (kStageBytes + kRound * 4);
};

template <typename ValT, typename OutT, bool kKahan, int kLanes, bool kWords>
__device__ void UnitSum(const FastArgs<ValT, OutT> &a, unsigned char *sWarp)
{
    using Shape = UnitShape<kLanes>;
    constexpr int kPieces = Shape::kPieces, kRound = Shape::kRound, kStages = Shape::kStages;
    constexpr int kCols = 4 / (int)sizeof(ValT);  // columns of a word
    constexpr int kCopyBytes = kWords ? 4 : 16;
    constexpr int kPerEntry = kPieces * 16 / kCopyBytes;
    constexpr int kCopies = kRound * kPerEntry / 32;  // of a lane per round
    const int lane = threadIdx.x & 31;
    const long long at = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
    const int unit = (int)(at / a.slices), slice = (int)(at - (long long)unit * a.slices);
    if (unit >= a.nUnits) return;
    const SegEntry seg = unit < a.longUnits ? a.segs[unit] : a.segsEnd[a.longUnits - 1 - unit];
    const int rowEnd = a.rowPtr[seg.row + 1];
    const int s = a.rowPtr[seg.row] + seg.seg * kSegNnz;
    const int length = rowEnd - s > kSegNnz ? kSegNnz : rowEnd - s;
    const int rounds = (length + kRound - 1) / kRound;
    unsigned char *sData = sWarp;                                                                     // [kStages][kStageBytes]
    float *sVal = reinterpret_cast<float *>(sWarp + kStages * Shape::kStageBytes);                    // [kStages][kRound]
    const int first = slice * kPieces * 4 * kCols + (lane & (kPerEntry - 1)) * (kCopyBytes / (int)sizeof(ValT));
    const bool live = first < a.nB;
    const ValT *Bs = a.B + (live ? first : 0);

    struct Batch {  // of kStages rounds; lane l holds entry l of each
        int col[kStages];
        float val[kStages];
    };
    auto load = [&](Batch &b, int round0) {
#pragma unroll
        for (int i = 0; i < kStages; ++i) {
            const int p = (round0 + i) * kRound + lane;
            const bool in = lane < kRound && p < length;
            b.col[i] = in ? __ldcs(a.colInd + s + p) : 0;
            b.val[i] = in ? ToF32(__ldcs(a.val + s + p)) : 0.0f;
        }
    };
    auto request = [&](const Batch &b, int i, int round) {
        if (round < rounds) {
#pragma unroll
            for (int u = 0; u < kCopies; ++u) {
                const int entry = u * (32 / kPerEntry) + lane / kPerEntry;
                const int c = __shfl_sync(0xffffffffu, b.col[i], entry);
                CopyAsync<kCopyBytes>(sData + i * Shape::kStageBytes + (u * 32 + lane) * kCopyBytes, Bs + c * a.ldb,
                                      live && round * kRound + entry < length);
            }
            if (lane < kRound) sVal[i * kRound + lane] = b.val[i];
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    Batch now, next;
    load(now, 0);
    load(next, kStages);
#pragma unroll
    for (int i = 0; i < kStages; ++i) request(now, i, i);
    const int word = lane & (4 * kPieces - 1);  // lanes past the last word repeat others' work
    float acc[kCols] = {}, comp[kCols] = {};
#pragma unroll 1
    for (int r0 = 0; r0 < rounds; r0 += kStages) {
        Batch after;
        load(after, r0 + 2 * kStages);
#pragma unroll
        for (int i = 0; i < kStages; ++i) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
            __syncwarp();
            const uint32_t *data = reinterpret_cast<const uint32_t *>(sData + i * Shape::kStageBytes) + word;
            const int left = length - (r0 + i) * kRound;
            // Entries past the end count as 0 * 0 (the compensated sum skips them).
#pragma unroll
            for (int t0 = 0; t0 < kRound; t0 += 8) {
                if (t0 >= left) break;
                alignas(16) float v[8];
                uint32_t w[8];
                *reinterpret_cast<float4 *>(v) = *reinterpret_cast<const float4 *>(sVal + i * kRound + t0);
                *reinterpret_cast<float4 *>(v + 4) = *reinterpret_cast<const float4 *>(sVal + i * kRound + t0 + 4);
#pragma unroll
                for (int t = 0; t < 8; ++t) w[t] = data[(t0 + t) * 4 * kPieces];
#pragma unroll
                for (int t = 0; t < 8; ++t) {
                    if constexpr (kKahan) {
                        if (t0 + t < left) AccumulateKahan(v[t], __uint_as_float(w[t]), acc[0], comp[0]);
                    } else if constexpr (kCols == 1) {
                        acc[0] = __fadd_rn(acc[0], __fmul_rn(v[t], __uint_as_float(w[t])));
                    } else {
                        float lo, hi;
                        if constexpr (std::is_same_v<ValT, __half>) {
                            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[t]));
                            lo = f.x;
                            hi = f.y;
                        } else {
                            lo = __uint_as_float(w[t] << 16);
                            hi = __uint_as_float(w[t] & 0xffff0000u);
                        }
                        MulAdd2(acc[0], acc[1], lo, hi, v[t], a.negZeros);
                    }
                }
            }
            __syncwarp();
            request(next, i, r0 + kStages + i);
        }
        next = after;
    }
    if (kKahan) acc[0] -= comp[0];
    const float alpha = a.sc.Alpha();
    const float beta = a.sc.Beta();
    const int col = (slice * kPieces * 4 + word) * kCols;
    const bool owner = lane < 4 * kPieces;
    auto store = [&](const float (&v)[kCols]) {
#pragma unroll
        for (int i = 0; i < kCols; ++i) {
            if (owner && col + i < a.n) {
                OutT *dst = a.C + seg.row * a.cRow + (col + i) * a.cCol;
                *dst = Finish<OutT>(v[i], alpha, beta, dst);
            }
        }
    };
    if (seg.longIdx < 0) {
        store(acc);
        return;
    }
    // The unit that comes last adds the row's partial sums of these columns in order.  The lanes fetch 8 of them each,
    // the sets of lanes that own the same columns in turn (a row of 3 M entries, fp32, N = 64: 285 us with one set fetching, 225 so).
    const LongRow lr = a.longRows[seg.longIdx];
    float *partial = static_cast<float *>(a.partials) + (long long)lr.partBase * a.n + col;
#pragma unroll
    for (int i = 0; i < kCols; ++i)
        if (owner && col + i < a.n) __stcg(partial + (long long)seg.seg * a.n + i, acc[i]);
    __threadfence();
    __syncwarp();
    int last = 0;
    if (lane == 0) {
        int32_t *counter = a.counters + (long long)seg.longIdx * a.arrivals + slice;
        last = atomicAdd(counter, 1) == lr.nseg - 1;
        if (last) *counter = 0;  // ready for the next launch
    }
    if (__shfl_sync(0xffffffffu, last, 0) == 0) return;
    __threadfence();
    constexpr int kOwners = 4 * kPieces, kSets = 32 / kOwners, kDeep = 8;
    float tot[kCols] = {};
#pragma unroll 1
    for (int g0 = 0; g0 < lr.nseg; g0 += kDeep * kSets) {
        float v[kDeep][kCols];
#pragma unroll
        for (int g = 0; g < kDeep; ++g) {
            const int at = g0 + g * kSets + lane / kOwners;
#pragma unroll
            for (int i = 0; i < kCols; ++i)
                v[g][i] = at < lr.nseg && col + i < a.n ? __ldcg(partial + (long long)at * a.n + i) : 0.0f;
        }
#pragma unroll
        for (int g = 0; g < kDeep; ++g) {
#pragma unroll
            for (int t = 0; t < kSets; ++t) {
#pragma unroll
                for (int i = 0; i < kCols; ++i) tot[i] += __shfl_sync(0xffffffffu, v[g][i], t * kOwners + word);
            }
        }
    }
    store(tot);
}

// kLanes lanes lie side by side on one row of B (16 bytes each); a warp therefore carries
// 32 / kLanes rows of A at once.  Rows of up to a.rowLimit entries are summed by their group in
// CSR order; longer rows are units, at the front of the grid.  A lane past the end of a B row works on the
// row's first columns once more and stores nothing.
//
// kLayout: kPlain wants C row-major with 16-byte aligned rows, like B; kAnyC takes any C, kAnyCWords also rows of B on
// any 4-byte boundaries, by words (see WorthRepacking); the kinds with Add are for a beta other than 0.  Sums of kAnyC go through shared memory and are written along the
// contiguous direction of C: by a warp where that is the row's, else by the CTA, which takes a.genRows rows (of
// column-major fp16 C, 32 rows are 64 bytes; straight from registers every element would be a 32-byte sector of its
// own) unless there are too few rows to give every SM a CTA.
template <typename ValT, int kLanes> struct FastShape {
    static constexpr int kTileCols = kLanes * Pack<ValT>::kElems;
    static constexpr int kGroup = std::is_same_v<ValT, int8_t> ? Group8<kLanes>::kLanesOfRow : kLanes;  // lanes of a row of A
    static constexpr int kCtaRows = kWarps * (32 / kGroup);                   // rows of A per pass of the CTA
    static constexpr int kFit = 8192 / kTileCols < 32 ? 8192 / kTileCols : 32;  // at most 32 KB of tile
    static constexpr int kGenRows = kCtaRows > kFit ? kCtaRows : kFit;
    // 32 rows of a CTA may be taken in order of their lengths (int8 loses: 44.6 and 50.3 us on 55,686 rows of 0 to 232 entries, N = 16).
    static constexpr bool kMayOrder = !std::is_same_v<ValT, int8_t> && kCtaRows <= 32 && kGroup < 32;
    // int8 instead: the pass over the rows compiled as a loop, although it has one turn.  More of a row's loads are then asked for together, at
    // some spilled registers: faster where the SMs wait for single rows, slower where they have warps enough (see launchFast).
    static constexpr bool kMayLoop = std::is_same_v<ValT, int8_t> && (kLanes == 2 || kLanes == 4);
};

enum { kPlain, kAnyC, kAnyCWords, kAnyCAdd, kAnyCWordsAdd };
// Rows of a few entries are a chain of dependent loads (row offsets, columns, B, C): warps hide it, so registers are held to
// what 36 warps per SM leave (24 for wide int8 rows, whose quads of B rows need more).
template <typename ValT, int kLanes> constexpr int kFastCtas = std::is_same_v<ValT, int8_t> && kLanes >= 8 ? 6 : 9;
template <typename ValT, typename OutT, bool kKahan, int kLanes, int kLayout, bool kOrdered>
__global__ void __launch_bounds__(kThreads, kFastCtas<ValT, kLanes>) SpmmFastKernel(const FastArgs<ValT, OutT> a)
{
    using Acc = typename Arith<ValT>::Acc;
    using Shape = FastShape<ValT, kLanes>;
    constexpr bool kInt8 = std::is_same_v<ValT, int8_t>;
    constexpr bool kGenC = kLayout != kPlain, kWords = kLayout == kAnyCWords || kLayout == kAnyCWordsAdd;
    constexpr bool kAdds = kLayout >= kAnyCAdd;  // beta may be other than 0 (fp types)
    constexpr int E = Pack<ValT>::kElems;
    constexpr int kGroup = Shape::kGroup;
    constexpr int kRowsPerWarp = 32 / kGroup;
    constexpr int kTileCols = Shape::kTileCols;
    constexpr int kTileStride = kTileCols + 1;
    constexpr int kWarpWords = kInt8 ? 32 * E : UnitShape<kLanes>::kWarpBytes / 4;  // what a warp keeps of a unit
    constexpr int kTileWords = kGenC ? (Shape::kGenRows * kTileStride > kThreads * E ? Shape::kGenRows * kTileStride : kThreads * E) : 0;
    __shared__ __align__(16) Acc sBuf[kWarps * kWarpWords > kTileWords ? kWarps * kWarpWords : kTileWords];
    __shared__ unsigned char sSkip[kGenC ? Shape::kGenRows : 1];
    constexpr bool kByLength = kOrdered && !kInt8;
    __shared__ unsigned char sOrder[kByLength ? kWarps : 1][32];
    __shared__ int sLast;

    b200sp::WaitForPrevious();
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int li = lane & (kLanes - 1);
    const bool owner = (lane & (kGroup - 1)) < kLanes;  // of the row's sums once they are joined
    const bool isUnit = (int)blockIdx.x < a.unitCtas;
    if constexpr (!kInt8) {
        if (isUnit) {
            UnitSum<ValT, OutT, kKahan, kLanes, kWords>(a, reinterpret_cast<unsigned char *>(sBuf + warp * kWarpWords));
            return;
        }
    }
    const auto alpha = a.sc.Alpha();
    const auto beta = a.sc.Beta();
    // one element of C at a time, whatever its layout
    auto storeOne = [&](long long row, int col, Acc v) {
        OutT *dst = a.C + row * a.cRow + col * a.cCol;
        *dst = Finish<OutT>(v, alpha, beta, dst);
    };

    // Some of them, beta not 0: what C holds is read for all before any is written, since a load waits for the store before it otherwise, a round
    // trip to memory per element (column-major, beta = 0.5, bf16, 900,000 rows of 2, N = 100 471 us and 323 in eights, 341 in fours).  In kernels of
    // their own: with beta = 0, where nothing is read, the code for it costs 1 to 10 %.
    [[maybe_unused]] constexpr int kStoreBatch = 8;
    [[maybe_unused]] auto addSome = [&]<int kSome>(auto elementOf) {  // elementOf(u, row, column, value): whether there is such an element
        OutT *dst[kSome], old[kSome];
        Acc v[kSome];
#pragma unroll
        for (int u = 0; u < kSome; ++u) {
            long long row = 0;
            int col = 0;
            v[u] = Acc(0);
            dst[u] = elementOf(u, row, col, v[u]) ? a.C + row * a.cRow + col * a.cCol : nullptr;
            old[u] = OutT{};
            if (dst[u] != nullptr) old[u] = *dst[u];
        }
#pragma unroll
        for (int u = 0; u < kSome; ++u)
            if (dst[u] != nullptr) *dst[u] = Finish<OutT>(v[u], alpha, beta, &old[u]);
    };

    constexpr int kCols = kInt8 ? 1 : 4 / (int)sizeof(ValT);
    auto columnOf = [&](int colT, int i) {  // that acc[i] of this lane is for
        return kWords ? colT + (i / kCols * kLanes + li) * kCols + i % kCols : colT + li * E + i;
    };

    const bool splitRow = kInt8 && a.splitRows && !isUnit;
    if (!isUnit && !splitRow) {
        // ---- one lane group per row ----
        constexpr int kChunk = kInt8 ? Group8<kLanes>::kChunk : Chunk<kLanes>::kChunk;
        const bool rowsRun = kGenC && a.cCol != 1;  // column-major C
        const int blockRows = kByLength ? 32 : rowsRun || kOrdered ? a.genRows : Shape::kCtaRows;
        const long long row0 = (long long)(blockIdx.x - a.unitCtas) * blockRows;
        if constexpr (kByLength) {  // sOrder[i]: the row with the i-th most entries (every warp has its own copy: no barrier)
            int len = row0 + lane < a.m ? a.rowPtr[row0 + lane + 1] - a.rowPtr[row0 + lane] : 0;
            if (len > a.rowLimit) len = 0;
            const int key = len << 5 | (31 - lane);
            int rank = 0;
#pragma unroll
            for (int j = 1; j < 32; ++j) rank += __shfl_xor_sync(0xffffffffu, key, j) > key;
            sOrder[warp][rank] = (unsigned char)lane;
            __syncwarp();
        }
        for (int col0 = 0; col0 < (rowsRun ? a.n : 1); col0 += kTileCols) {  // column-major C: a tile of columns at a time
#pragma unroll 1
            for (int pass = 0; pass < blockRows; pass += Shape::kCtaRows) {
                int rowIn = pass + warp * kRowsPerWarp + lane / kGroup;
                if constexpr (kByLength) {
                    // every other pass the other way round: the warp with the longest rows of one has the shortest of the next
                    const int turn = pass & Shape::kCtaRows ? kWarps - 1 - warp : warp;
                    rowIn = sOrder[warp][pass + turn * kRowsPerWarp + lane / kGroup];
                }
                const long long row = row0 + rowIn;
                int s = 0, e = 0;
                bool skip = row >= a.m;
                if (row < a.m) {
                    s = a.rowPtr[row];
                    e = a.rowPtr[row + 1];
                    if (e - s > a.rowLimit) {  // a unit
                        e = s;
                        skip = true;
                    }
                }
                int trips = (e - s + kChunk - 1) / kChunk;
#pragma unroll
                for (int off = kGroup; off < 32; off <<= 1) {
                    const int other = __shfl_xor_sync(0xffffffffu, trips, off);
                    trips = other > trips ? other : trips;
                }
                const int colFirst = rowsRun ? col0 : 0, colLast = rowsRun ? col0 + 1 : a.n;
                for (int colT = colFirst; colT < colLast; colT += kTileCols) {
                    const int col = colT + li * E;
                    const bool colLive = col < a.nB;
                    Acc acc[E], comp[E];
#pragma unroll
                    for (int i = 0; i < E; ++i) acc[i] = comp[i] = Acc(0);
                    if constexpr (kInt8) {
                        RowDot8<kLanes>(a.colInd, a.val, a.B + (colLive ? col : 0), a.ldb, s, e, trips, acc);
#pragma unroll
                        for (int i = 0; i < E; ++i) {
                            if (kLanes == 1 && i >= a.n) break;
#pragma unroll
                            for (int off = kLanes; off < kGroup; off <<= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], off);
                        }
                    } else {
                        Slice<ValT, kWords> slice;
                        if constexpr (kWords) {
#pragma unroll
                            for (int j = 0; j < 4; ++j) slice.first[j] = columnOf(colT, j * kCols) < a.n ? columnOf(colT, j * kCols) : 0;
                        } else {
                            slice.first[0] = colLive ? col : 0;
                        }
                        RowDot<ValT, kKahan, kLanes, kWords, kOrdered>(a.colInd, a.val, a.B, slice, a.ldb, s, e, trips, a.negZeros, acc, comp);
                    }
                    if (kKahan) {
#pragma unroll
                        for (int i = 0; i < E; ++i) acc[i] -= comp[i];
                    }
                    if constexpr (kGenC) {
                        if (rowsRun) {
#pragma unroll
                            for (int i = 0; i < E; ++i)
                                if (owner) sBuf[rowIn * kTileStride + columnOf(0, i)] = acc[i];
                            if (li == 0) sSkip[rowIn] = skip;
                        } else if constexpr (kWords && kLanes >= 8) {  // a group writes whole sectors: consecutive lanes hold consecutive words
#pragma unroll
                            for (int i = 0; i < E; ++i)
                                if (!skip && columnOf(colT, i) < a.n) storeOne(row, columnOf(colT, i), acc[i]);
                        } else {
                            Acc *sWarp = sBuf + warp * 32 * E;
                            const unsigned skipped = __ballot_sync(0xffffffffu, skip);
                            __syncwarp();
#pragma unroll
                            for (int i = 0; i < E; ++i)
                                if (owner) sWarp[lane / kGroup * kTileCols + columnOf(0, i)] = acc[i];
                            __syncwarp();
                            auto element = [&](int i, long long &toRow, int &toCol, Acc &v) {
                                const int g = i / kTileCols;
                                const int r = kByLength ? __shfl_sync(0xffffffffu, rowIn, g * kGroup) : warp * kRowsPerWarp + g;
                                toRow = row0 + r;
                                toCol = colT + i % kTileCols;
                                v = sWarp[i];
                                return toCol < a.n && !(skipped >> (g * kGroup) & 1);
                            };
                            constexpr int kElements = kRowsPerWarp * kTileCols;  // a multiple of 32: all lanes take part in every step
                            if (!kAdds || beta == 0) {
#pragma unroll
                                for (int i = lane; i < kElements; i += 32) {
                                    long long toRow;
                                    int toCol;
                                    Acc v;
                                    if (element(i, toRow, toCol, v)) storeOne(toRow, toCol, v);
                                }
                            } else if constexpr (kAdds) {
                                constexpr int kSome = kElements / 32 < kStoreBatch ? kElements / 32 : kStoreBatch;
                                static_assert(kElements % (32 * kSome) == 0);
                                for (int i0 = lane; i0 < kElements; i0 += 32 * kSome)
                                    addSome.template operator()<kSome>([&](int u, long long &toRow, int &toCol, Acc &v) {
                                        return element(i0 + u * 32, toRow, toCol, v);
                                    });
                            }
                        }
                    } else {
                        if (!skip && colLive && owner) StoreRowSlice(a.C + row * a.ldc + col, acc, alpha, beta);
                    }
                }
            }
            if (rowsRun) {
                __syncthreads();
                if (!kAdds || beta == 0) {
                    for (int i = threadIdx.x; i < blockRows * kTileCols; i += kThreads) {  // consecutive threads on consecutive rows
                        const int c = i / blockRows, r = i - c * blockRows;
                        if (col0 + c < a.n && !sSkip[r]) storeOne(row0 + r, col0 + c, sBuf[r * kTileStride + c]);
                    }
                } else if constexpr (kAdds) {
                    for (int i0 = threadIdx.x; i0 < blockRows * kTileCols; i0 += kThreads * kStoreBatch)
                        addSome.template operator()<kStoreBatch>([&](int u, long long &toRow, int &toCol, Acc &v) {
                            const int i = i0 + u * kThreads;
                            if (i >= blockRows * kTileCols) return false;
                            const int c = i / blockRows, r = i - c * blockRows;
                            toRow = row0 + r;
                            toCol = col0 + c;
                            v = sBuf[r * kTileStride + c];
                            return toCol < a.n && !sSkip[r];
                        });
                }
                __syncthreads();
            }
        }
        return;
    }

    // ---- int8: one CTA per unit (with split rows also per row), the four warps take a quarter each ----
    if constexpr (kInt8) {
        const SegEntry seg = splitRow ? SegEntry{(int)blockIdx.x - a.unitCtas, 0, -1, 0}
                             : (int)blockIdx.x < a.longUnits ? a.segs[blockIdx.x]
                                                             : a.segsEnd[a.longUnits - 1 - (int)blockIdx.x];
        const LongRow lr = seg.longIdx < 0 ? LongRow{seg.row, 0, 1, 0} : a.longRows[seg.longIdx];
        const int rowStart = a.rowPtr[seg.row];
        const int rowEnd = a.rowPtr[seg.row + 1];
        if (splitRow && rowEnd - rowStart > a.rowLimit) return;
        const int segStart = rowStart + seg.seg * kSegNnz;
        const int segEnd = rowEnd - segStart > kSegNnz ? segStart + kSegNnz : rowEnd;
        // inside a warp the lane groups take interleaved chunks of the warp's quarter
        const int quarter = ((segEnd - segStart + 4 * kWarps - 1) / (4 * kWarps)) * 4;
        int ws = segStart + warp * quarter;
        int we = ws + quarter;
        if (ws > segEnd) ws = segEnd;
        if (we > segEnd) we = segEnd;
        constexpr int kChunk = Group8<kLanes>::kChunk;
        const int g = lane / kGroup;
        Acc *partial = static_cast<Acc *>(a.partials) + (long long)(lr.partBase + seg.seg) * a.n;
        auto storeSlice = [&](int col, const Acc (&v)[E]) {
            if constexpr (kGenC) {
#pragma unroll
                for (int i = 0; i < E; ++i)
                    if (col + i < a.n) storeOne(seg.row, col + i, v[i]);
            } else {
                StoreRowSlice(a.C + (long long)seg.row * a.ldc + col, v, alpha, beta);
            }
        };

        for (int col0 = 0; col0 < a.n; col0 += kTileCols) {
            const int col = col0 + li * E;
            const bool colLive = col < a.nB;
            Acc acc[E];
#pragma unroll
            for (int i = 0; i < E; ++i) acc[i] = Acc(0);
            // group g walks chunks g, g + kRowsPerWarp, ... of [ws, we)
            const int nChunks = (we - ws + kChunk - 1) / kChunk;
            for (int ch0 = 0; ch0 < nChunks; ch0 += kRowsPerWarp) {  // same trip count in every group
                const int ch = ch0 + g;
                const int cs = ws + ch * kChunk < we ? ws + ch * kChunk : we;
                const int ce = cs + kChunk < we ? cs + kChunk : we;
                RowDot8<kLanes>(a.colInd, a.val, a.B + (colLive ? col : 0), a.ldb, cs, ce, 1, acc);
            }
#pragma unroll
            for (int i = 0; i < E; ++i) {
#pragma unroll
                for (int off = kLanes; off < 32; off <<= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], off);
            }
            if (lane < kLanes) {
#pragma unroll
                for (int i = 0; i < E; ++i) sBuf[warp * 32 * E + li * E + i] = acc[i];
            }
            __syncthreads();
            // warp 0 adds the four warps' slices
            if (warp == 0 && lane < kLanes && colLive) {
                Acc tot[E];
#pragma unroll
                for (int i = 0; i < E; ++i) {
                    tot[i] = sBuf[li * E + i];
#pragma unroll
                    for (int w = 1; w < kWarps; ++w) tot[i] += sBuf[w * 32 * E + li * E + i];
                }
                if (lr.nseg == 1) {
                    storeSlice(col, tot);
                } else {
#pragma unroll
                    for (int i = 0; i < E; ++i)
                        if (!kGenC || col + i < a.n) partial[col + i] = tot[i];
                }
            }
            __syncthreads();
        }
        if (lr.nseg == 1) return;

        // Arrival: the unit that comes last sums all partial rows.
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            int32_t *counter = a.counters + (long long)seg.longIdx * a.arrivals;
            const int old = atomicAdd(counter, 1);
            sLast = (old == lr.nseg - 1);
            if (sLast) *counter = 0;  // ready for the next launch
        }
        __syncthreads();
        if (!sLast) return;
        __threadfence();
        const Acc *first = static_cast<const Acc *>(a.partials) + (long long)lr.partBase * a.n;
        for (int col = threadIdx.x * E; col < a.n; col += kThreads * E) {
            Acc tot[E];
#pragma unroll
            for (int i = 0; i < E; ++i) tot[i] = Acc(0);
            for (int sgi = 0; sgi < lr.nseg; ++sgi) {
#pragma unroll
                for (int i = 0; i < E; ++i)
                    if (!kGenC || col + i < a.n) tot[i] += __ldcg(first + (long long)sgi * a.n + col + i);
            }
            storeSlice(col, tot);
        }
    }
}

// ---------------------------------------------------------------- long rows by column blocks

// When B is much larger than L2, a long row of A gathers every one of its B rows from DRAM.  Rows of more than
// kLongRow entries are few and hold a large share of the non-zeros (a graph's hubs); with ascending columns the
// entries of such a row that fall into one block of consecutive B rows are contiguous in col_ind.  So B is cut
// into blocks of about kBlockBytes and the grid walks the pieces (row, block) block by block: while one block
// is being worked on, every long row gathers from the same few megabytes, which the first touch brings into L2
// and the evict-last policy of the B loads keeps there.  Pieces are cut into units of at most kUnitNnz entries so
// that all units take about the same time and the grid stays inside a window of one or two blocks.  A warp sums
// one unit in CSR order into one partial row; SpmmLongSumKernel then adds the partial rows of a row in column order (fixed
// order: the same bits every run) and applies the epilogue.
struct BlockArgs {
    int nUnits;
    const BlockUnit *units;   // ordered by column block
    const int2 *rowSlots;     // [long row] {first partial slot, slots}
    int nLong;
    float *partials;          // [slot][n]
    unsigned long long share; // of the units in the row-stream kernel's grid, times 2^32
};

// Packed fp32 arithmetic of sm_100: one instruction, two fused multiply-adds.  The long rows are not bound to the
// golden's separate multiply and add (their sums are regrouped by block anyway), and this kernel, fed from L2,
// is limited by instruction issue rather than by DRAM.
__device__ __forceinline__ void Fma2(float2 &acc, float x, float y, float v)
{
    unsigned long long a, bq, c;
    asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(x), "f"(y));
    asm("mov.b64 %0, {%1, %1};" : "=l"(bq) : "f"(v));
    asm("mov.b64 %0, {%1, %2};" : "=l"(c) : "f"(acc.x), "f"(acc.y));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(bq));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(acc.x), "=f"(acc.y) : "l"(c));
}

// acc[0 .. E/2) += v * (the E values of 16 bytes of a B row)
template <typename ValT> struct FusedRow;
template <> struct FusedRow<float> {
    static __device__ __forceinline__ void Add(const uint4 &q, float v, float2 (&acc)[2])
    {
        Fma2(acc[0], __uint_as_float(q.x), __uint_as_float(q.y), v);
        Fma2(acc[1], __uint_as_float(q.z), __uint_as_float(q.w), v);
    }
};
template <> struct FusedRow<__nv_bfloat16> {
    static __device__ __forceinline__ void Add(const uint4 &q, float v, float2 (&acc)[4])
    {
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
            Fma2(acc[i], __uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u), v);
    }
};
template <> struct FusedRow<__half> {
    static __device__ __forceinline__ void Add(const uint4 &q, float v, float2 (&acc)[4])
    {
        const __half2 *h = reinterpret_cast<const __half2 *>(&q);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(h[i]);
            Fma2(acc[i], f.x, f.y, v);
        }
    }
};

// ---------------------------------------------------------------- row-stream path

// For B rows of 512 or 1024 bytes.  A warp owns up to 32 consecutive rows of A and walks their
// non-zeros as one stream, in CSR order, across the row boundaries; the B row of every entry
// is brought into shared memory by the copy engine (cp.async.bulk, one row per copy, completion
// counted on an mbarrier) several batches ahead of its use, so the chain row_ptr -> col_ind ->
// B row -> C row that bounds a row-at-a-time kernel on matrices full of one- and two-entry
// rows is paid once per warp, not once per row, and no registers hold data in flight.
// Every lane owns kRowBytes / 32 bytes of the row; each output keeps one fp32 accumulator
// that takes its products in CSR order with separate multiply and add, as in the kernel above,
// so the results are the same bits.  Rows above kLongRow entries are left to the segment CTAs
// of SpmmFastKernel or, by column blocks of B, are units of the same grid.
// Measured on the 2 M x 2 M graph matrix with 512-byte rows (ms per product, segment CTAs included):
// 3 buffers x 16 rows x 4 warps per CTA 5.28; 2 x 16 x 4 3.97; 2 x 8 x 4 3.29; 2 x 4 x 4 3.38;
// 2 x 8 x 2 2.99; 2 x 8 x 1 2.91.  Less shared memory per warp means more warps per SM, and
// one warp per CTA gives the memory of a finished warp back at once.
// The rows are bound by DRAM, the units of long rows by the latency of L2.  One kernel after the other (two streams do not
// help: the first takes every SM until its last CTA has started) they took 2610 us; in one grid, units spread evenly
// among the rows, 2300; 13.0 GB of DRAM traffic now (1985 us at the copy rate), 13.5 as two.  The entries are looked up 32 at a time,
// not one batch at a time, which is 120 of those 310 us: issue slots 57 % busy.
#ifndef B200SP_SPMM_STREAM_BUFFERS
#define B200SP_SPMM_STREAM_BUFFERS 2
#endif
#ifndef B200SP_SPMM_STREAM_BATCH_BYTES
#define B200SP_SPMM_STREAM_BATCH_BYTES 4096
#endif
#ifndef B200SP_SPMM_STREAM_WARPS
#define B200SP_SPMM_STREAM_WARPS 1
#endif
constexpr int kStreamBuffers = B200SP_SPMM_STREAM_BUFFERS;  // batches of B rows per warp: one in use, the rest in flight
constexpr int kStreamWarps = B200SP_SPMM_STREAM_WARPS;
constexpr int kStreamThreads = kStreamWarps * 32;
constexpr long long kStreamWaitCycles = 1ll << 31;           // SM clocks (about a second) to wait on one barrier before giving up
// What the next launches pass to the kernel as its wait limit and as bytes to expect beyond those it copies
// (b200sp_spmm_stream_wait_test: a test makes a wait run out without any fault by expecting bytes nobody sends).
long long gHostStreamWaitCycles = kStreamWaitCycles;
unsigned gHostStreamExtraTx = 0;

__device__ int gStreamError;  // set when a wait of the row-stream kernel ran out (never observed; it then stops writing C)

__device__ __forceinline__ uint32_t SmemAddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void MbarInit(uint64_t *bar, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(SmemAddr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void MbarExpectTx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(SmemAddr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool MbarTryWait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(SmemAddr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Polls with a time limit; false when the limit was reached.
__device__ __forceinline__ bool MbarWait(uint64_t *bar, uint32_t parity, long long limit)
{
    if (MbarTryWait(bar, parity)) return true;
    const long long t0 = clock64();
    while (!MbarTryWait(bar, parity)) {
        if (clock64() - t0 > limit) return false;
    }
    return true;
}
// One row: global -> shared through the copy engine; both addresses 16-byte aligned, bytes a multiple of 16.  kOnce: with an
// L2 evict-first policy, so that rows that stream through L2 do not displace the block of B that units of long rows in the
// same grid gather from (2 M x 2 M graph matrix, 512-byte rows: 2290 us with it, 2390 without; by itself the row stream
// loses 5 % to it).  A policy is made where it is used, by one instruction, and is never one of two: see the note at SDDMM's kNearSpan.
template <bool kOnce> __device__ __forceinline__ void BulkLoadRow(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    if constexpr (kOnce) {
        uint64_t pol;
        asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
                SmemAddr(dst)),
            "l"(src), "r"(bytes), "r"(SmemAddr(bar)), "l"(pol)
            : "memory");
    } else {
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         SmemAddr(dst)),
                     "l"(src), "r"(bytes), "r"(SmemAddr(bar))
                     : "memory");
    }
}

// What bounds a unit is the latency of its gathers from L2: the rows of B come through shared memory by cp.async, three
// requests of four rows in flight per warp, and a lane reads back what it asked for itself.  (The copy engine starts a row
// per 20 clocks and SM, which the ordinary rows of the same grid use up; plain loads into registers leave a warp without
// any in flight while it sums.)
constexpr int kUnitRows = 4;      // rows of B per request
constexpr int kUnitRequests = 4;  // three in flight, one being summed
constexpr int kUnitTile = 512;    // bytes of a row of B that a warp takes at a time
constexpr int kUnitRing = kUnitRequests * kUnitRows * kUnitTile;

// One unit by one warp; ring: kUnitRing bytes of shared memory of its own.
template <typename ValT, typename OutT>
__device__ __forceinline__ void LongUnit(const FastArgs<ValT, OutT> &a, const BlockArgs &b, int unit, unsigned char *ring)
{
    constexpr int E = Pack<ValT>::kElems;
    constexpr int kTileCols = kUnitTile / (int)sizeof(ValT);
    constexpr int kChunkRequests = 32 / kUnitRows;
    static_assert(kUnitTile == 32 * 16 && kUnitRequests - 1 <= kChunkRequests && kChunkRequests % kUnitRequests == 0);
    const int lane = threadIdx.x & 31;
    const int4 raw = __ldg(reinterpret_cast<const int4 *>(b.units) + unit);
    const int s = raw.x, total = raw.y - raw.x, slot = raw.w;
    float *partial = b.partials + (long long)slot * a.n;
    unsigned char *const mine = ring + lane * 16;
    uint64_t policy;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(policy));
    for (int col0 = 0; col0 < a.n; col0 += kTileCols) {
        const int col = col0 + lane * E;
        const bool colLive = col < a.n;
        const ValT *Bs = a.B + (colLive ? col : 0);
        float2 acc[E / 2];
#pragma unroll
        for (int i = 0; i < E / 2; ++i) acc[i] = make_float2(0.0f, 0.0f);
        // 32 entries at a time, one per lane (column -1 after the last), and the next 32 on their way
        auto fetch = [&](int first, int &c, float &v) {
            c = -1;
            v = 0.0f;
            if (first + lane < total) {
                c = __ldcs(a.colInd + s + first + lane);
                v = ToF32(__ldcs(a.val + s + first + lane));
            }
        };
        int colNow, colNext;
        float valNow, valNext;
        fetch(0, colNow, valNow);
        fetch(32, colNext, valNext);
        auto request = [&](int from, int first, int place) {  // past the last entry: zeros, nothing is read
#pragma unroll
            for (int u = 0; u < kUnitRows; ++u) {
                const int c = __shfl_sync(0xffffffffu, from, first + u);
                asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;" ::"r"(
                                 SmemAddr(mine + (place * kUnitRows + u) * kUnitTile)),
                             "l"(Bs + (long long)(c < 0 ? 0 : c) * a.ldb), "r"(c < 0 ? 0 : 16), "l"(policy)
                             : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll
        for (int r = 0; r < kUnitRequests - 1; ++r) request(colNow, kUnitRows * r, r);
        for (int done = 0; done < total; done += 32) {
#pragma unroll
            for (int r = 0; r < kChunkRequests; ++r) {
                if (done + kUnitRows * r >= total) break;
                constexpr int kAhead = kUnitRequests - 1;
                __syncwarp();  // the place asked for next has been read
                if (r + kAhead < kChunkRequests) request(colNow, kUnitRows * (r + kAhead), (r + kAhead) % kUnitRequests);
                else request(colNext, kUnitRows * (r + kAhead - kChunkRequests), (r + kAhead) % kUnitRequests);
                asm volatile("cp.async.wait_group %0;" ::"n"(kAhead) : "memory");
#pragma unroll
                for (int u = 0; u < kUnitRows; ++u) {
                    const float v = __shfl_sync(0xffffffffu, valNow, kUnitRows * r + u);
                    const uint4 q = *reinterpret_cast<const uint4 *>(mine + ((r % kUnitRequests) * kUnitRows + u) * kUnitTile);
                    FusedRow<ValT>::Add(q, v, acc);
                }
            }
            colNow = colNext;
            valNow = valNext;
            fetch(done + 64, colNext, valNext);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        if (colLive) {
#pragma unroll
            for (int i = 0; i < E / 2; i += 2)
                __stcg(reinterpret_cast<float4 *>(partial + col + 2 * i),
                       make_float4(acc[i].x, acc[i].y, acc[i + 1].x, acc[i + 1].y));
        }
    }
}

// The units alone, beside SpmmFastKernel for the other rows.  A CTA per kBlockWarps units, in their order: a fixed grid that walks them with a
// stride drifts apart until the window of blocks in use outgrows L2 (1739 us instead of 714).
constexpr int kBlockWarps = 2;
template <typename ValT, typename OutT>
__global__ void __launch_bounds__(32 * kBlockWarps) SpmmLongBlockKernel(const FastArgs<ValT, OutT> a, const BlockArgs b)
{
    __shared__ __align__(16) unsigned char ring[kBlockWarps][kUnitRing];
    const long long unit = (long long)blockIdx.x * kBlockWarps + (threadIdx.x >> 5);
    if (unit < b.nUnits) LongUnit<ValT, OutT>(a, b, (int)unit, ring[threadIdx.x >> 5]);
}

// C of the long rows from their partial rows: a warp per 32 columns of a row, which are added up in slot (= column) order.
template <typename OutT, typename ArgsT>
__global__ void __launch_bounds__(256) SpmmLongSumKernel(const ArgsT a, const BlockArgs b)
{
    b200sp::WaitForPrevious();
    const int slices = (a.n + 31) / 32;
    const long long w = (long long)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (w >= (long long)b.nLong * slices) return;
    const int li = (int)(w / slices);
    const int col = (int)(w % slices) * 32 + (threadIdx.x & 31);
    if (col >= a.n) return;
    const int2 rs = __ldg(b.rowSlots + li);
    const float *at = b.partials + (long long)rs.x * a.n + col;
    float tot = 0.0f;
#pragma unroll 16
    for (int sl = 0; sl < rs.y; ++sl) tot += __ldcs(at + (long long)sl * a.n);
    OutT *dst = a.C + (long long)a.longRows[li].row * a.ldc + col;
    *dst = Finish(tot, a.sc.Alpha(), a.sc.Beta(), dst);
}

template <int kBytes> struct LaneWords {  // kBytes of shared memory as 32-bit words
    static constexpr int kWords = kBytes / 4;
    static __device__ __forceinline__ void Load(const unsigned char *p, uint32_t (&w)[kWords])
    {
        if constexpr (kBytes == 4) {
            w[0] = *reinterpret_cast<const uint32_t *>(p);
        } else if constexpr (kBytes == 8) {
            const uint2 q = *reinterpret_cast<const uint2 *>(p);
            w[0] = q.x; w[1] = q.y;
        } else {
            static_assert(kBytes % 16 == 0, "a lane owns 4, 8 or a multiple of 16 bytes of a B row");
#pragma unroll
            for (int i = 0; i < kBytes / 16; ++i) {
                const uint4 q = reinterpret_cast<const uint4 *>(p)[i];
                w[4 * i] = q.x; w[4 * i + 1] = q.y; w[4 * i + 2] = q.z; w[4 * i + 3] = q.w;
            }
        }
    }
};

template <typename ValT, int kWords> struct WordsToF32;
template <int kWords> struct WordsToF32<float, kWords> {
    static constexpr int kElems = kWords;
    static __device__ __forceinline__ void Convert(const uint32_t (&w)[kWords], float (&out)[kElems])
    {
#pragma unroll
        for (int i = 0; i < kWords; ++i) out[i] = __uint_as_float(w[i]);
    }
};
template <int kWords> struct WordsToF32<__half, kWords> {
    static constexpr int kElems = 2 * kWords;
    static __device__ __forceinline__ void Convert(const uint32_t (&w)[kWords], float (&out)[kElems])
    {
#pragma unroll
        for (int i = 0; i < kWords; ++i) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
            out[2 * i] = f.x;
            out[2 * i + 1] = f.y;
        }
    }
};
template <int kWords> struct WordsToF32<__nv_bfloat16, kWords> {
    static constexpr int kElems = 2 * kWords;
    static __device__ __forceinline__ void Convert(const uint32_t (&w)[kWords], float (&out)[kElems])
    {
#pragma unroll
        for (int i = 0; i < kWords; ++i) {  // bf16 -> fp32 is a 16-bit shift
            out[2 * i] = __uint_as_float(w[i] << 16);
            out[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
};

// E consecutive outputs of one lane: z = alpha * acc + beta * old, stored with the widest aligned vector.
template <typename OutT, int E>
__device__ __forceinline__ void LoadOld(const OutT *src, float (&old)[E])
{
#pragma unroll
    for (int i = 0; i < E; ++i) old[i] = ToF32(src[i]);  // contiguous: the compiler merges these into vector loads
}
template <typename OutT, int E>
__device__ __forceinline__ void StoreSlice(OutT *dst, const float (&acc)[E], const float (&old)[E], float alpha,
                                           float beta)
{
    float z[E];
#pragma unroll
    for (int i = 0; i < E; ++i)
        z[i] = beta != 0.0f ? __fadd_rn(__fmul_rn(alpha, acc[i]), __fmul_rn(beta, old[i])) : __fmul_rn(alpha, acc[i]);
    constexpr int kBytes = E * (int)sizeof(OutT);
    alignas(16) OutT o[E];
#pragma unroll
    for (int i = 0; i < E; ++i) o[i] = FromF32<OutT>(z[i]);
    if constexpr (kBytes % 16 == 0) {
#pragma unroll
        for (int i = 0; i < kBytes / 16; ++i)
            __stcs(reinterpret_cast<uint4 *>(dst) + i, reinterpret_cast<const uint4 *>(o)[i]);
    } else if constexpr (kBytes == 8) {
        *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(o);
    } else {
        static_assert(kBytes == 4, "a lane writes 4, 8 or a multiple of 16 bytes of a C row");
        *reinterpret_cast<uint32_t *>(dst) = *reinterpret_cast<const uint32_t *>(o);
    }
}

template <typename ValT, typename OutT>
struct StreamArgs {
    const int32_t *rowPtr;
    const int32_t *colInd;
    const ValT *val;
    const ValT *B;
    OutT *C;
    int m;
    int warpRows;            // rows of A per warp, up to 32
    int rowLimit;
    long long ldb;
    long long ldc;
    ScalarsF sc;
    long long waitCycles;   // limit of every wait on a copy barrier, in SM clocks
    unsigned long long negZeros;
    unsigned extraTx;       // bytes expected on every barrier beyond those copied (0 outside the wait test)
};

template <int kRowBytes> struct StreamShape {
    static constexpr int kBatch = B200SP_SPMM_STREAM_BATCH_BYTES / kRowBytes;  // B rows per batch
    static_assert(kBatch >= 1 && kBatch <= 32, "a lane issues at most one row copy per batch");
    static constexpr int kWarpBytes = kStreamBuffers * (kBatch * kRowBytes + kBatch * 8) + 64;  // data, val, meta, barriers
    static constexpr int kCtaBytes = kStreamWarps * kWarpBytes;
};

// kUnits: units of long rows are CTAs of this grid.
template <typename ValT, typename OutT, int kRowBytes, bool kUnits>
__global__ void __launch_bounds__(kStreamThreads) SpmmRowStreamKernel(const StreamArgs<ValT, OutT> a,
                                                                      [[maybe_unused]] const FastArgs<ValT, OutT> fa,
                                                                      [[maybe_unused]] const BlockArgs ba)
{
    using Shape = StreamShape<kRowBytes>;
    constexpr int kBatch = Shape::kBatch;
    constexpr int kLaneBytes = kRowBytes / 32;
    constexpr int kWords = kLaneBytes / 4;
    constexpr int E = WordsToF32<ValT, kWords>::kElems;
    extern __shared__ __align__(128) unsigned char sRaw[];
    static_assert(kStreamWarps == 1 && Shape::kCtaBytes >= kUnitRing, "a unit takes the place of a warp");

    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    unsigned before = 0;
    if constexpr (kUnits) {  // spread evenly over the grid
        before = (unsigned)((blockIdx.x * ba.share) >> 32);
        if ((unsigned)(((blockIdx.x + 1ull) * ba.share) >> 32) != before) {
            LongUnit<ValT, OutT>(fa, ba, (int)before, sRaw);
            return;
        }
    }
    unsigned char *base = sRaw + (size_t)warp * Shape::kWarpBytes;
    unsigned char *sData = base;                                                          // [buffers][kBatch][kRowBytes]
    float *sVal = reinterpret_cast<float *>(base + kStreamBuffers * kBatch * kRowBytes);  // [buffers][kBatch]
    int *sMeta = reinterpret_cast<int *>(sVal + kStreamBuffers * kBatch);                 // [buffers][kBatch]
    uint64_t *sBar = reinterpret_cast<uint64_t *>(sMeta + kStreamBuffers * kBatch);       // [buffers]

    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < kStreamBuffers; ++i) MbarInit(sBar + i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();

    const float alpha = a.sc.Alpha();
    const float beta = a.sc.Beta();
    const long long r0 = ((blockIdx.x - before) * kStreamWarps + warp) * a.warpRows;
    if (r0 >= a.m) return;

    // This lane's row: bounds, length, and where its entries start in the warp's stream.
    const long long myRow = r0 + lane;
    int s = 0, len = 0;
    bool mine = false;
    if (lane < a.warpRows && myRow < a.m) {
        s = a.rowPtr[myRow];
        len = a.rowPtr[myRow + 1] - s;
        mine = len <= a.rowLimit;  // longer rows are units
        if (!mine) len = 0;
    }
    int off = len;  // inclusive scan over the lanes, then made exclusive
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, off, d);
        if (lane >= d) off += t;
    }
    const int total = __shfl_sync(0xffffffffu, off, 31);
    off -= len;

    OutT *cRow0 = a.C + r0 * a.ldc + lane * E;
    // Rows without entries: C = beta * C.
    unsigned emptyMask = __ballot_sync(0xffffffffu, mine && len == 0);
    while (emptyMask != 0) {
        const int l = __ffs(emptyMask) - 1;
        emptyMask &= emptyMask - 1;
        float zero[E], old[E];
#pragma unroll
        for (int i = 0; i < E; ++i) zero[i] = old[i] = 0.0f;
        OutT *dst = cRow0 + (long long)l * a.ldc;
        if (beta != 0.0f) LoadOld<OutT, E>(dst, old);
        StoreSlice<OutT, E>(dst, zero, old, alpha, beta);
    }
    if (total == 0) return;
    const unsigned liveMask = __ballot_sync(0xffffffffu, len > 0);

    const int nBatches = (total + kBatch - 1) / kBatch;
    // The stream's entries, 32 at a time, an entry per lane: column, value, and which row it belongs to / whether it ends
    // that row.  The chunk in use, and the next one, on its way.
    constexpr int kPerChunk = 32 / kBatch;
    int eCol = 0, eMeta = 0, nCol = 0, nMeta = 0;
    float eVal = 0.0f, nVal = 0.0f;
    auto fetchChunk = [&](int chunk) {
        const int q = chunk * 32 + lane;
        // last lane whose stream offset is <= q: the row that holds entry q
        int lo = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
            const int cand = lo + step;
            const int offC = __shfl_sync(0xffffffffu, off, cand & 31);
            if (cand < 32 && offC <= q) lo = cand;
        }
        const int sL = __shfl_sync(0xffffffffu, s, lo);
        const int offL = __shfl_sync(0xffffffffu, off, lo);
        const int lenL = __shfl_sync(0xffffffffu, len, lo);
        if (q < total) {
            const int p = sL + (q - offL);
            nCol = __ldcs(a.colInd + p);
            nVal = ToF32(__ldcs(a.val + p));
            nMeta = lo | ((q - offL == lenL - 1) ? 0x100 : 0);
        }
    };
    auto issueBatch = [&](int k) {
        if (k % kPerChunk == 0) {
            eCol = nCol;
            eVal = nVal;
            eMeta = nMeta;
            if ((k + kPerChunk) * kBatch < total) fetchChunk(k / kPerChunk + 1);
        }
        const int buf = k % kStreamBuffers;
        const int live = total - k * kBatch < kBatch ? total - k * kBatch : kBatch;
        if (lane == 0) MbarExpectTx(sBar + buf, (uint32_t)live * kRowBytes + a.extraTx);
        __syncwarp();
        const int i = lane - (k % kPerChunk) * kBatch;
        if (i >= 0 && i < live) {
            sVal[buf * kBatch + i] = eVal;
            sMeta[buf * kBatch + i] = eMeta;
            BulkLoadRow<kUnits>(sData + ((size_t)buf * kBatch + i) * kRowBytes, a.B + (long long)eCol * a.ldb, kRowBytes, sBar + buf);
        }
    };

    // prologue: all but one buffer in flight
    const int ahead = kStreamBuffers - 1;
    fetchChunk(0);
    for (int k = 0; k < ahead && k < nBatches; ++k) issueBatch(k);

    float acc[E], old[E];
#pragma unroll
    for (int i = 0; i < E; ++i) acc[i] = old[i] = 0.0f;
    // C of the row being summed is requested when the row before it is written (when the warp starts, for the first)
    if (beta != 0.0f) LoadOld<OutT, E>(cRow0 + (long long)(__ffs(liveMask) - 1) * a.ldc, old);

    int failedAt = -1;
    for (int k = 0; k < nBatches; ++k) {
        if (k + ahead < nBatches) issueBatch(k + ahead);
        const int buf = k % kStreamBuffers;
        __syncwarp();
        if (!MbarWait(sBar + buf, (uint32_t)(k / kStreamBuffers) & 1u, a.waitCycles)) {
            failedAt = k;
            if (lane == 0) atomicExch(&gStreamError, 1);
            break;
        }
        const int live = total - k * kBatch < kBatch ? total - k * kBatch : kBatch;
        const unsigned char *rowData = sData + (size_t)buf * kBatch * kRowBytes + lane * kLaneBytes;
#pragma unroll 4
        for (int j = 0; j < live; ++j) {
            const int meta = sMeta[buf * kBatch + j];
            const float v = sVal[buf * kBatch + j];
            uint32_t w[kWords];
            LaneWords<kLaneBytes>::Load(rowData + (size_t)j * kRowBytes, w);
            float b[E];
            WordsToF32<ValT, kWords>::Convert(w, b);
#pragma unroll
            for (int i = 0; i < E; i += 2) MulAdd2(acc[i], acc[i + 1], b[i], b[i + 1], v, a.negZeros);
            if (meta & 0x100) {  // last entry of its row (warp-uniform)
                const int l = meta & 0xff;
                StoreSlice<OutT, E>(cRow0 + (long long)l * a.ldc, acc, old, alpha, beta);
#pragma unroll
                for (int i = 0; i < E; ++i) acc[i] = 0.0f;
                const unsigned rest = l < 31 ? liveMask & (0xfffffffeu << l) : 0u;
                if (beta != 0.0f && rest != 0) LoadOld<OutT, E>(cRow0 + (long long)(__ffs(rest) - 1) * a.ldc, old);
            }
        }
        __syncwarp();  // every lane is done with this buffer before a later batch is copied into it
    }
    if (failedAt >= 0) {
        // A wait ran out: this warp writes no more of C.  Give the copies still in flight (batches
        // failedAt .. failedAt + ahead) a bounded chance to land before the shared memory they
        // target is released.
        for (int k = failedAt; k <= failedAt + ahead && k < nBatches; ++k)
            (void)MbarWait(sBar + k % kStreamBuffers, (uint32_t)(k / kStreamBuffers) & 1u, a.waitCycles);
    }
}

// ---------------------------------------------------------------- int8 on the tensor cores

#include "int8_tensor.cuh"

// ---------------------------------------------------------------- repacking B

// Copies op(B) (k rows of n elements, any layout) into rows of `vecs` 16-byte pieces, zeros after element n.  One
// pass over B; worth it when B is read back often enough (see WorthRepacking).
template <typename ValT>
__global__ void __launch_bounds__(256) SpmmRepackRowsKernel(const ValT *__restrict__ B, long long ldb, long long k, int n,
                                                            int vecs, uint4 *__restrict__ out)
{
    b200sp::WaitForPrevious();
    constexpr int E = 16 / (int)sizeof(ValT);
    const long long total = k * vecs;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / vecs;
        const int c = (int)(i - r * vecs) * E;
        alignas(16) ValT v[E];
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = c + e < n ? __ldcs(B + r * ldb + c + e) : ValT(0);
        out[i] = *reinterpret_cast<const uint4 *>(v);
    }
}

// The same from a B whose columns are contiguous (element (r, j) at j * ldb + r), through a tile of 64 rows.
constexpr int kRepackRows = 64;
template <typename ValT>
__global__ void __launch_bounds__(256) SpmmRepackColsKernel(const ValT *__restrict__ B, long long ldb, long long k, int n,
                                                            int vecs, uint4 *__restrict__ out)
{
    b200sp::WaitForPrevious();
    constexpr int E = 16 / (int)sizeof(ValT);
    constexpr int kCols = 64;                            // columns per step
    constexpr int kVecs = kCols / E;
    __shared__ ValT tile[kCols][kRepackRows + 2 * 4 / sizeof(ValT)];  // rows two words apart: no bank is hit twice on the way out
    const long long r0 = (long long)blockIdx.x * kRepackRows;
    const int rIn = threadIdx.x & (kRepackRows - 1);
    for (int c0 = 0; c0 < vecs * E; c0 += kCols) {
#pragma unroll
        for (int c = threadIdx.x / kRepackRows; c < kCols; c += 256 / kRepackRows)
            tile[c][rIn] = (c0 + c < n && r0 + rIn < k) ? __ldcs(B + (c0 + c) * ldb + r0 + rIn) : ValT(0);
        __syncthreads();
        for (int i = threadIdx.x; i < kRepackRows * kVecs; i += 256) {
            const int v = i % kVecs, r = i / kVecs;
            if (r0 + r < k && c0 / E + v < vecs) {
                alignas(16) ValT w[E];
#pragma unroll
                for (int e = 0; e < E; ++e) w[e] = tile[v * E + e][r];
                out[(r0 + r) * vecs + c0 / E + v] = *reinterpret_cast<const uint4 *>(w);
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- generic path

struct GenericShape {
    long long m, n, ldb, ldc;
    int bRowMajor, cRowMajor, opB, kahan;
};

__device__ __forceinline__ long long BIndex(const GenericShape &g, long long c, long long j)
{
    // op(B)(c, j): same four cases as the golden SpmmCpuFp32 (spmm_test.cpp:142-151).
    if (!g.opB) return g.bRowMajor ? c * g.ldb + j : j * g.ldb + c;
    return g.bRowMajor ? j * g.ldb + c : c * g.ldb + j;
}

template <typename ValT, typename OutT>
__global__ void __launch_bounds__(256) SpmmGenericFloatKernel(const int32_t *__restrict__ rowPtr,
                                                               const int32_t *__restrict__ colInd,
                                                               const ValT *__restrict__ val,
                                                               const ValT *__restrict__ B, OutT *__restrict__ C,
                                                               GenericShape g, ScalarsF sc)
{
    b200sp::WaitForPrevious();
    const float alpha = sc.Alpha();
    const float beta = sc.Beta();
    const long long total = g.m * g.n;
    for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < total;
         w += (long long)gridDim.x * blockDim.x) {
        const long long r = w / g.n;
        const long long j = w - r * g.n;
        float acc = 0.0f, comp = 0.0f;
        const int e = rowPtr[r + 1];
        for (int p = rowPtr[r]; p < e; ++p) {
            const float b = ToF32(B[BIndex(g, colInd[p], j)]);
            if (g.kahan) AccumulateKahan(ToF32(val[p]), b, acc, comp);
            else acc = __fadd_rn(acc, __fmul_rn(ToF32(val[p]), b));
        }
        if (g.kahan) acc -= comp;
        const long long ci = g.cRowMajor ? r * g.ldc + j : j * g.ldc + r;
        float z = __fmul_rn(alpha, acc);
        if (beta != 0.0f) z = __fadd_rn(z, __fmul_rn(beta, ToF32(C[ci])));
        C[ci] = FromF32<OutT>(z);
    }
}

__global__ void __launch_bounds__(256) SpmmGenericInt8Kernel(const int32_t *__restrict__ rowPtr,
                                                              const int32_t *__restrict__ colInd,
                                                              const int8_t *__restrict__ val,
                                                              const int8_t *__restrict__ B, int32_t *__restrict__ C,
                                                              GenericShape g, ScalarsI sc)
{
    b200sp::WaitForPrevious();
    const int32_t alpha = sc.Alpha();
    const int32_t beta = sc.Beta();
    const long long total = g.m * g.n;
    for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < total;
         w += (long long)gridDim.x * blockDim.x) {
        const long long r = w / g.n;
        const long long j = w - r * g.n;
        int32_t acc = 0;
        const int e = rowPtr[r + 1];
        for (int p = rowPtr[r]; p < e; ++p)
            acc += (int32_t)val[p] * (int32_t)B[BIndex(g, colInd[p], j)];
        const long long ci = g.cRowMajor ? r * g.ldc + j : j * g.ldc + r;
        // int64 epilogue with saturation (reference spmm_kernel.cpp:251-266)
        long long wide = (long long)alpha * (long long)acc;
        if (beta != 0) wide += (long long)beta * (long long)C[ci];
        if (wide > 2147483647LL) wide = 2147483647LL;
        if (wide < -2147483648LL) wide = -2147483648LL;
        C[ci] = (int32_t)wide;
    }
}

// ---------------------------------------------------------------- host dispatch

template <typename S> S MakeScalars(const b200spScalars *s);
template <> ScalarsF MakeScalars<ScalarsF>(const b200spScalars *s)
{
    return {s->alpha_f, s->beta_f, static_cast<const float *>(s->alpha_dev), static_cast<const float *>(s->beta_dev)};
}
template <> ScalarsI MakeScalars<ScalarsI>(const b200spScalars *s)
{
    return {s->alpha_i, s->beta_i, static_cast<const int32_t *>(s->alpha_dev),
            static_cast<const int32_t *>(s->beta_dev)};
}

bool Aligned16(const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

#ifndef B200SP_SPMM_USE_STREAM
#define B200SP_SPMM_USE_STREAM 1
#endif
// Which of the two takes B rows of 512 or 1024 bytes.  A warp of the row stream sums its rows one after the other: that
// spares the chain of loads per row, which rows of few entries and a B far from the SMs cost most by, and needs rows enough for
// all warps; SpmmFastKernel spends fewer instructions per entry and shares out the rows above four times the mean.  bf16,
// N = 256, us by the stream and by SpmmFastKernel:
//   few rows: 1000 of 30 11 (a row per warp; 133 with 32) and 7, 16,000 of 32 on 16,000 columns 41 and 30, 16,000 of 12 on 1 M
//   28 and 26, 30,000 of 12 on 1 M 41 and 45;
//   B of up to 61 MB: 120,000 of 6 60 and 74, of 12 95 and 99, of 30 209 and 185, 800,000 of 4 226 and 354, of 30 1224 and 1085;
//   B above: 200,000 of 16 on as many columns 194 and 253, of 60 637 and 613, 800,000 of 30 1575 and 1915;
//   power-law rows: 60,000 of 16 204 and 100, 200,000 of 24 on 1 M columns 419 and 414, 250,000 of 8 270 and 234, 300,000 of 24
//   on 1 M 501 and 566, 800,000 of 4 367 and 465.
constexpr int64_t kStreamMinRows = 16384, kStreamMinSkewed = 262144, kStreamMaxMean = 16;
bool StreamPays(const b200spSpmmShape *sh, int32_t segments, int64_t rowBytes)
{
    if (gHostStreamExtraTx != 0) return true;  // the wait test is about the stream
    if (sh->m < kStreamMinRows) return false;
    if (sh->mid_units + (int64_t)segments > sh->m / 1000) return sh->m >= kStreamMinSkewed;
    return sh->k * rowBytes >= kBlockMinB || sh->nnz < kStreamMaxMean * sh->m;
}
bool ToRowStream(const b200spSpmmShape *sh, int32_t segments, int64_t rowBytes)  // of B and C in 16-byte aligned rows, not int8
{
    return !sh->kahan && (rowBytes == 512 || rowBytes == 1024) && StreamPays(sh, segments, rowBytes);
}

// The copy engine of an SM starts about one row copy per 20 clocks (measured: 16.8 M copies of
// 256 bytes took 1.25 ms on 148 SMs), so rows shorter than 512 bytes move faster through plain
// 128-bit loads and stay with SpmmFastKernel (256-byte rows, 64 per row of A: 1249 us against 265 us).

template <typename ValT, typename OutT, int kRowBytes, bool kUnits>
int LaunchRowStream(const StreamArgs<ValT, OutT> &sa, const FastArgs<ValT, OutT> &fa, BlockArgs ba, cudaStream_t stream)
{
    constexpr int kSmem = StreamShape<kRowBytes>::kCtaBytes;
    static bool configured[64] = {};  // per device: this instantiation uses kSmem bytes of dynamic shared memory
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return (int)cudaErrorInvalidDevice;
    if (!configured[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(SpmmRowStreamKernel<ValT, OutT, kRowBytes, kUnits>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
        if (e != cudaSuccess) return (int)e;
        configured[dev] = true;
    }
    const unsigned grid = (unsigned)(((long long)sa.m + sa.warpRows - 1) / sa.warpRows);
    const unsigned long long all = (unsigned long long)grid + (unsigned)ba.nUnits;
    ba.share = (((unsigned long long)(unsigned)ba.nUnits << 32) + all - 1) / all;  // rounded up: the last CTA's count is nUnits
    SpmmRowStreamKernel<ValT, OutT, kRowBytes, kUnits><<<(unsigned)all, kStreamThreads, kSmem, stream>>>(sa, fa, ba);
    b200sp_note_launches(1);
    return (int)cudaGetLastError();
}

// B rows contiguous in memory: (N, row-major) or (T, column-major).
bool RowsContiguous(int opB, int orderB) { return (opB != 0) == (orderB != 0); }

bool RowsOfWords(const b200spSpmmShape *sh, int valBytes)  // fp types only: int8 products take 16 bytes at a time
{
    return RowsContiguous(sh->op_b, sh->order_b) && (valBytes == 4 || (valBytes == 2 && sh->n % 2 == 0 && sh->ldb % 2 == 0));
}

// Bytes of a repacked B, 0 when its layout is the kernels' own.  From sizes and layout alone, never from the pointer:
// a caller may size the buffer before B exists (an unaligned B then goes to the generic kernel).
size_t RepackBytes(const b200spSpmmShape *sh, int valBytes)
{
    const int E = 16 / valBytes;
    if (RowsContiguous(sh->op_b, sh->order_b) && sh->n % E == 0 && sh->ldb % E == 0) return 0;
    return (size_t)sh->k * (size_t)((sh->n + E - 1) / E) * 16;
}

// Lanes side by side on a row of B of n elements, `perLane` of them a lane.
int LanesOf(int64_t n, int perLane)
{
    int lanes = 1;
    while (lanes < 32 && (int64_t)lanes * perLane < n) lanes <<= 1;
    return lanes;
}

// Repacking reads and writes k * n elements; the generic kernel reads nnz * n of them, with a load per product instead
// of one per 16 bytes, and a 32-byte sector per load where the columns of B are the contiguous ones: there the copy is
// fewer bytes from nnz = k * valBytes / 16 on (65,537 x 50,001 with 24 entries a row, fp16, N = 40: generic 257 us, copy
// and product 50 us).  Rows on 4-byte boundaries can be read where they are: 298,261 rows of 6 entries, fp32, N = 150, k =
// 737,797: 579 us with the copy, 408 us without; 415,892 power-law rows of 10, bf16, N = 50: 203 and 245 us.
bool WorthRepacking(const b200spSpmmShape *sh, int valBytes)
{
    if (RowsOfWords(sh, valBytes)) return sh->nnz >= 8 * sh->k;
    if (RowsContiguous(sh->op_b, sh->order_b)) return sh->nnz >= sh->k;
    return 16 * sh->nnz >= sh->k * valBytes;
}

// Products whose rows are a few entries, on a few columns of B that do not lie in 16-byte rows: a thread per output (the generic
// kernel) has nothing to wait for one after the other, and a copy of B or a lane group per row costs more than it saves
// unless the copy is read back very often.  Thread per output / lane groups, us:
//   columns of B contiguous: 500,000 rows of one entry, fp32, N = 1, 3 and 8: 8 / 32, 14 / 33 and 30 / 43; a million of three, 18 / 62,
//     42 / 64 and 113 / 86; 700,000 of three, N = 5: 50 / 62; of three on 43,750 columns, N = 3: 28 / 24; of one, N = 13: 63 / 54;
//   rows of B contiguous: a million rows of three, fp16, N = 1 and 3: 18 / 33 and 24 / 33;
//   int8: 500,000 rows of one entry, columns, N = 1, 8 and 33: 8 / 78, 30 / 94 and 171 / 132; 700,000 of four, N = 9 and 13: 111 / 137 and
//     162 / 148, rows, N = 9: 41 / 115.  Rows of up to 32 entries whose B rows are eight bytes at most go the same way: eight lanes of 16 columns join more
//     sums than they save loads (275,178 rows of 26, N = 8: 51 to 53 / 63).
bool FewEntries(const b200spSpmmShape *sh, int valBytes, int32_t segments)
{
    if (segments + sh->mid_units != 0) return false;
    const bool rows = RowsContiguous(sh->op_b, sh->order_b);
    if (valBytes == 1)
        return (sh->n <= 16 && sh->nnz <= 4 * sh->m && (rows || sh->nnz * sh->n <= 40 * sh->m)) ||
               (rows && sh->n <= 8 && sh->nnz <= 32 * sh->m);
    if (sh->nnz > 24 * sh->k) return false;
    return rows ? sh->n <= 4 && sh->nnz <= 4 * sh->m : sh->n <= 12 && sh->nnz * sh->n <= 16 * sh->m;
}

// Whether a product with this much room for a copy makes one.
bool Copies(const b200spSpmmShape *sh, int valBytes, int32_t segments, const void *plan)
{
    const size_t repack = RepackBytes(sh, valBytes);
    // A product of one wave of short rows takes less time than the second launch.
    const bool small = sh->m * sh->n < 148ll * 2048 && segments + sh->mid_units == 0 && sh->nnz <= 16 * sh->m;
    // The copy follows the plan (a multiple of 256 bytes) and is stored 16 bytes at a time; the plan itself may start on any word.
    return repack > 0 && sh->repack_bytes >= (int64_t)repack && WorthRepacking(sh, valBytes) && !small &&
           !FewEntries(sh, valBytes, segments) && plan != nullptr && Aligned16(plan);
}

// Whether an int8 product of rows whose columns ascend is one for the tensor cores.
//   - A is at least one twelfth full as it is written out, in rows of a multiple of 128 bytes, and takes at most 4 GB so.
//   - There is work enough for the two passes over it: 700 x 1500 at 0.2, N = 128, takes 6.1 us in lane groups and 12.7 on the tensor
//     cores, 1500 x 1100 at 0.18, N = 64, 8.1 and 13.2, 4000 x 1050 at 0.11, N = 9, in columns, 11.5 and 18.
//   - With rows enough to fill the SMs either way the two times are estimated, in us.  Lane groups cost by the entry, half as much
//     again for rows of 0 to twice the mean, and by the row: mostly so where a CTA takes one; where C is not in rows of
//     16-byte pieces, by the element of C too.  The tensor cores cost by the tile of 128 rows, of which an SM has one at a time.  Fitted
//     to 523 products of 3,000 to 800,000 rows, k = 64 to 4096, N = 16 to 512; for 514 the choice is within 10 % of the better
//     one.  Lane groups / tensor cores, us, 100,000 rows: 19 entries on 128 columns, N = 64: 25 / 65; 38 on 256, N = 256: 91 / 99; 60
//     on 200, N = 256: 124 / 100; 77 on 512, N = 64: 60 / 78, N = 128: 87 / 78; 154 on 1024, N = 16: 274 / 94, N = 128: 166 / 94; in columns,
//     200,000 rows, 50 on 256, N = 40: 100 / 141, N = 128: 174 / 167, 120 on 768, N = 40: 185 / 169, N = 128: 310 / 196.
// longest: entries of the longest row, 0 while it is not known.
bool TensorPays(const b200spSpmmShape *sh, long long longest)
{
    const bool plain = RowsContiguous(sh->op_b, sh->order_b) && sh->order_c == 0 && sh->n % 16 == 0;
    const long long denseCols = DenseCols(sh->k);
    if (sh->m == 0 || sh->k > kTcMaxK || 12 * sh->nnz < sh->m * denseCols || sh->m * denseCols > kTcMaxDense) return false;
    if (sh->nnz * sh->n < (plain ? 96ll : 24ll) << 20 || (!plain && sh->n < 24)) return false;
    const long long sms = b200sp_sm_count();
    if (sh->m < 64 * sms || sh->nnz > kLongRow * sh->m) return true;
    const double n = (double)sh->n, mean = (double)sh->nnz / (double)sh->m, rows = 1e-5 * (double)sh->m;
    const double spread = longest > 0 ? 0.525 * (1 + fmin((double)longest / mean, 2.0)) : 1.575;
    const int across = LanesOf(sh->n, 16);
    double lanes;
    if (!plain)
        lanes = 5 + 0.05 * n + rows * (8 + (sh->order_c != 0 ? 0.28 : 0.1) * n + spread * mean * (0.2 + 0.006 * fmax(n, 16.0 * across)));
    else if (sh->nnz >= 128 * sh->m && sh->m * across / 32 < 64 * sms)
        lanes = 4 + rows * fmax(265, 230 + 0.0069 * n * mean);
    else
        lanes = 4 + rows * spread * (8 + mean * (0.2 + 0.006 * n));
    const long long tiles = (sh->m + kTcRows - 1) / kTcRows * ((sh->n + kTcCols - 1) / kTcCols);
    const double turns = tiles <= sms ? 1 : (double)tiles / (double)sms + 0.65;  // of an SM: the last is short, on average
    const double share = fmin(ceil(n / kTcCols), kTcCluster);                    // CTAs that write the rows of A out together
    const double tile = 5.1 + 4.9 / share + (double)denseCols * (0.0033 + 0.0027 / share) +
                        4 / share * floor(mean / (32 * kTcWindows)) + (sh->order_c != 0 ? 0.027 * fmin(n, kTcCols) : 0);
    return lanes > tile * turns;
}

// Whether a CTA takes its 32 rows in order of their lengths (ctaRows, genRows: those it takes otherwise, of row- and of column-major
// C): the rows that a warp takes together wait for the longest of them.  It costs a pass over the lengths and fewer CTAs.  Never where the
// longest row has less than a quarter more entries than the mean.  Rows in their own order and so, us; ragged: rows of 0 to twice the mean,
// 150,000 of them where not said.
//   - Column-major C, whose CTAs have 32 rows anyway: ragged rows of 3, f16, N = 64, 53 and 43; of 40, 166 and 111.
//   - Eight lanes a row and more, with four CTAs of 32 rows for every SM (six where that takes four passes instead of one) and 1700
//     entries: ragged rows of 3, bf16, N = 128, 45 and 38, of 40, 182 and 138; power-law rows of 16, f32, N = 64, 103 and 94; but 30,000 rows of 6, 9.3
//     and 10.3, 20,000 of 24, 15.6 and 17.1.
//   - Four lanes, where 32 rows are one pass and a warp's eight rows are not shared out better: rows of like lengths, or long ones, in 16-bit
//     types from 8 entries on (f16, N = 32: ragged rows of 6 17.3 and 18.0, of 9 23.1 and 22.6, of 40 74 and 61; 4000 power-law rows of 16 22.6 and 27.1,
//     150,000 of 24 74 and 72), in fp32, whose rows of B take twice as long, from 64 (N = 16: ragged rows of 5 13.6 and 15.1, of 16 25.7
//     and 26.5, of 100 130 and 125).
bool OrderPays(const b200spSpmmShape *sh, long long longest, int valBytes, int ctaRows, int genRows)
{
    if (4 * longest * sh->m < 5 * sh->nnz) return false;
    if (sh->order_c != 0) return genRows == 32;
    const long long sms = b200sp_sm_count();
    const bool many = sh->m >= (ctaRows < 16 ? 6 : 4) * 32 * sms;
    if (ctaRows < 32) return many && sh->nnz >= 1700 * sms;
    return sh->nnz >= (valBytes == 2 ? 8 : 64) * sh->m && (longest * sh->m <= 4 * sh->nnz || (many && sh->nnz >= 24 * sh->m));
}

// What an analysed buffer holds after the plan: a copy of B (from a multiple of 256 bytes) and an A written out.
size_t ExtraBytes(const b200spSpmmShape *sh, int valBytes)
{
    const size_t repack = WorthRepacking(sh, valBytes) ? RepackBytes(sh, valBytes) : 0;
    if (valBytes != 1 || !TensorPays(sh, 0)) return repack;
    return AlignUp(repack, 256) + DenseBytes(sh->m, sh->k);
}

// Whether an int8 product with this much room, on rows found to ascend, writes A out.
bool OnTensorCores(const b200spSpmmShape *sh, const b200spSpmmFound &found, const void *plan)
{
    return found.ascending != 0 && TensorPays(sh, found.longest_row) && sh->repack_bytes >= (int64_t)ExtraBytes(sh, 1) && plan != nullptr &&
           Aligned16(plan);
}

template <typename ValT, typename OutT>
int LaunchGeneric(const int32_t *rowPtr, const int32_t *colInd, const void *val, const void *B, void *C,
                  const b200spSpmmShape *sh, const b200spScalars *s, cudaStream_t stream)
{
    GenericShape g{sh->m, sh->n, sh->ldb, sh->ldc, sh->order_b == 0, sh->order_c == 0, sh->op_b, sh->kahan};
    const long long total = sh->m * sh->n;
    if (total == 0) return 0;
    const long long want = (total + 255) / 256;
    const long long cap = (long long)b200sp_sm_count() * 32;
    const unsigned grid = (unsigned)(want < cap ? want : cap);
    const auto sc = MakeScalars<typename Arith<ValT>::Scalars>(s);
    cudaError_t e;
    if constexpr (std::is_same_v<ValT, int8_t>)
        e = b200sp::LaunchChained(SpmmGenericInt8Kernel, grid, 256, 0, stream, rowPtr, colInd, static_cast<const ValT *>(val),
                                  static_cast<const ValT *>(B), static_cast<OutT *>(C), g, sc);
    else
        e = b200sp::LaunchChained(SpmmGenericFloatKernel<ValT, OutT>, grid, 256, 0, stream, rowPtr, colInd,
                                  static_cast<const ValT *>(val), static_cast<const ValT *>(B), static_cast<OutT *>(C), g, sc);
    b200sp_note_launches(1);
    return (int)e;
}

// A matrix of bytes, `rows` rows of `cols` with `stride` bytes between them, in tiles of 128 rows by 128, 64 or 32 columns, swizzled
// over their whole width.
using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                 const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
bool ByteTiles(EncodeTiled encode, const void *at, long long rows, long long cols, long long stride, int tileCols, CUtensorMap *map)
{
    const cuuint64_t size[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)stride};
    const cuuint32_t box[2] = {(cuuint32_t)tileCols, 128}, step[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(at), size, strides, box, step,
                  CU_TENSOR_MAP_INTERLEAVE_NONE,
                  tileCols == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : tileCols == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// dense: DenseBytes(m, k), 16-byte aligned.  False, with nothing launched, where tensor maps or the shared memory are not to be had;
// else *error is the launches' status.
bool LaunchInt8Tensor(const FastArgs<int8_t, int32_t> &f, const b200spSpmmShape *sh, unsigned char *dense, cudaStream_t stream, int *error)
{
    *error = 0;
    static const EncodeTiled encode = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found{};
        const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found);
        return e == cudaSuccess && found == cudaDriverEntryPointSuccess ? reinterpret_cast<EncodeTiled>(fn) : nullptr;
    }();
    static std::atomic<bool> allowed[64] = {};  // per device: the kernel may use kTcSmem bytes of shared memory
    int dev = 0;
    if (encode == nullptr || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    if (!allowed[dev].load(std::memory_order_relaxed)) {
        if (cudaFuncSetAttribute(SpmmInt8TensorKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem) != cudaSuccess) {
            (void)cudaGetLastError();
            return false;
        }
        allowed[dev].store(true, std::memory_order_relaxed);
    }
    const long long denseCols = DenseCols(sh->k);
    TcArgs t{};
    t.dense = dense;
    t.odd = dense + AlignUp((size_t)sh->m * (size_t)denseCols, 256);
    t.rowPtr = f.rowPtr;
    t.colInd = f.colInd;
    t.val = f.val;
    t.B = f.B;
    t.C = f.C;
    t.m = f.m;
    t.n = f.n;
    t.chunks = (int)(denseCols / kTcDepth);
    t.ldb = f.ldb;
    t.cRow = f.cRow;
    t.cCol = f.cCol;
    t.cVectors = f.cCol == 1 && f.cRow % 4 == 0 && Aligned16(f.C);
    t.sc = f.sc;
    t.waitCycles = gHostStreamWaitCycles;
    t.extraTx = gHostStreamExtraTx;
    const long long rowTiles = (sh->m + kTcRows - 1) / kTcRows;
    // Narrower tiles where the widest leave half of the SMs without work.  Clusters of eight find their SMs free only where they are few:
    // 10 of them 19.7 us against 23.8 with 4 CTAs each, 16 of them 27.9 against 18.1.
    const int cluster = rowTiles <= 12 ? 2 * kTcCluster : kTcCluster;
    t.cols = kTcCols;
    while (t.cols > 32 && (2 * sh->n <= t.cols || (2 * sh->n <= cluster * t.cols &&
                                                   2 * rowTiles * ((sh->n + t.cols - 1) / t.cols) <= b200sp_sm_count())))
        t.cols /= 2;
    CUtensorMap mapA, mapB;
    if (!ByteTiles(encode, dense, sh->m, denseCols, denseCols, kTcDepth, &mapA) ||
        !ByteTiles(encode, f.B, sh->k, f.nB, f.ldb, t.cols, &mapB))
        return false;
    for (; t.firstCol < t.n; t.firstCol += cluster * t.cols) {  // a launch for every 512 or 1024 columns
        const int left = t.n - t.firstCol;
        t.colTiles = left < cluster * t.cols ? (left + t.cols - 1) / t.cols : cluster;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(rowTiles * t.colTiles));
        cfg.blockDim = dim3(kTcThreads);
        cfg.dynamicSmemBytes = kTcSmem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[2] = {};
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = (unsigned)t.colTiles;
        attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        b200sp_note_launches(1);
        *error = (int)cudaLaunchKernelEx(&cfg, SpmmInt8TensorKernel, t, mapA, mapB);
        if (*error != 0) break;
    }
    return true;
}

template <typename ValT, typename OutT>
int LaunchTyped(const int32_t *rowPtr, const int32_t *colInd, const void *val, const void *B, void *C,
                const b200spSpmmShape *sh, const b200spSpmmFound &found, const b200spScalars *s, void *plan, int32_t segments,
                cudaStream_t stream)
{
    constexpr bool kInt8 = std::is_same_v<ValT, int8_t>;
    constexpr int E = Pack<ValT>::kElems;
    const bool vectors = RowsContiguous(sh->op_b, sh->order_b) && sh->n % E == 0 && sh->ldb % E == 0 && Aligned16(B);
    const bool copy = Copies(sh, (int)sizeof(ValT), segments, plan);
    const bool words = !vectors && !copy && RowsOfWords(sh, (int)sizeof(ValT)) && reinterpret_cast<uintptr_t>(B) % 4 == 0;
    // By words, rows of up to four entries: 695,764 of them, fp32, N = 11: 70 us, by lane groups 79.
    const bool few = !vectors && (FewEntries(sh, (int)sizeof(ValT), segments) ||
                                  (words && sh->n <= 16 && sh->nnz <= 4 * sh->m && segments + sh->mid_units == 0));
    const bool bReady = !few && (vectors || words || copy);
    if (plan == nullptr || !bReady)
        return LaunchGeneric<ValT, OutT>(rowPtr, colInd, val, B, C, sh, s, stream);
    if (sh->m == 0 || sh->n == 0) return 0;
    const bool cPlain = !words && sh->order_c == 0 && sh->n % E == 0 && sh->ldc % E == 0 && Aligned16(C);
    const PlanLayout L = LayoutFor(sh->m, sh->nnz, sh->n);
    char *p = static_cast<char *>(plan);
    FastArgs<ValT, OutT> a;
    a.rowPtr = rowPtr;
    a.colInd = colInd;
    a.val = static_cast<const ValT *>(val);
    a.B = static_cast<const ValT *>(B);
    a.C = static_cast<OutT *>(C);
    a.m = (int)sh->m;
    a.n = (int)sh->n;
    a.nB = a.n;
    a.ldb = sh->ldb;
    a.ldc = sh->ldc;
    a.cRow = sh->order_c == 0 ? sh->ldc : 1;
    a.cCol = sh->order_c == 0 ? 1 : sh->ldc;
    a.sc = MakeScalars<typename Arith<ValT>::Scalars>(s);
    a.longRows = reinterpret_cast<const LongRow *>(p + L.offLong);
    a.segs = reinterpret_cast<const SegEntry *>(p + L.offSegs);
    a.segsEnd = a.segs + L.capSegs;
    a.counters = reinterpret_cast<int32_t *>(p + L.offCounters);
    a.partials = p + L.offPartials;
    a.arrivals = (int)ArrivalsPerRow(sh->n);
    a.rowLimit = sh->mid_units > 0 ? MidRowLimit(sh->m, sh->nnz, sh->n) : kLongRow;
    a.splitRows = 0;
    a.negZeros = kNegZeros;
    if (copy) {
        const int vecs = (int)((sh->n + E - 1) / E);
        auto *out = reinterpret_cast<uint4 *>(p + L.total);
        cudaError_t e;
        if (RowsContiguous(sh->op_b, sh->order_b)) {
            const long long want = (sh->k * vecs + 255) / 256;
            const long long cap = (long long)b200sp_sm_count() * 32;
            e = b200sp::LaunchChained(SpmmRepackRowsKernel<ValT>, (unsigned)(want < cap ? want : cap), 256, 0, stream, a.B,
                                      sh->ldb, sh->k, a.n, vecs, out);
        } else {
            e = b200sp::LaunchChained(SpmmRepackColsKernel<ValT>, (unsigned)((sh->k + kRepackRows - 1) / kRepackRows), 256, 0,
                                      stream, a.B, sh->ldb, sh->k, a.n, vecs, out);
        }
        b200sp_note_launches(1);
        if (e != cudaSuccess) return (int)e;
        a.B = reinterpret_cast<const ValT *>(out);
        a.ldb = (long long)vecs * E;
        a.nB = vecs * E;
    }
    int midUnits = sh->mid_units;
    int lanes_ = LanesOf(sh->n, E);
    // Rows of several tiles: half as wide a group where that leaves a fifth fewer lanes idle in the last one (bf16, N = 277,
    // 35,891 rows of 27: 162 us with 32 lanes, 122 with 16).  Narrower still loses more to rows of different lengths in one
    // warp than it gains, except by words, which wait for more loads (N = 150 above: 542, 460 and 408 us).
    if (!kInt8 && lanes_ == 32) {
        auto padded = [&](int l) { return (sh->n + l * E - 1) / (l * E) * l; };
        if (10 * padded(16) <= 8 * padded(32)) lanes_ = 16;
        if (words && 10 * padded(8) < 9 * padded(lanes_)) lanes_ = 8;
    }
    // Grid of SpmmFastKernel: CTAs for the units of long rows, for those of one row each, and for all rows.
    auto launchFast = [&](int longUnits, int midUnits, bool rowCtas, cudaStream_t st) {
        const int units = longUnits + midUnits;
        cudaError_t err = cudaSuccess;
        auto launch = [&]<int kLanes>() {
            using Shape = FastShape<ValT, kLanes>;
            constexpr int kPieces = UnitShape<kLanes>::kPieces;
            a.longUnits = longUnits;
            a.nUnits = units;
            a.slices = ((a.nB + E - 1) / E + kPieces - 1) / kPieces;
            const long long unitCtas = kInt8 ? units : ((long long)units * a.slices + kWarps - 1) / kWarps;
            a.unitCtas = (int)unitCtas;
            a.genRows = sh->m < 2ll * Shape::kGenRows * b200sp_sm_count() ? Shape::kCtaRows : Shape::kGenRows;
            const bool byLength = Shape::kMayOrder && rowCtas && OrderPays(sh, found.longest_row, (int)sizeof(ValT), Shape::kCtaRows, a.genRows);
            // int8, where rows above four times the mean (which units would take in other types) or few rows are waited for; N = 32 / 64, us
            // straight and as a loop: power-law rows, 20,000 of 30, 50 / 81 and 40 / 67, 100,000 of 40, 84 / 131 and 76 / 117; 3,000
            // ragged rows of 60, 9.8 / 15.4 and 8.3 / 12.7; but 100,000 equal rows of 40, 31 / 42 and 35 / 43, 20,000 of 150, a CTA each, 57 / 58 and 59 / 61.
            const bool loop = Shape::kMayLoop && cPlain && rowCtas &&
                              (sh->mid_units > 0 || (!a.splitRows && sh->m < 4ll * Shape::kCtaRows * b200sp_sm_count()));
            if (loop) a.genRows = Shape::kCtaRows;
            const long long rows = a.splitRows ? 1 : byLength ? 32 : sh->order_c == 0 ? Shape::kCtaRows : a.genRows;
            const long long grid = unitCtas + (rowCtas ? (sh->m + rows - 1) / rows : 0);
            if (grid == 0) return;
            auto go = [&](auto kernel) { err = b200sp::LaunchChained(kernel, (unsigned)grid, kThreads, 0, st, a); };
            auto pick = [&]<bool kKahan, bool kOrdered>() {
                if (cPlain) return go(SpmmFastKernel<ValT, OutT, kKahan, kLanes, kPlain, kOrdered>);
                // Kernels that read C in eights, where beta may be other than 0: into a column-major C only if hardly any of a tile's columns lie past
                // the last one, or rows are long; these take part in every batch.  Time without them by time with them, 100,000 to 900,000 rows of 2 to
                // 60, beta = 0.5: row-major N = 3 to 203 0.95 to 1.44, two thirds above 1.05; column-major fp16 / fp32, N = 5 0.89 to 1.13 / 0.88 to
                // 1.02, 24 0.93 to 1.02 / 0.97 to 1.16, 33 0.85 to 1.08 / 0.90 to 1.03, 60 0.97 to 1.18 / 1.03 to 1.23, 72 0.86 to 1.05 / 0.97 to 1.05, 100
                // 0.93 to 1.06 / 0.99 to 1.17, 128 0.98 to 1.17 / 1.02 to 1.27, 200 0.98 to 1.22 / 1.01 to 1.20.  Compensated sums lose up to 5 %
                // and gain up to 10: not worth the kernels.
                if constexpr (!kInt8 && !kKahan) {
                    const long long tileCols = kLanes * (16 / (int)sizeof(ValT)), padded = (sh->n + tileCols - 1) / tileCols * tileCols;
                    const bool adds = (s->beta_dev != nullptr || s->beta_f != 0.0f) &&
                                      (sh->order_c == 0 || 16 * sh->n >= 15 * padded || sh->n * (long long)sizeof(ValT) >= 384);
                    if (words && adds) return go(SpmmFastKernel<ValT, OutT, kKahan, kLanes, kAnyCWordsAdd, kOrdered>);
                    if (!words && adds) return go(SpmmFastKernel<ValT, OutT, kKahan, kLanes, kAnyCAdd, kOrdered>);
                }
                if constexpr (!kInt8)
                    if (words) return go(SpmmFastKernel<ValT, OutT, kKahan, kLanes, kAnyCWords, kOrdered>);
                go(SpmmFastKernel<ValT, OutT, kKahan, kLanes, kAnyC, kOrdered>);
            };
            auto pickOrder = [&]<bool kKahan>() {
                if constexpr (Shape::kMayOrder)
                    if (byLength) return pick.template operator()<kKahan, true>();
                if constexpr (Shape::kMayLoop)
                    if (loop) return go(SpmmFastKernel<ValT, OutT, kKahan, kLanes, kPlain, true>);
                pick.template operator()<kKahan, false>();
            };
            if constexpr (std::is_same_v<ValT, float>) {
                if (sh->kahan) pickOrder.template operator()<true>();
                else pickOrder.template operator()<false>();
            } else {
                pickOrder.template operator()<false>();
            }
            b200sp_note_launches(1);
        };
        switch (lanes_) {
            case 1: launch.template operator()<1>(); break;
            case 2: launch.template operator()<2>(); break;
            case 4: launch.template operator()<4>(); break;
            case 8: launch.template operator()<8>(); break;
            case 16: launch.template operator()<16>(); break;
            default: launch.template operator()<32>(); break;
        }
        return err;
    };
    if constexpr (kInt8) {
        if (OnTensorCores(sh, found, plan)) {
            auto *dense = reinterpret_cast<unsigned char *>(p + L.total + ExtraBytes(sh, 1) - DenseBytes(sh->m, sh->k));
            int error = 0;
            if (LaunchInt8Tensor(a, sh, dense, stream, &error)) return error;
        }
        if (lanes_ <= 4) {  // 16 to 64 entries of a row are in flight as it is
            a.rowLimit = kLongRow;
            midUnits = 0;
        }
        // Integer sums may be regrouped: where a warp per row would not fill the SMs and rows are long enough to be
        // shared, a CTA takes a row (4096 rows of 410 entries, N = 512: 104 us with a warp per row, 74 us so).
        a.splitRows = cPlain && sh->nnz >= 128 * sh->m && sh->m * lanes_ / 32 < 64ll * b200sp_sm_count();
        return (int)launchFast(segments, midUnits, true, stream);
    } else {
        if (!cPlain) return (int)launchFast(segments, midUnits, true, stream);
        // B rows of 512 / 1024 bytes: rows of up to kLongRow entries go to the row-stream kernel,
        // and SpmmFastKernel is launched for its segment CTAs only.
        const long long rowBytes = sh->n * (long long)sizeof(ValT);
        const bool stream_ = ToRowStream(sh, segments, rowBytes);
        // Long rows by column blocks of B (found applicable by b200sp_spmm_analyze_blocks) instead of by segments.
        const bool byBlocks = sh->block_units > 0 && sh->long_rows > 0 && !sh->kahan && rowBytes >= kBlockMinRowBytes &&
                              sh->block_units <= L.capBlockSlots;
        if (byBlocks) segments = 0;
        if (stream_) {  // which has enough copies in flight for any row it takes
            a.rowLimit = kLongRow;
            midUnits = 0;
        }
        // With both kernels to run, the long rows (few CTAs, each with much work) are forked onto the side stream
        // first and the other rows' kernel shares the SMs with them.
        b200sp::SideLanes *lanes = nullptr;
        cudaStream_t longStream = stream;
        BlockArgs ba{};
        if (byBlocks) {
            ba.nUnits = sh->block_units;
            ba.nLong = sh->long_rows;
            ba.units = reinterpret_cast<const BlockUnit *>(p + L.offUnits);
            ba.rowSlots = reinterpret_cast<const int2 *>(p + L.offRowSlots);
            ba.partials = reinterpret_cast<float *>(p + L.offBlockPartials);
        }
        auto sumLongRows = [&](cudaStream_t st) {
            const long long warps = (long long)ba.nLong * ((sh->n + 31) / 32);
            b200sp_note_launches(1);
            return b200sp::LaunchChained(SpmmLongSumKernel<OutT, FastArgs<ValT, OutT>>, (unsigned)((warps + 7) / 8), 256, 0, st, a, ba);
        };
        if ((stream_ && segments > 0) || (byBlocks && !stream_)) {
            lanes = b200sp::GetSideLanes();
            if (lanes != nullptr) {
                if (cudaEventRecord(lanes->fork, stream) != cudaSuccess ||
                    cudaStreamWaitEvent(lanes->stream[0], lanes->fork, 0) != cudaSuccess)
                    return (int)cudaGetLastError();
                longStream = lanes->stream[0];
            }
            if (byBlocks) {
                const unsigned grid = (unsigned)(((long long)ba.nUnits + kBlockWarps - 1) / kBlockWarps);
                SpmmLongBlockKernel<ValT, OutT><<<grid, 32 * kBlockWarps, 0, longStream>>>(a, ba);
                b200sp_note_launches(1);
                if (cudaGetLastError() != cudaSuccess || sumLongRows(longStream) != cudaSuccess) return (int)cudaErrorLaunchFailure;
            } else if (lanes != nullptr) {
                if (launchFast(segments, 0, false, longStream) != cudaSuccess) return (int)cudaErrorLaunchFailure;
                segments = 0;
            }
            if (lanes != nullptr && cudaEventRecord(lanes->join[0], longStream) != cudaSuccess)
                return (int)cudaErrorLaunchFailure;
        }
        if (stream_) {
            StreamArgs<ValT, OutT> sa;
            sa.rowPtr = rowPtr;
            sa.colInd = colInd;
            sa.val = a.val;
            sa.B = a.B;
            sa.C = a.C;
            sa.m = a.m;
            sa.rowLimit = a.rowLimit;
            // Eight rows a warp, fewer where that leaves less than two waves of some 24 warps an SM: 200,000 rows of 16, 32 / 16 / 8 / 4 / 2
            // a warp, 214 / 200 / 194 / 195 / 208 us, 30,000 of 12 68 / 48 / 46 / 41 / -, 2 M power-law rows 2255 / 2245 / 2230 / 2300 / -.
            sa.warpRows = 8;
            while (sa.warpRows > 1 && sh->m < sa.warpRows * 48ll * b200sp_sm_count()) sa.warpRows /= 2;
            sa.ldb = a.ldb;
            sa.ldc = sh->ldc;
            sa.sc = a.sc;
            sa.negZeros = kNegZeros;
            sa.waitCycles = gHostStreamWaitCycles;
            sa.extraTx = gHostStreamExtraTx;
            auto launchStream = [&]<bool kUnits>() {
                return rowBytes == 512 ? LaunchRowStream<ValT, OutT, 512, kUnits>(sa, a, ba, stream)
                                       : LaunchRowStream<ValT, OutT, 1024, kUnits>(sa, a, ba, stream);
            };
            const int rc = ba.nUnits > 0 ? launchStream.template operator()<true>() : launchStream.template operator()<false>();
            if (rc != 0) return rc;
            if (byBlocks && sumLongRows(stream) != cudaSuccess) return (int)cudaErrorLaunchFailure;
        }
        // What is left for SpmmFastKernel on the caller's stream: the segment CTAs unless they were forked (or
        // replaced by the column-block kernel), and the rows of up to kLongRow entries unless the row-stream
        // kernel took them.
        if (launchFast(segments, midUnits, !stream_, stream) != cudaSuccess) return (int)cudaErrorLaunchFailure;
        if (lanes != nullptr)  // the long rows are already running beside: join them
            return (int)cudaStreamWaitEvent(stream, lanes->join[0], 0);
        return 0;
    }
}

}  // namespace

extern "C" {

int b200sp_spmm_stream_error(void)
{
    int flag = 0;
    if (cudaMemcpyFromSymbol(&flag, gStreamError, sizeof(flag)) != cudaSuccess) return -1;
    return flag;
}

int b200sp_spmm_stream_error_clear(void)
{
    const int zero = 0;
    return (int)cudaMemcpyToSymbol(gStreamError, &zero, sizeof(zero));
}

void b200sp_spmm_stream_wait_test(long long wait_cycles, unsigned extra_tx)
{
    gHostStreamWaitCycles = wait_cycles > 0 ? wait_cycles : kStreamWaitCycles;
    gHostStreamExtraTx = extra_tx;
}

int b200sp_spmm_to_row_stream(const b200spSpmmShape *shape, int val_type, int32_t segments)
{
    const int bytes = val_type == B200SP_F32 ? 4 : 2;
    return shape != nullptr && val_type != B200SP_I8 && ToRowStream(shape, segments, shape->n * bytes) ? 1 : 0;
}

size_t b200sp_spmm_plan_bytes(int64_t rows, int64_t nnz, int64_t n) { return LayoutFor(rows, nnz, n).total; }

static int BytesOf(int val_type) { return val_type == B200SP_F32 ? 4 : val_type == B200SP_I8 ? 1 : 2; }

size_t b200sp_spmm_repack_bytes(const b200spSpmmShape *shape, int val_type)
{
    return WorthRepacking(shape, BytesOf(val_type)) ? RepackBytes(shape, BytesOf(val_type)) : 0;
}

size_t b200sp_spmm_operand_bytes(const b200spSpmmShape *shape, int val_type) { return ExtraBytes(shape, BytesOf(val_type)); }

int b200sp_spmm_copies(const b200spSpmmShape *shape, int val_type, int32_t segments, const void *plan)
{
    return b200sp_spmm_copies_found(shape, nullptr, val_type, segments, plan);
}

int b200sp_spmm_copies_found(const b200spSpmmShape *shape, const b200spSpmmFound *found, int val_type, int32_t segments,
                             const void *plan)
{
    const bool dense = found != nullptr && val_type == B200SP_I8 && OnTensorCores(shape, *found, plan);
    return dense || Copies(shape, BytesOf(val_type), segments, plan) ? 1 : 0;
}

int b200sp_spmm_columns_ascend(const int32_t *row_ptr, const int32_t *col_ind, const b200spSpmmShape *shape, int val_type,
                               void *plan, size_t plan_bytes, b200spSpmmFound *found, void *stream)
{
    if (found == nullptr) return (int)cudaErrorInvalidValue;
    found->ascending = 0;
    if (val_type != B200SP_I8 || !TensorPays(shape, found->longest_row) || col_ind == nullptr) return 0;
    const PlanLayout L = LayoutFor(shape->m, shape->nnz, shape->n);
    if (plan == nullptr || plan_bytes < L.total) return (int)cudaErrorInvalidValue;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int32_t *flag = reinterpret_cast<int32_t *>(static_cast<char *>(plan) + L.offCounts) + 6;  // zero since the analysis of the rows
    const long long want = (shape->m + 7) / 8, cap = (long long)b200sp_sm_count() * 8;
    SpmmAscendingKernel<<<(unsigned)(want < cap ? want : cap), 256, 0, st>>>(row_ptr, col_ind, (int)shape->m, flag);
    b200sp_note_launches(1);
    int32_t bad = 1;
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&bad, flag, sizeof(bad), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return (int)e;
    found->ascending = bad == 0;
    return 0;
}

int b200sp_spmm_analyze(const int32_t *row_ptr, int64_t rows, int64_t nnz, int64_t n, void *plan,
                        size_t plan_bytes, int32_t *segments, void *stream)
{
    int32_t mid = 0;
    return b200sp_spmm_analyze_rows(row_ptr, rows, nnz, n, plan, plan_bytes, segments, &mid, nullptr, stream);
}

int b200sp_spmm_analyze_units(const int32_t *row_ptr, int64_t rows, int64_t nnz, int64_t n, void *plan,
                              size_t plan_bytes, int32_t *segments, int32_t *mid_units, void *stream)
{
    return b200sp_spmm_analyze_rows(row_ptr, rows, nnz, n, plan, plan_bytes, segments, mid_units, nullptr, stream);
}

int b200sp_spmm_analyze_rows(const int32_t *row_ptr, int64_t rows, int64_t nnz, int64_t n, void *plan,
                             size_t plan_bytes, int32_t *segments, int32_t *mid_units, b200spSpmmFound *found,
                             void *stream)
{
    const PlanLayout L = LayoutFor(rows, nnz, n);
    if (plan == nullptr || segments == nullptr || mid_units == nullptr || plan_bytes < L.total) return (int)cudaErrorInvalidValue;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    char *p = static_cast<char *>(plan);
    cudaError_t e = cudaMemsetAsync(p + L.offCounts, 0, 256, st);
    if (e != cudaSuccess) return (int)e;
    if (rows > 0) {
        const long long want = (rows + 255) / 256;
        const long long cap = (long long)b200sp_sm_count() * 16;
        SpmmFindLongRowsKernel<<<(unsigned)(want < cap ? want : cap), 256, 0, st>>>(
            row_ptr, (int)rows, MidRowLimit(rows, nnz, n), (int)ArrivalsPerRow(n), (int)L.capSegs,
            reinterpret_cast<int32_t *>(p + L.offCounts),
            reinterpret_cast<LongRow *>(p + L.offLong), reinterpret_cast<SegEntry *>(p + L.offSegs),
            reinterpret_cast<int32_t *>(p + L.offCounters));
        b200sp_note_launches(1);
        e = cudaGetLastError();
        if (e != cudaSuccess) return (int)e;
    }
    int32_t counts[8] = {};
    e = cudaMemcpyAsync(counts, p + L.offCounts, sizeof(counts), cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess) return (int)e;
    e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return (int)e;
    *segments = counts[1];
    *mid_units = counts[5];
    if (found != nullptr) *found = {counts[7], 0};
    return 0;
}

int b200sp_spmm_analyze_blocks(const int32_t *row_ptr, const int32_t *col_ind, int64_t rows, int64_t cols,
                               int64_t nnz, int64_t n, int64_t b_row_bytes, void *plan, size_t plan_bytes,
                               int32_t *block_units, int32_t *long_rows, void *stream)
{
    const PlanLayout L = LayoutFor(rows, nnz, n);
    if (plan == nullptr || block_units == nullptr || long_rows == nullptr || plan_bytes < L.total)
        return (int)cudaErrorInvalidValue;
    *block_units = 0;
    *long_rows = 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    char *p = static_cast<char *>(plan);
    // counts: long rows, their units, partial slots of the long rows' units, "a long row's columns do not ascend", units (and
    // the rows that are a unit each)
    int32_t counts[5] = {0, 0, 0, 0, 0};
    cudaError_t e = cudaMemcpyAsync(counts, p + L.offCounts, sizeof(counts), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return (int)e;
    const int nLong = counts[0];
    *long_rows = nLong;
    if (nLong <= 0 || col_ind == nullptr || L.capBlockSlots == 0 || b_row_bytes < kBlockMinRowBytes ||
        cols * b_row_bytes < kBlockMinB)
        return 0;
    long long blocks = (cols * b_row_bytes + kBlockBytes - 1) / kBlockBytes;
    if (blocks > kMaxBlocks) blocks = kMaxBlocks;
    if (blocks < 2) return 0;
    const long long blockCols = (cols + blocks - 1) / blocks;
    int32_t *countsDev = reinterpret_cast<int32_t *>(p + L.offCounts);
    int32_t *meta = reinterpret_cast<int32_t *>(p + L.offBlockMeta);
    int2 *rowSlots = reinterpret_cast<int2 *>(p + L.offRowSlots);
    int32_t *cuts = reinterpret_cast<int32_t *>(p + L.offCuts);
    e = cudaMemsetAsync(meta, 0, sizeof(int32_t) * 3 * kMaxBlocks, st);
    if (e != cudaSuccess) return (int)e;
    SpmmCutBlocksKernel<<<(unsigned)((nLong + 7) / 8), 256, 0, st>>>(
        row_ptr, col_ind, reinterpret_cast<const LongRow *>(p + L.offLong), nLong, blockCols, (int)blocks, cuts,
        rowSlots, meta, countsDev + 3);
    SpmmBlockScanKernel<<<1, 1024, 0, st>>>(rowSlots, nLong, meta, (int)blocks, countsDev + 4);
    SpmmFillUnitsKernel<<<(unsigned)((nLong + 7) / 8), 256, 0, st>>>(
        cuts, rowSlots, nLong, (int)blocks, meta, reinterpret_cast<BlockUnit *>(p + L.offUnits),
        (int)(L.capBlockSlots < INT32_MAX ? L.capBlockSlots : INT32_MAX));
    b200sp_note_launches(3);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(counts, countsDev, sizeof(counts), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return (int)e;
    // Unsorted long rows, or more units than the plan has partial rows for: the segments stay in charge.
    if (counts[3] == 0 && counts[4] > 0 && counts[4] <= L.capBlockSlots) *block_units = counts[4];
    return 0;
}

int b200sp_spmm_launch(const int32_t *row_ptr, const int32_t *col_ind, const void *val, const void *B, void *C,
                       const b200spSpmmShape *shape, const b200spScalars *scalars, int val_type, int out_type,
                       void *plan, int32_t segments, void *stream)
{
    return b200sp_spmm_launch_found(row_ptr, col_ind, val, B, C, shape, nullptr, scalars, val_type, out_type, plan, segments, stream);
}

int b200sp_spmm_launch_found(const int32_t *row_ptr, const int32_t *col_ind, const void *val, const void *B, void *C,
                             const b200spSpmmShape *shape, const b200spSpmmFound *found, const b200spScalars *scalars,
                             int val_type, int out_type, void *plan, int32_t segments, void *stream)
{
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto go = [&]<typename ValT, typename OutT>() {
        return LaunchTyped<ValT, OutT>(row_ptr, col_ind, val, B, C, shape, found != nullptr ? *found : b200spSpmmFound{}, scalars, plan, segments,
                                         st);
    };
    if (val_type == B200SP_F32 && out_type == B200SP_F32) return go.template operator()<float, float>();
    if (val_type == B200SP_F16 && out_type == B200SP_F16) return go.template operator()<__half, __half>();
    if (val_type == B200SP_BF16 && out_type == B200SP_BF16) return go.template operator()<__nv_bfloat16, __nv_bfloat16>();
    if (val_type == B200SP_BF16 && out_type == B200SP_F32) return go.template operator()<__nv_bfloat16, float>();
    if (val_type == B200SP_I8 && out_type == B200SP_I32) return go.template operator()<int8_t, int32_t>();
    return (int)cudaErrorInvalidValue;
}

}  // extern "C"
