// SpMVOp kernels for sm_100a: Z = alpha * A * X + beta * Y with doubly compensated row sums.
//
// The reference gives every row to one SIMT thread, which walks the row's entries in CSR order
// with Priest's doubly compensated dot product: three accumulators hi + md + lo, the product split
// into its rounded value and its rounding error by one fused multiply-add
// (sparse/spmv_op/arch35/spmv_op_kernel.cpp:88-127), and combines
//     z = fma(alpha, hi, fma(alpha, md + lo, beta * y))                         (:172-176).
// Here a row gets G lanes (G a power of two up to 32): every lane runs exactly that recurrence
// over the entries lane, lane + G, lane + 2G, ... and the G triples are then joined pairwise by
// error-free additions on a fixed butterfly, so a row's result does not depend on scheduling and is
// the same bits on every run; the final combination is the reference's.  With G = 1 the arithmetic
// is the reference's, operation for operation.
//
// SpmvOpRowsKernel (ALG1, and ALG2 where row lengths are alike): rows up to 16 * G entries get G lanes, longer ones a
// warp, in row order; G comes from the mean length.
// SpmvOpClassesKernel (ALG2 on skewed lengths): the plan orders the rows by descending length class (class c: lengths that
// need c bits; a histogram and a scatter, the counterpart of the reference's reorder / bin_edge tables,
// spmv_op_kernel.cpp:425-540), and a class gets as many lanes per row as leave each of them four to eight entries; rows of
// 512 entries and more get a CTA.  One grid, longest rows first.
// SpmvOpLongRowsKernel (ALG2): rows that either grid would wait for, a wider CTA each, beside it on the side stream.
#include <cstdint>

#include <cuda_runtime.h>

#include "b200sp_kernels.h"
#include "../common/chained.cuh"
#include "../common/side_stream.h"

namespace {

constexpr int kClasses = B200SP_SPMVOP_CLASSES;
constexpr int kLongBits = 10;  // rows of this many bits of length and more (512 entries) are long
constexpr int kThreads = 128;

inline size_t AlignUp(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct OpPlanLayout {
    size_t offReorder, offHist, total;
};
inline OpPlanLayout OpLayoutFor(int64_t rows)
{
    OpPlanLayout L;
    L.offReorder = 0;
    L.offHist = AlignUp(sizeof(int32_t) * (size_t)(rows > 0 ? rows : 1), 256);
    L.total = L.offHist + 256;  // kClasses cursors
    return L;
}

struct Triple {
    float hi, md, lo;
};
// One step of the reference recurrence (spmv_op_kernel.cpp:101-122).
__device__ __forceinline__ void PriestStep(Triple &t, float val, float xv)
{
    const float prod = __fmul_rn(val, xv);
    const float pi = __fmaf_rn(val, xv, -prod);
    const float s1 = __fadd_rn(t.hi, prod);
    const float v1 = __fsub_rn(s1, t.hi);
    const float e1 = __fadd_rn(__fsub_rn(t.hi, __fsub_rn(s1, v1)), __fsub_rn(prod, v1));
    t.hi = s1;
    const float ee = __fadd_rn(e1, pi);
    const float s2 = __fadd_rn(t.md, ee);
    const float v2 = __fsub_rn(s2, t.md);
    const float e2 = __fadd_rn(__fsub_rn(t.md, __fsub_rn(s2, v2)), __fsub_rn(ee, v2));
    t.md = s2;
    t.lo = __fadd_rn(t.lo, e2);
}

__device__ __forceinline__ void TwoSum(float a, float b, float &s, float &e)
{
    s = __fadd_rn(a, b);
    const float v = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, v)), __fsub_rn(b, v));
}

// a += b without losing what the additions round away.
__device__ __forceinline__ void JoinTriples(Triple &a, const Triple &b)
{
    float hi, e1, md, e2, md2, e3;
    TwoSum(a.hi, b.hi, hi, e1);
    TwoSum(a.md, b.md, md, e2);
    TwoSum(md, e1, md2, e3);
    a.hi = hi;
    a.md = md2;
    a.lo = __fadd_rn(__fadd_rn(a.lo, b.lo), __fadd_rn(e2, e3));
}

__device__ __forceinline__ long long LoadOffset(const void *rowOffsets, bool is64, long long i)
{
    return is64 ? static_cast<const long long *>(rowOffsets)[i] : (long long)static_cast<const int32_t *>(rowOffsets)[i];
}

struct OpArgs {
    const void *rowOffsets;
    const int32_t *colInd;
    const float *val;
    const float *x;
    const float *y;
    float *z;
    const int32_t *reorder;  // rows by descending length class (SpmvOpClassesKernel)
    long long rows;
    int indexBase;
    float alpha, beta;
    const float *alphaDev, *betaDev;
};

__device__ __forceinline__ float Combine(const Triple &t, float alpha, float betaY)  // spmv_op_kernel.cpp:172-176
{
    const float corr = __fadd_rn(t.md, t.lo);
    return __fmaf_rn(alpha, t.hi, __fmaf_rn(alpha, corr, betaY));
}

// kCount entries p, p + step, ...: all of them requested before the first is used.  kWhole: none of them lies beyond e.
template <int kCount, bool kWhole>
__device__ __forceinline__ void SumSome(const OpArgs &a, Triple &t, long long p, long long e, int step)
{
    int c[kCount];
    float v[kCount], xv[kCount];
#pragma unroll
    for (int u = 0; u < kCount; ++u) {
        const bool in = kWhole || p + u * step < e;
        c[u] = in ? __ldcs(a.colInd + p + u * step) - a.indexBase : 0;
        v[u] = in ? __ldcs(a.val + p + u * step) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < kCount; ++u) xv[u] = kWhole || p + u * step < e ? __ldg(a.x + c[u]) : 0.0f;
#pragma unroll
    for (int u = 0; u < kCount; ++u)
        if (kWhole || p + u * step < e) PriestStep(t, v[u], xv[u]);
}

// Entries first, first + step, ... below e, in that order, four in flight; kLong: eight as long as there are so many.
template <bool kLong = false>
__device__ __forceinline__ Triple SumEntries(const OpArgs &a, long long first, long long e, int step)
{
    Triple t{0.0f, 0.0f, 0.0f};
    long long p = first;
    if constexpr (kLong)
        for (; p + 7 * step < e; p += 8 * step) SumSome<8, true>(a, t, p, e, step);
    for (; p + 3 * step < e; p += 4 * step) SumSome<4, true>(a, t, p, e, step);
    if (p < e) SumSome<3, false>(a, t, p, e, step);
    return t;
}

template <int kLanes> __device__ __forceinline__ void JoinLanes(Triple &t)  // lane 0 of every group gets the sum
{
#pragma unroll
    for (int off = kLanes >> 1; off > 0; off >>= 1) {
        Triple o;
        o.hi = __shfl_down_sync(0xffffffffu, t.hi, off, kLanes);
        o.md = __shfl_down_sync(0xffffffffu, t.md, off, kLanes);
        o.lo = __shfl_down_sync(0xffffffffu, t.lo, off, kLanes);
        JoinTriples(t, o);  // lanes >= off of a group compute values nobody reads
    }
}

// A row per CTA: thread t runs the recurrence on entries t, t + kRowThreads, ...; the lanes of a warp are joined on the
// butterfly, then warp 0 joins the warps' triples the same way: a fixed shape again.
template <bool kIs64, int kRowThreads>
__device__ __forceinline__ void LongRow(const OpArgs &a, long long row, float alpha, float beta)
{
    __shared__ Triple sWarp[kRowThreads / 32];
    const int tid = threadIdx.x;
    const long long s = LoadOffset(a.rowOffsets, kIs64, row) - a.indexBase;
    const long long e = LoadOffset(a.rowOffsets, kIs64, row + 1) - a.indexBase;
    float yOld = 0.0f;
    if (tid == 0 && beta != 0.0f) yOld = a.y[row];
    Triple t = SumEntries<true>(a, s + tid, e, kRowThreads);
    JoinLanes<32>(t);
    if ((tid & 31) == 0) sWarp[tid >> 5] = t;
    __syncthreads();
    if (tid < 32) {
        Triple w = tid < kRowThreads / 32 ? sWarp[tid] : Triple{0.0f, 0.0f, 0.0f};
        JoinLanes<kRowThreads / 32>(w);
        if (tid == 0) a.z[row] = Combine(w, alpha, __fmul_rn(beta, yOld));
    }
}

// Rows so long that a grid of lane groups or of CTAs of kThreads would wait for them: wider CTAs, on the side stream (see
// OutlierBits).  The rows come from the front of the row order.
template <bool kIs64, int kRowThreads>
__global__ void __launch_bounds__(kRowThreads) SpmvOpLongRowsKernel(const OpArgs a, int first)
{
    const float alpha = a.alphaDev ? *a.alphaDev : a.alpha;
    const float beta = a.betaDev ? *a.betaDev : a.beta;
    LongRow<kIs64, kRowThreads>(a, a.reorder[first + blockIdx.x], alpha, beta);
}

// Light on registers and without barriers: it lives on warps in flight (the gathers of x go to L2, one sector per clock and
// SM).  CTAs of 128 threads: 466,673 rows of 51 entries 69 us, with 256 threads 78.
template <int G, bool kIs64>
__global__ void __launch_bounds__(kThreads, 12) SpmvOpRowsKernel(const OpArgs a, long long outlier)  // rows from there on are others' work
{
    b200sp::WaitForPrevious();
    const float alpha = a.alphaDev ? *a.alphaDev : a.alpha;
    const float beta = a.betaDev ? *a.betaDev : a.beta;
    const int lane = threadIdx.x & 31, li = lane & (G - 1);
    const long long row = ((long long)blockIdx.x * kThreads + threadIdx.x) / G;
    bool mine = row < a.rows;
    long long s = 0, e = 0;
    if (mine) {
        s = LoadOffset(a.rowOffsets, kIs64, row) - a.indexBase;
        e = LoadOffset(a.rowOffsets, kIs64, row + 1) - a.indexBase;
        if (e - s >= outlier) {
            mine = false;
            e = s;
        }
    }
    const bool wide = e - s > 16 * G;
    float yOld = 0.0f;
    if (mine && li == 0 && beta != 0.0f) yOld = a.y[row];  // requested now, used at the end
    Triple t{0.0f, 0.0f, 0.0f};
    if (!wide) t = SumEntries(a, s + li, e, G);
    JoinLanes<G>(t);
    unsigned todo = __ballot_sync(0xffffffffu, wide && li == 0);
    while (todo != 0) {
        const int owner = __ffs(todo) - 1;
        todo &= todo - 1;
        const long long ws = __shfl_sync(0xffffffffu, s, owner), we = __shfl_sync(0xffffffffu, e, owner);
        Triple w = SumEntries<true>(a, ws + lane, we, 32);
        JoinLanes<32>(w);
        w.hi = __shfl_sync(0xffffffffu, w.hi, 0);
        w.md = __shfl_sync(0xffffffffu, w.md, 0);
        w.lo = __shfl_sync(0xffffffffu, w.lo, 0);
        if (lane == owner) t = w;
    }
    if (mine && li == 0) a.z[row] = Combine(t, alpha, __fmul_rn(beta, yOld));
}

// Places first .. first + count of the row order, from block firstBlock on, with G lanes per row (0: a CTA).
struct Range {
    int firstBlock, first, count;
};
// long rows; 128 to 511 entries; 64 to 127; 32 to 63; 16 to 31; 4 to 15; up to 3
constexpr int kRanges = 7;
constexpr int kRangeLanes[kRanges] = {0, 32, 16, 8, 4, 2, 1};
constexpr int kRangeBits[kRanges] = {kLongBits, 8, 7, 6, 5, 3, 0};  // fewest bits of a length in the range
struct Ranges {
    Range r[kRanges];
};

template <int G, bool kIs64>
__device__ __forceinline__ void ClassRow(const OpArgs &a, const Range &range, float alpha, float beta)
{
    const int li = threadIdx.x & (G - 1);
    const int i = ((int)blockIdx.x - range.firstBlock) * (kThreads / G) + (int)threadIdx.x / G;
    const bool mine = i < range.count;
    long long row = 0, s = 0, e = 0;
    if (mine) {
        row = a.reorder[range.first + i];
        s = LoadOffset(a.rowOffsets, kIs64, row) - a.indexBase;
        e = LoadOffset(a.rowOffsets, kIs64, row + 1) - a.indexBase;
    }
    float yOld = 0.0f;
    if (mine && li == 0 && beta != 0.0f) yOld = a.y[row];
    Triple t = SumEntries(a, s + li, e, G);
    JoinLanes<G>(t);
    if (mine && li == 0) a.z[row] = Combine(t, alpha, __fmul_rn(beta, yOld));
}

// 31.2 M entries in 1 M power-law rows: a warp per row from 64 entries and four lanes below, long rows on a side stream:
// 165 us; 138 to 141 us so.  The long rows wait for their gathers (L2 delivers one sector per clock and SM), the others
// for issue slots: an entry is some twenty instructions and a join of two lanes' sums as many, so lanes must not idle.
template <bool kIs64>
__global__ void __launch_bounds__(kThreads, 12) SpmvOpClassesKernel(const OpArgs a, const Ranges ranges)
{
    b200sp::WaitForPrevious();
    const float alpha = a.alphaDev ? *a.alphaDev : a.alpha;
    const float beta = a.betaDev ? *a.betaDev : a.beta;
    const int b = blockIdx.x;
    if (b < ranges.r[1].firstBlock) LongRow<kIs64, kThreads>(a, a.reorder[ranges.r[0].first + b], alpha, beta);
    else if (b < ranges.r[2].firstBlock) ClassRow<32, kIs64>(a, ranges.r[1], alpha, beta);
    else if (b < ranges.r[3].firstBlock) ClassRow<16, kIs64>(a, ranges.r[2], alpha, beta);
    else if (b < ranges.r[4].firstBlock) ClassRow<8, kIs64>(a, ranges.r[3], alpha, beta);
    else if (b < ranges.r[5].firstBlock) ClassRow<4, kIs64>(a, ranges.r[4], alpha, beta);
    else if (b < ranges.r[6].firstBlock) ClassRow<2, kIs64>(a, ranges.r[5], alpha, beta);
    else ClassRow<1, kIs64>(a, ranges.r[6], alpha, beta);
}

__global__ void SpmvOpScaleKernel(const float *__restrict__ y, float *__restrict__ z, long long rows, float beta,
                                  const float *betaDev)
{
    const float b = betaDev ? *betaDev : beta;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < rows;
         i += (long long)gridDim.x * blockDim.x)
        z[i] = b != 0.0f ? __fmul_rn(b, y[i]) : 0.0f;
}

__device__ __forceinline__ int LengthClass(long long len)
{
    return len <= 0 ? 0 : 64 - __clzll((unsigned long long)len);  // bits needed: 1 -> 1, 2..3 -> 2, 4..7 -> 3, ...
}

// cursors[c] += rows of class c
template <bool kIs64>
__global__ void SpmvOpHistogramKernel(const void *rowOffsets, long long rows, int32_t *cursors)
{
    __shared__ int sHist[kClasses];
    if (threadIdx.x < kClasses) sHist[threadIdx.x] = 0;
    __syncthreads();
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < rows;
         r += (long long)gridDim.x * blockDim.x) {
        const long long len = LoadOffset(rowOffsets, kIs64, r + 1) - LoadOffset(rowOffsets, kIs64, r);
        int c = LengthClass(len);
        if (c >= kClasses) c = kClasses - 1;
        atomicAdd(&sHist[c], 1);
    }
    __syncthreads();
    if (threadIdx.x < kClasses && sHist[threadIdx.x] != 0) atomicAdd(&cursors[threadIdx.x], sHist[threadIdx.x]);
}

template <bool kIs64>
__global__ void SpmvOpScatterKernel(const void *rowOffsets, long long rows, int32_t *cursors, int32_t *reorder)
{
    // A CTA first counts its rows per class, reserves that many slots of each class with one atomic,
    // then places its rows; the order inside a class is arbitrary and no result depends on it.
    __shared__ int sCount[kClasses];
    __shared__ int sBase[kClasses];
    const long long chunk = (rows + gridDim.x - 1) / gridDim.x;
    const long long r0 = (long long)blockIdx.x * chunk;
    const long long r1 = r0 + chunk < rows ? r0 + chunk : rows;
    if (threadIdx.x < kClasses) sCount[threadIdx.x] = 0;
    __syncthreads();
    for (long long r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
        const long long len = LoadOffset(rowOffsets, kIs64, r + 1) - LoadOffset(rowOffsets, kIs64, r);
        int c = LengthClass(len);
        if (c >= kClasses) c = kClasses - 1;
        atomicAdd(&sCount[c], 1);
    }
    __syncthreads();
    if (threadIdx.x < kClasses) {
        sBase[threadIdx.x] = sCount[threadIdx.x] != 0 ? atomicAdd(&cursors[threadIdx.x], sCount[threadIdx.x]) : 0;
        sCount[threadIdx.x] = 0;
    }
    __syncthreads();
    for (long long r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
        const long long len = LoadOffset(rowOffsets, kIs64, r + 1) - LoadOffset(rowOffsets, kIs64, r);
        int c = LengthClass(len);
        if (c >= kClasses) c = kClasses - 1;
        reorder[sBase[c] + atomicAdd(&sCount[c], 1)] = (int32_t)r;
    }
}

template <bool kIs64>
cudaError_t LaunchRows(const OpArgs &a, double mean, long long outlier, cudaStream_t st)
{
    auto launch = [&]<int G>() {
        b200sp_note_launches(1);
        return b200sp::LaunchChained(SpmvOpRowsKernel<G, kIs64>, (unsigned)((a.rows * G + kThreads - 1) / kThreads), kThreads, 0, st, a,
                                     outlier);
    };
    // lanes for which rows of the mean length give each of them four to eight entries: fewer idle the memory, more the lanes
    if (mean <= 1) return launch.template operator()<1>();  // mostly empty rows: 2 M of them, 20,000 entries: 18.9 us with two lanes
    if (mean <= 6) return launch.template operator()<2>();
    if (mean <= 28) return launch.template operator()<4>();
    if (mean <= 64) return launch.template operator()<8>();
    if (mean <= 128) return launch.template operator()<16>();
    return launch.template operator()<32>();
}

// Entries in rows four times as long as the mean and longer, as a share: from the classes, whose lengths lie between
// 2^(c-1) and 2^c - 1.  Ragged rows (up to twice the mean) have none, power-law rows more than half.  Below 15 % the rows
// in their own order win: their offsets and results coalesce, and the few long ones cost less than the indirection.
bool Skewed(const int32_t *class_start, double mean)
{
    double all = 0.0, heavy = 0.0;
    for (int i = 0; i < kClasses; ++i) {
        const int c = kClasses - 1 - i;
        if (c == 0) continue;
        const double entries = (class_start[i + 1] - class_start[i]) * 0.75 * (double)(1ll << c);
        all += entries;
        if ((double)(1ll << (c - 1)) >= 4 * mean) heavy += entries;
    }
    return heavy > 0.15 * all;
}

// Bits of a length from which a row gets a CTA of SpmvOpLongRowsKernel.  A warp takes 128 entries of a row per round trip to
// memory (0.9 us), a CTA of kThreads 512, while a grid that is full takes some 220 entries per ns.  So a row of nnz / 8192
// entries costs a warp, which may come to it late, a quarter of what the whole grid takes (half is fair for rows below twice
// the mean), and one of nnz / 512 entries a CTA, which comes to it first, as long as the grid takes; the rows beyond are
// few, by their number.  With a warp each, and so: 300,000 rows of 20 and 40 of 16,000: 136 and 31 us; 1 M rows of 30 and
// one of a million: 10.5 and 0.35 ms; 2000 rows of up to 8000: 71 and 37 us; 5000 rows of 1100: 23 and 27, left to warps.
int OutlierBits(int64_t nnz, double mean, bool skewed)
{
    double least = skewed ? 4096 : 1024, share = (double)nnz / (skewed ? 512 : 8192);
    if (!skewed && least < 2 * mean) least = 2 * mean < 2 * share ? 2 * mean : 2 * share > least ? 2 * share : least;
    int bits = 1;
    while (bits < 62 && (double)(1ll << (bits - 1)) < (share > least ? share : least)) ++bits;
    return bits;  // the shortest length of that many bits is 2^(bits - 1)
}
constexpr int kHugeBits = 15;  // rows of 16384 entries and more: CTAs of 1024 threads, the others of 256

// The rows of `bits` bits and more, count of them at the front of the row order; long ones first.
template <bool kIs64>
cudaError_t LaunchOutliers(const OpArgs &a, const int32_t *class_start, int count, cudaStream_t st)
{
    const int huge = class_start[kClasses - kHugeBits] < count ? class_start[kClasses - kHugeBits] : count;
    if (huge > 0) SpmvOpLongRowsKernel<kIs64, 1024><<<(unsigned)huge, 1024, 0, st>>>(a, 0);
    if (count > huge) SpmvOpLongRowsKernel<kIs64, 256><<<(unsigned)(count - huge), 256, 0, st>>>(a, huge);
    b200sp_note_launches((huge > 0) + (count > huge));
    return cudaGetLastError();
}

template <bool kIs64>
cudaError_t LaunchAll(const OpArgs &a, int64_t nnz, const int32_t *class_start, cudaStream_t st)
{
    const double mean = (double)nnz / (double)a.rows;
    if (class_start == nullptr) return LaunchRows<kIs64>(a, mean, INT64_MAX, st);
    const bool skewed = Skewed(class_start, mean);
    const int bits = OutlierBits(nnz, mean, skewed);
    const int outliers = bits < kClasses ? class_start[kClasses - bits] : 0;
    if (outliers == a.rows) return LaunchOutliers<kIs64>(a, class_start, outliers, st);
    // They write rows of z of their own: forked onto the side stream, ahead of the grid for the others.
    b200sp::SideLanes *lanes = outliers > 0 ? b200sp::GetSideLanes() : nullptr;
    cudaError_t e = cudaSuccess;
    if (outliers > 0) {
        if (lanes != nullptr) e = cudaEventRecord(lanes->fork, st);
        if (lanes != nullptr && e == cudaSuccess) e = cudaStreamWaitEvent(lanes->stream[0], lanes->fork, 0);
        if (e == cudaSuccess) e = LaunchOutliers<kIs64>(a, class_start, outliers, lanes != nullptr ? lanes->stream[0] : st);
        if (lanes != nullptr && e == cudaSuccess) e = cudaEventRecord(lanes->join[0], lanes->stream[0]);
        if (e != cudaSuccess) return e;
    }
    if (!skewed) {
        e = LaunchRows<kIs64>(a, mean, outliers > 0 ? 1ll << (bits - 1) : INT64_MAX, st);
    } else {
        Ranges ranges;
        long long blocks = 0;
        for (int i = 0; i < kRanges; ++i) {
            Range &r = ranges.r[i];
            r.firstBlock = (int)blocks;
            r.first = i == 0 ? outliers : ranges.r[i - 1].first + ranges.r[i - 1].count;
            const int end = class_start[kClasses - kRangeBits[i]];
            r.count = end > r.first ? end - r.first : 0;
            const int perBlock = kRangeLanes[i] == 0 ? 1 : kThreads / kRangeLanes[i];
            blocks += (r.count + perBlock - 1) / perBlock;
        }
        if (blocks > 0) {
            b200sp_note_launches(1);
            e = b200sp::LaunchChained(SpmvOpClassesKernel<kIs64>, (unsigned)blocks, kThreads, 0, st, a, ranges);
        }
    }
    if (lanes != nullptr) {
        const cudaError_t joined = cudaStreamWaitEvent(st, lanes->join[0], 0);
        if (e == cudaSuccess) e = joined;
    }
    return e;
}

}  // namespace

extern "C" {

size_t b200sp_spmvop_plan_bytes(int64_t rows) { return OpLayoutFor(rows).total; }

int b200sp_spmvop_analyze(const void *row_offsets, int offsets_are_64, int64_t rows, void *plan, size_t plan_bytes,
                          int32_t *class_start, void *stream)
{
    const OpPlanLayout L = OpLayoutFor(rows);
    if (plan == nullptr || class_start == nullptr || plan_bytes < L.total) return (int)cudaErrorInvalidValue;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    char *p = static_cast<char *>(plan);
    auto *reorder = reinterpret_cast<int32_t *>(p + L.offReorder);
    auto *cursors = reinterpret_cast<int32_t *>(p + L.offHist);
    cudaError_t e = cudaMemsetAsync(cursors, 0, 256, st);
    if (e != cudaSuccess) return (int)e;
    for (int c = 0; c <= kClasses; ++c) class_start[c] = 0;
    if (rows <= 0) return 0;
    const long long want = (rows + 255) / 256;
    const long long cap = (long long)b200sp_sm_count() * 8;
    const unsigned blocks = (unsigned)(want < cap ? want : cap);
    // Histogram on the device; the 33 counts come back once and the class starts are summed on the host.
    if (offsets_are_64) SpmvOpHistogramKernel<true><<<blocks, 256, 0, st>>>(row_offsets, rows, cursors);
    else SpmvOpHistogramKernel<false><<<blocks, 256, 0, st>>>(row_offsets, rows, cursors);
    b200sp_note_launches(1);
    int32_t hist[kClasses];
    e = cudaMemcpyAsync(hist, cursors, sizeof(hist), cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess) return (int)e;
    e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return (int)e;
    int32_t cursorInit[kClasses];
    int running = 0;
    for (int k = 0; k < kClasses; ++k) {
        const int c = kClasses - 1 - k;
        class_start[k] = running;
        cursorInit[c] = running;
        running += hist[c];
    }
    class_start[kClasses] = running;
    e = cudaMemcpyAsync(cursors, cursorInit, sizeof(cursorInit), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return (int)e;
    if (offsets_are_64) SpmvOpScatterKernel<true><<<blocks, 256, 0, st>>>(row_offsets, rows, cursors, reorder);
    else SpmvOpScatterKernel<false><<<blocks, 256, 0, st>>>(row_offsets, rows, cursors, reorder);
    b200sp_note_launches(1);
    e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    // cursorInit lives on this frame: the copy above must have read it before we return
    return (int)cudaStreamSynchronize(st);
}

int b200sp_spmvop_launch(const void *row_offsets, int offsets_are_64, const int32_t *col_ind, const float *val,
                         const float *x, const float *y, float *z, int64_t rows, int64_t nnz, int index_base,
                         float alpha, float beta, const float *alpha_dev, const float *beta_dev, const void *plan,
                         const int32_t *class_start, void *stream)
{
    if (rows <= 0) return 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    OpArgs a;
    a.rowOffsets = row_offsets;
    a.colInd = col_ind;
    a.val = val;
    a.x = x;
    a.y = y;
    a.z = z;
    a.indexBase = index_base;
    a.alpha = alpha;
    a.beta = beta;
    a.alphaDev = alpha_dev;
    a.betaDev = beta_dev;
    a.reorder = static_cast<const int32_t *>(plan);
    a.rows = rows;
    const int32_t *classes = plan != nullptr ? class_start : nullptr;
    return (int)(offsets_are_64 ? LaunchAll<true>(a, nnz, classes, st) : LaunchAll<false>(a, nnz, classes, st));
}

int b200sp_spmvop_scale(const float *y, float *z, int64_t rows, float beta, const float *beta_dev, void *stream)
{
    if (rows <= 0) return 0;
    const long long want = (rows + 255) / 256;
    const long long cap = (long long)b200sp_sm_count() * 16;
    SpmvOpScaleKernel<<<(unsigned)(want < cap ? want : cap), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        y, z, rows, beta, beta_dev);
    b200sp_note_launches(1);
    return (int)cudaGetLastError();
}

}  // extern "C"
