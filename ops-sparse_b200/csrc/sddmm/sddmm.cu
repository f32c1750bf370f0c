// aclsparseSDDMM*: C = (alpha * op(X) * op(Y) + beta * C) sampled on the pattern of C (CSR, values in place).
// op(X) is m x k, op(Y) is k x n; fp32, or fp16 storage with fp32 accumulation and a saturating cast back
// (the reference's device arithmetic, sparse/sddmm/arch35/sddmm_kernel.cpp:26-27, 424-437).  Checks, their
// order and status codes follow the reference host layer (sparse/sddmm/arch35/sddmm_host.cpp:145-320, 478-510,
// 660-764).  The reference reorders rows greedily over its cores in Preprocess; here the work is cut by
// non-zeros (a warp per 32 or 64 consecutive entries of C), which needs no analysis.  Preprocess notes the rows of these tiles and, for a Y that L2
// does not hold, an order that finds more of it there; for small products BufferSize reports a token 256 bytes (the
// API wants a buffer) and Preprocess only checks its arguments.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cstdint>
#include <type_traits>

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "b200sp_kernels.h"
#include "common/chained.cuh"
#include "common/internal.h"
#include "common/rows.cuh"

namespace {

struct Strides {  // op(X)(i, kk) = X[i * xi + kk * xk];  op(Y)(kk, j) = Y[kk * yk + j * yj]
    long long xi, xk, yk, yj;
};

template <typename T> __device__ __forceinline__ float Load(const T *p);
template <> __device__ __forceinline__ float Load<float>(const float *p) { return __ldg(p); }
template <> __device__ __forceinline__ float Load<__half>(const __half *p) { return __half2float(__ldg(p)); }
template <typename T> __device__ __forceinline__ T Store(float v);
template <> __device__ __forceinline__ float Store<float>(float v) { return v; }
template <> __device__ __forceinline__ __half Store<__half>(float v)
{
    return __float2half_rn(fminf(fmaxf(v, -65504.0f), 65504.0f));  // saturate, then round
}

template <typename T>
__global__ void __launch_bounds__(256) SddmmKernel(const int32_t *__restrict__ rowPtr, const int32_t *__restrict__ colInd,
                                                   T *__restrict__ cVal, const T *__restrict__ X,
                                                   const T *__restrict__ Y, int m, int k, long long nnz, Strides st,
                                                   float alpha, float beta, const T *alphaDev, const T *betaDev)
{
    const float a = alphaDev ? Load<T>(alphaDev) : alpha;
    const float b = betaDev ? Load<T>(betaDev) : beta;
    const int lane = threadIdx.x & 31;
    const long long warpsTotal = (long long)gridDim.x * (blockDim.x >> 5);
    const long long chunks = (nnz + 31) / 32;
    for (long long c = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < chunks; c += warpsTotal) {
        const long long p0 = c * 32;
        const long long p1 = p0 + 32 < nnz ? p0 + 32 : nnz;
        int lo = 0, hi = m - 1;  // row of entry p0: largest r with rowPtr[r] <= p0 (the same search in every lane)
        while (lo < hi) {
            const int mid = lo + ((hi - lo + 1) >> 1);
            if ((long long)__ldg(rowPtr + mid) <= p0) lo = mid;
            else hi = mid - 1;
        }
        int r = lo;
        for (long long p = p0; p < p1; ++p) {
            while ((long long)__ldg(rowPtr + r + 1) <= p) ++r;
            const int j = __ldg(colInd + p);
            const T *xr = X + (long long)r * st.xi;
            const T *yc = Y + (long long)j * st.yj;
            float acc = 0.0f;
            for (int kk = lane; kk < k; kk += 32) acc = fmaf(Load<T>(xr + kk * st.xk), Load<T>(yc + kk * st.yk), acc);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
            if (lane == 0) {
                float z = a * acc;
                if (b != 0.0f) z += b * Load<T>(cVal + p);
                cVal[p] = Store<T>(z);
            }
        }
    }
}

// The same product when k runs along the contiguous direction of both operands.  An entry of C is the dot product of
// two short rows, so the work is fetching a row of Y per entry; what counts is how many of them an SM has in flight
// and how few instructions go into each.
//   - kLanes lanes lie side by side on a row, kBytes bytes each (the widest the rows' alignment allows) and kSlabs pieces
//     apart; a warp therefore works on 32 / kLanes entries at a time, and rows wider than kLanes * kSlabs pieces take
//     several turns.
//   - Rows come through shared memory by cp.async, two batches of kBatch entries deep per lane group: no registers
//     hold data in flight.  With warps enough the batches are short (kShortBatch), for what a warp's ring leaves free are more warps, and
//     those keep more copies in flight than longer rings do: 2.4 M entries, fp16, k = 400, 248 us with one entry a batch, k = 512, 258, 310 and
//     404 with one, two and four; but pieces of 4 bytes, fp32, k = 211, 593, 499 and 477.  Three or four batches deep, with as many copies
//     in flight per warp, take 1.1 to 1.6 times as long.  Where all warps find room on the SMs with a longer batch, it is as long as that: a small
//     product waits for one copy after the other.  2000 entries, fp16, k = 64, 4.2 us with two entries a batch, 3.5 with four; fp32, k = 512, 13.1
//     with one, 8.3 with four; 38,400 entries, 14.9 and, with two, 11.9.
//   - A row of X is copied only when it differs from the entry before, and stays in registers, converted, until then.  Two products
//     share an instruction (packed fp32): a row of 512 bytes in fp16 takes some 30 instead of 47 instructions.
//   - A warp owns a tile of consecutive entries.  What is done once per entry (row, column, old value, store) is done
//     for the whole tile with coalesced accesses; lane group g works on the tile's g-th part.
//   - The kBatch sums of a batch are reduced together: a butterfly step that halves the number of values a lane
//     carries costs as many shuffles as values are left.
// fp16 rows that start on odd 2-byte addresses (kBytes = 2) are copied as the 4-byte words that cover them and
// realigned when they are read from shared memory.
// Measured (1 M nodes, 16.0 M entries, fp16, k = 256): 1256 us with 32 lanes a row and scalar products, 1157 us as it is here, which is the 7.6 GB
// of Y rows that come from DRAM at 6.6 TB/s, 890 us with the tiles in an order (see TileOrder): 5.0 GB.  Cutting rows of 64 entries and more into
// the pieces that lie in a block of columns cost 1930 us and more: short pieces, and X rows fetched anew for each.
template <int kBytes> struct Words { using Type = uint32_t; };  // 4, and the words of kBytes = 2
template <> struct Words<16> { using Type = uint4; };
template <> struct Words<8> { using Type = uint2; };

// The fp32 values of a piece, in pairs: packed arithmetic takes two of them per instruction.
template <typename T, typename Piece> struct Pairs {
    static constexpr int kCount = sizeof(Piece) / (2 * sizeof(T)) > 0 ? sizeof(Piece) / (2 * sizeof(T)) : 1;
    float2 v[kCount];
    __device__ __forceinline__ void Set(const Piece &p)
    {
        const uint32_t *w = reinterpret_cast<const uint32_t *>(&p);
        if constexpr (sizeof(T) == 2) {
#pragma unroll
            for (int i = 0; i < kCount; ++i) v[i] = __half22float2(reinterpret_cast<const __half2 *>(w)[i]);
        } else {
#pragma unroll
            for (int i = 0; i < kCount; ++i)
                v[i] = make_float2(__uint_as_float(w[2 * i]), sizeof(Piece) > 4 ? __uint_as_float(w[2 * i + 1]) : 0.0f);
        }
    }
};
__device__ __forceinline__ void FmaPair(float2 &acc, const float2 &x, const float2 &y)
{
    asm("{\n\t.reg .b64 a, b, c;\n\t"
        "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%0, %1};\n\t"
        "fma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
        : "+f"(acc.x), "+f"(acc.y)
        : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y));
}

// kSize bytes from global to shared memory; `bytes` of them are read, the rest is zero.  Copies of 16 bytes go past L1
// (.cg) or, kNear, through it.
template <int kSize, bool kNear = true> __device__ __forceinline__ void CopyAsync(void *dst, const void *src, int bytes)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (!kNear)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(kSize), "r"(bytes) : "memory");
}
__device__ __forceinline__ void CopyCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending> __device__ __forceinline__ void CopyWait() { asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory"); }

constexpr int kSddmmTile = 64;  // entries a warp works on at a time, at most
// Entries of a batch where there are warps enough: about 2 KB of copies a batch, half as much of the widest pieces.  Four lanes of three
// pieces have few entries a group, and warps enough from the start (fp16, k = 36, 320,000 entries: 11.5 us with one, 13.9 with two).
template <int kBytes, int kLanes, int kSlabs>
constexpr int kShortBatch = kLanes == 4 && kSlabs == 3 ? 1
                            : kBytes < 8  ? 4
                            : kBytes == 8 ? (kSlabs <= 2 ? 4 : kSlabs == 3 || kLanes == 16 ? 2 : 1)
                                          : (kSlabs <= 2 ? 2 : 1);

template <int kBytes, int kSlabs, int kBatch, bool kOrdered = false> struct SddmmShape {
    static constexpr int kStages = 2;
    static constexpr int kCopy = kBytes == 2 ? 4 : kBytes;
    static constexpr int kSlotBytes = 32 * kSlabs * kCopy;                       // one entry of every lane group
    static constexpr int kRing = 2 * kStages * kBatch * kSlotBytes;              // rows of Y, rows of X
    static constexpr int kTileBytes = kSddmmTile * 12;                           // row, column, sum per entry
    // Warps of a CTA.  Ordered tiles of wide rows: one, whose memory is free again as soon as it is done (1 M nodes, k = 256: 966 us with two,
    // 934 with one; k = 128 602 and 578).  Otherwise two (150,000 nodes, k = 256, no order: 91 and 93; k = 64 56 and 60, where the 32 CTAs of
    // an SM would not fill it).
    static constexpr int kWarps = kOrdered && kRing + kTileBytes > 7000 ? 1 : 2;
    static constexpr int kShared = kWarps * (kRing + kTileBytes);
    static constexpr int kWarpsPerSm = kWarps * ((228 << 10) / (kShared + 1024));  // that find room at once
};

struct RowsOf {  // the operands' rows and how far apart they are
    const char *X, *Y;
    long long xRowBytes, yRowBytes;
    int k;
};

// ---------------------------------------------------------------- the order of the tiles

// In a row of many entries a tile of consecutive ones lies on few rows of Y: with ascending columns, 64 of 4096 entries span a
// sixty-fourth of it.  Worked on in the order of their columns, such tiles of all rows ask for the same few megabytes of Y at any
// time, and those stay in L2, where the tiles of short rows, in between, fetch every row of Y from DRAM.  The order is found by Preprocess (the
// values and rows may change afterwards, the product is the same in any order) and kept in the caller's buffer: the near tiles by
// column, then the others.  Tiles of both kinds take turns in the grid, so that neither L2 nor DRAM waits for the other.  With a smaller Y, or few such
// tiles, what remains of this are the rows of the tiles.
//
// What the buffer holds when a product runs is not known: it may have been written by code that this library does not see, or be other memory at the
// same address, and a product in a graph may run after any call.  So nothing is taken from it on trust: rows are compared with the row
// offsets, and before an order is followed a kernel looks whether it names every tile once; if not, the tiles are taken as they lie.  (That kernel takes
// 4 us of 1000.  A kernel whose warps see for themselves whose tile is whose takes 31 us longer.)
struct TileOrder {
    const int2 *tiles = nullptr;       // {tile, row of its first entry}; near tiles by column, then the others; nullptr: no order and no rows
    const int *place = nullptr;        // [tile] where it stands in `tiles`
    unsigned ticket = 0;               // of the product that looks it over
    long long near = 0;                // 0: all tiles stand where they lie, and there is nothing to look at but rows
    unsigned long long share = 0;      // of the near tiles among all, times 2^32, rounded up
};
// Products do not write the caller's buffer.  Where the check finds that there is no order, it leaves the product's ticket here, which the product compares; a ticket's
// place serves another product 65,536 tickets later.  One that a graph repeats has the same ticket each time: once it was left here
// it may take the tiles as they lie from then on.
constexpr unsigned kTickets = 1 << 16;
__device__ unsigned gNoOrder[kTickets];
constexpr int kOrderBuckets = 1024;
// A smaller Y stays in L2 as a whole.
constexpr long long kOrderMinY = 96ll << 20;
// Bytes of Y that a near tile may lie on, a third of Y at most.  1 M nodes, fp16, k = 256 (Y of 537 MB), DRAM traffic 7.6 GB without an order: 32 MB
// 1046 us and 5.5 GB, 64 MB 1034, 96 MB 1029; with the rows of the tiles found by Preprocess, too, 976, 970 and (160 MB) 966.  (Copies with L2 policies, near tiles
// evict-last and the others evict-first, picked at run time and handed to every copy, ended in an illegal instruction when the code around
// them changed: no policy here.)
constexpr long long kNearSpan = 160ll << 20;
// Entries from which Preprocess notes the rows of the tiles (of 64 entries; fewer entries have shorter ones), in the order they lie in if none is
// near: a warp's search in the row offsets are four loads one after the other.  320,000 to 1.6 M entries of even and power-law rows, without and with
// them, us: fp16, k = 16 7.8 and 7.2, 26.0 and 24.1, k = 64 17.0 and 16.2, k = 128 55.3 and 51.1, k = 256 22.4 and 21.0, 91 and 86, fp32, k = 64 15.2 and
// 12.9, k = 128 83 and 76.
constexpr long long kOrderLeast = 1 << 18;
// Wider rows are as they were: their tiles are long, one warp a CTA and no tiles of 32 cost more than the search (fp16, k = 512 34.1 and 34.3, k =
// 640 56.0 and 60.4, 248 and 258; fp32, k = 256 29.7 and 31.8, k = 1024 104 and 113, at best 122 and 114).
constexpr int kRowsPieces = 32;
// Entries from which tiles may be near, for rows of up to eight pieces and wider ones: the check costs 2 us or more.  Y of 100 MB, a tenth / 60 % of the entries in rows of
// thousands, us without an order and with one: fp16, k = 16, 280,000 entries 7.3 / 7.0 and 8.7 / 8.8, 600,000 12.7 / 12.1 and 12.9 / 12.1, 1.5 M 30.0 / 28.4 and
// 28.3 / 26.3; k = 64 10.1 / 9.7 and 10.6 / 10.3, 17.8 / 16.8 and 17.8 / 17.4, 41 / 40 and 40 / 37; k = 512 39.6 / 37.6 and 43.3 / 39.8,
// 76 / 73 and 74 / 68, 185 / 165 and 174 / 160; fp32, k = 256 37.6 / 35.4 and 40.9 / 37.5, 75 / 69 and 70 / 62, 175 / 167 and 167 / 154.
constexpr long long kNearLeast = 1 << 20, kNearLeastWide = 1 << 19;
constexpr int kNearNarrow = 8;
// Fewer near tiles than one in so many are not worth the turns.
constexpr long long kNearShare = 16;
struct OrderLayout {
    long long tiles;
    size_t offCounts, offBucket, offTiles, offPlace, total;
};
inline OrderLayout OrderLayoutFor(long long nnz)
{
    OrderLayout L;
    L.tiles = (nnz + kSddmmTile - 1) / kSddmmTile;
    L.offCounts = 256;
    L.offBucket = L.offCounts + sizeof(int32_t) * 2 * (kOrderBuckets + 1);
    L.offBucket = (L.offBucket + 255) / 256 * 256;
    L.offTiles = (L.offBucket + sizeof(int16_t) * (size_t)L.tiles + 255) / 256 * 256;
    L.offPlace = L.offTiles + sizeof(int2) * (size_t)L.tiles;
    L.total = L.offPlace + sizeof(int32_t) * (size_t)L.tiles;
    return L;
}

// A warp per tile: its bucket of columns, kOrderBuckets if it is not near; how many tiles every bucket has.
__global__ void __launch_bounds__(256) SddmmTileBucketsKernel(const int32_t *__restrict__ colInd, int nnz, int cols, int span,
                                                              long long tiles, int16_t *__restrict__ bucket, int *__restrict__ counts)
{
    __shared__ int sCount[kOrderBuckets + 1];
    for (int i = threadIdx.x; i <= kOrderBuckets; i += blockDim.x) sCount[i] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long t = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < tiles; t += warps) {
        int low = INT_MAX, high = INT_MIN;
        for (int i = lane; i < kSddmmTile; i += 32) {
            const long long p = t * kSddmmTile + i;
            if (p >= nnz) continue;
            const int c = __ldg(colInd + p);
            low = min(low, c);
            high = max(high, c);
        }
        low = __reduce_min_sync(0xffffffffu, low);
        high = __reduce_max_sync(0xffffffffu, high);
        if (lane == 0) {
            const bool near = low >= 0 && high < cols && high - low <= span;
            const int b = near ? (int)(((long long)low + (high - low) / 2) * kOrderBuckets / cols) : kOrderBuckets;
            bucket[t] = (int16_t)b;
            atomicAdd(sCount + b, 1);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i <= kOrderBuckets; i += blockDim.x)
        if (sCount[i] != 0) atomicAdd(counts + i, sCount[i]);
}

// One CTA: where every bucket starts; what is in the last but one place after it is the number of near tiles.
__global__ void __launch_bounds__(kOrderBuckets) SddmmBucketStartsKernel(const int *__restrict__ counts, int *__restrict__ starts)
{
    __shared__ int sWarp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = counts[threadIdx.x];
    int upTo = n;
    for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upTo, off);
        if (lane >= off) upTo += v;
    }
    if (lane == 31) sWarp[warp] = upTo;
    __syncthreads();
    if (warp == 0) {
        int v = sWarp[lane];
        for (int off = 1; off < 32; off <<= 1) {
            const int w = __shfl_up_sync(0xffffffffu, v, off);
            if (lane >= off) v += w;
        }
        sWarp[lane] = v;
    }
    __syncthreads();
    upTo += warp > 0 ? sWarp[warp - 1] : 0;
    starts[threadIdx.x] = upTo - n;
    if (threadIdx.x == kOrderBuckets - 1) starts[kOrderBuckets] = upTo;
}

// Row of entry p: the last one that starts at or before it.
__device__ __forceinline__ int RowOfEntry(const int32_t *rowPtr, int m, long long p)
{
    int lo = 0, hi = m - 1;
    while (lo < hi) {
        const int mid = lo + ((hi - lo + 1) >> 1);
        if (__ldg(rowPtr + mid) <= p) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// A thread per tile: where it lies, and its row.
__global__ void __launch_bounds__(256) SddmmTileRowsKernel(const int32_t *__restrict__ rowPtr, int m, long long tiles, int2 *__restrict__ order)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < tiles) order[t] = make_int2((int)t, RowOfEntry(rowPtr, m, t * kSddmmTile));
}

// A CTA per 1024 tiles: their places.  Inside a bucket as the CTAs come, the others nearly as they lie.
__global__ void __launch_bounds__(256) SddmmOrderTilesKernel(const int32_t *__restrict__ rowPtr, int m, const int16_t *__restrict__ bucket,
                                                             long long tiles, int *__restrict__ starts, int2 *__restrict__ order,
                                                             int *__restrict__ place)
{
    __shared__ int sCount[kOrderBuckets + 1], sStart[kOrderBuckets + 1];
    for (int i = threadIdx.x; i <= kOrderBuckets; i += blockDim.x) sCount[i] = 0;
    __syncthreads();
    const long long t0 = (long long)blockIdx.x * 1024 + threadIdx.x;
    int mine[4], at[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const long long t = t0 + i * 256;
        mine[i] = t < tiles ? bucket[t] : -1;
        at[i] = mine[i] >= 0 ? atomicAdd(sCount + mine[i], 1) : 0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i <= kOrderBuckets; i += blockDim.x) sStart[i] = sCount[i] != 0 ? atomicAdd(starts + i, sCount[i]) : 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (mine[i] >= 0) {
            const int t = (int)(t0 + i * 256);
            const int to = sStart[mine[i]] + at[i];
            order[to] = make_int2(t, RowOfEntry(rowPtr, m, (long long)t * kSddmmTile));
            place[t] = to;
        }
}

// A thread per tile: whether it stands somewhere, and there alone.
__global__ void __launch_bounds__(256) SddmmOrderCheckKernel(const int2 *__restrict__ order, const int *__restrict__ place, int tiles, unsigned ticket)
{
    b200sp::WaitForPrevious();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= tiles) return;
    const int at = __ldg(place + t);
    if ((unsigned)at >= (unsigned)tiles || __ldg(&order[at].x) != t) gNoOrder[ticket % kTickets] = ticket;
}

// The dot products of a tile of entries: sDot[t] = X row sRow[t] . Y row sCol[t].  tile: a multiple of 32.
template <typename T, int kBytes, int kLanes, int kSlabs, bool kNear, int kBatch>
__device__ __forceinline__ void TileDots(const RowsOf &rows, unsigned char *ring, const int *sRow, const int *sCol, float *sDot,
                                         int tile, int lane)
{
    using Shape = SddmmShape<kBytes, kSlabs, kBatch>;
    using Piece = typename Words<kBytes>::Type;
    constexpr int kStages = Shape::kStages;
    constexpr int kCopy = Shape::kCopy;
    constexpr bool kOdd = kBytes == 2;
    static_assert(kLanes >= 4, "the sums of a batch are spread over four lanes");
    using Ints = std::conditional_t<kBatch == 4, int4, std::conditional_t<kBatch == 2, int2, int>>;
    const int li = lane & (kLanes - 1);
    const int group = lane / kLanes;
    Piece *const sY = reinterpret_cast<Piece *>(ring) + lane, *const sX = sY + kStages * kBatch * kSlabs * 32;
    const int k = rows.k;
    // unsigned: a row may hold 2^31 - 1 elements, and the last turn ends beyond its last piece
    const unsigned pieces = kOdd ? ((unsigned)k + 1) / 2 : (unsigned)((long long)k * (int)sizeof(T) / kBytes);
    const int perGroup = tile / (32 / kLanes);
    const int t0 = group * perGroup;
    const int batches = perGroup / kBatch;
    for (unsigned piece0 = 0; piece0 < pieces; piece0 += kLanes * kSlabs - (kOdd ? 1 : 0)) {
        const int width = kLanes * kSlabs - (kOdd ? 1 : 0);
        [[maybe_unused]] int inside[kSlabs];  // bytes of the lane's pieces that lie in the row, ...
        [[maybe_unused]] long long offset[kSlabs];  // ... and where they start
#pragma unroll
        for (int s = 0; s < kSlabs; ++s) {
            const unsigned q = piece0 + s * kLanes + li;
            inside[s] = q < pieces ? kCopy : 0;
            offset[s] = q < pieces ? (long long)q * kBytes : 0;
        }
        auto copyRow = [&](Piece *slot, const char *row) {
#pragma unroll
            for (int s = 0; s < kSlabs; ++s) {
                if constexpr (kOdd) {  // words from the one that holds the first element on, zeros after the row's last
                    const unsigned q = piece0 + s * kLanes + li;
                    const int off = (int)(reinterpret_cast<uintptr_t>(row) & 2);
                    const unsigned end = (unsigned)k + (unsigned)off / 2;  // of the row, in elements from the first word on
                    const int bytes = end >= 2 * q + 2 ? 4 : end > 2 * q ? 2 : 0;
                    CopyAsync<4>(slot + s * 32, row - off + (bytes > 0 ? 4ll * q : 0), bytes);
                } else {
                    CopyAsync<kCopy, kNear || kCopy != 16>(slot + s * 32, row + offset[s], inside[s]);
                }
            }
        };
        int asked = -1;  // the row of X copied last
        auto request = [&](int batch) {
            if (batch < batches) {
                const int slot0 = (batch % kStages) * kBatch * kSlabs * 32;
                const Ints rowOf = *reinterpret_cast<const Ints *>(sRow + t0 + batch * kBatch);
                const Ints colOf = *reinterpret_cast<const Ints *>(sCol + t0 + batch * kBatch);
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const int row = reinterpret_cast<const int *>(&rowOf)[u];
                    copyRow(sY + slot0 + u * kSlabs * 32, rows.Y + reinterpret_cast<const int *>(&colOf)[u] * rows.yRowBytes);
                    if (row != asked) copyRow(sX + slot0 + u * kSlabs * 32, rows.X + row * rows.xRowBytes);
                    asked = row;
                }
            }
            CopyCommit();
        };
        // A lane's pieces of a row: its own words, or (kOdd) the elements 2 q and 2 q + 1 wherever they lie.
        auto read = [&](const Piece *slot, const char *row, int s) -> Piece {
            if constexpr (kOdd) {
                const int i = s * kLanes + li;  // word of the turn; the last one only completes its neighbour
                const int next = i + 1 < kLanes * kSlabs ? i + 1 : i;
                const uint32_t w0 = slot[s * 32];
                const uint32_t w1 = slot[(next / kLanes) * 32 + group * kLanes + (next & (kLanes - 1)) - lane];
                const uint32_t v = __funnelshift_r(w0, w1, (uint32_t)(reinterpret_cast<uintptr_t>(row) & 2) * 8);
                return i < width ? v : 0u;
            } else {
                return slot[s * 32];
            }
        };
        Pairs<T, Piece> x[kSlabs];
#pragma unroll
        for (int s = 0; s < kSlabs; ++s) x[s].Set(Piece{});
        int held = -1;  // the row of X in x
#pragma unroll
        for (int i = 0; i < kStages - 1; ++i) request(i);
#pragma unroll 1
        for (int batch = 0; batch < batches; ++batch) {
            request(batch + kStages - 1);
            CopyWait<kStages - 1>();
            __syncwarp();
            const int slot0 = (batch % kStages) * kBatch * kSlabs * 32;
            const Ints rowOf = *reinterpret_cast<const Ints *>(sRow + t0 + batch * kBatch);
            Ints colOf{};
            if constexpr (kOdd) colOf = *reinterpret_cast<const Ints *>(sCol + t0 + batch * kBatch);
            float acc[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                const int row = reinterpret_cast<const int *>(&rowOf)[u];
                if (row != held) {
#pragma unroll
                    for (int s = 0; s < kSlabs; ++s) x[s].Set(read(sX + slot0 + u * kSlabs * 32, rows.X + row * rows.xRowBytes, s));
                    held = row;
                }
                float2 sum = make_float2(0.0f, 0.0f);
#pragma unroll
                for (int s = 0; s < kSlabs; ++s) {
                    Pairs<T, Piece> y;
                    y.Set(read(sY + slot0 + u * kSlabs * 32, rows.Y + reinterpret_cast<const int *>(&colOf)[u] * rows.yRowBytes, s));
#pragma unroll
                    for (int i = 0; i < Pairs<T, Piece>::kCount; ++i) FmaPair(sum, x[s].v[i], y.v[i]);
                }
                acc[u] = sum.x + sum.y;
            }
            // Lanes with bit kLanes/2 set keep the upper half of the values, then those with bit kLanes/4 the odd ones.
            [[maybe_unused]] const bool up = (li & (kLanes / 2)) != 0;
            float v;
            int u;  // the value this lane ends up with
            if constexpr (kBatch == 4) {
                const bool odd = (li & (kLanes / 4)) != 0;
                const float k0 = (up ? acc[2] : acc[0]) + __shfl_xor_sync(0xffffffffu, up ? acc[0] : acc[2], kLanes / 2);
                const float k1 = (up ? acc[3] : acc[1]) + __shfl_xor_sync(0xffffffffu, up ? acc[1] : acc[3], kLanes / 2);
                v = (odd ? k1 : k0) + __shfl_xor_sync(0xffffffffu, odd ? k0 : k1, kLanes / 4);
#pragma unroll
                for (int off = kLanes / 8; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                u = (up ? 2 : 0) + (odd ? 1 : 0);
            } else if constexpr (kBatch == 1) {
                v = acc[0];
#pragma unroll
                for (int off = kLanes / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                u = 0;
            } else {
                v = (up ? acc[1] : acc[0]) + __shfl_xor_sync(0xffffffffu, up ? acc[0] : acc[1], kLanes / 2);
#pragma unroll
                for (int off = kLanes / 4; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                u = up ? 1 : 0;
            }
            if ((li & (kLanes / kBatch - 1)) == 0) sDot[t0 + batch * kBatch + u] += v;
            __syncwarp();  // this stage's slots may be written again
        }
        CopyWait<0>();
        __syncwarp();
    }
}

template <typename T, int kBytes, int kLanes, int kSlabs, bool kNear, int kBatch, bool kOrdered>
__global__ void __launch_bounds__(32 * SddmmShape<kBytes, kSlabs, kBatch, kOrdered>::kWarps) SddmmRowsKernel(const int32_t *__restrict__ rowPtr,
                                                                    const int32_t *__restrict__ colInd, T *__restrict__ cVal,
                                                                    const RowsOf rows, int m, int nnz, int tile, float alpha,
                                                                    float beta, const T *alphaDev, const T *betaDev,
                                                                    [[maybe_unused]] const TileOrder order)
{
    using Shape = SddmmShape<kBytes, kSlabs, kBatch, kOrdered>;
    static_assert(!kOrdered || (kBytes == 16 && !kNear));
    extern __shared__ __align__(16) unsigned char sRaw[];
    b200sp::WaitForPrevious();
    const float a = alphaDev ? Load<T>(alphaDev) : alpha;
    const float b = betaDev ? Load<T>(betaDev) : beta;
    const int lane = threadIdx.x & 31;
    long long p0 = (long long)blockIdx.x * Shape::kWarps + (threadIdx.x >> 5);
    if (p0 * tile >= nnz) return;
    int r0 = -1;
    if constexpr (kOrdered) {
        const unsigned before = (unsigned)((p0 * order.share) >> 32);
        const bool near = (unsigned)(((p0 + 1) * order.share) >> 32) != before;
        const int2 at = __ldg(order.tiles + (near ? before : order.near + (p0 - before)));
        if (order.near != 0 && gNoOrder[order.ticket % kTickets] != order.ticket) p0 = at.x;
        r0 = at.y;
    }
    p0 *= tile;
    if (kOrdered && (p0 < 0 || p0 >= nnz)) return;
    unsigned char *ring = sRaw + (threadIdx.x >> 5) * (Shape::kRing + Shape::kTileBytes);
    int *sRow = reinterpret_cast<int *>(ring + Shape::kRing), *sCol = sRow + kSddmmTile;
    float *sDot = reinterpret_cast<float *>(sCol + kSddmmTile);
    // All columns, and the bounds of the row that Preprocess found, are asked for at once: one round trip instead of three (1 M nodes, k = 256, in
    // order 942 us and 881 so; 100,000 rows of 10, fp32, k = 60 47 and 42).
    int cols[kSddmmTile / 32];
#pragma unroll
    for (int i = 0; i < kSddmmTile / 32; ++i) {
        const int t = i * 32 + lane;
        cols[i] = t < tile ? __ldg(colInd + (p0 + t < nnz ? p0 + t : nnz - 1)) : 0;
    }
    long long end = -1;  // of that row, if the tile's first entry still lies in it
    if (kOrdered && (unsigned)r0 < (unsigned)m) {
        const int s = __ldg(rowPtr + r0), e = __ldg(rowPtr + r0 + 1);
        if (s <= p0 && p0 < e) end = e;
    }
    const bool single = end >= p0 + tile;  // one row: a near tile's usual case
    if (end < 0) r0 = b200sp::WarpRowOf(rowPtr, m, p0, lane);
#pragma unroll
    for (int i = 0; i < kSddmmTile / 32; ++i) {
        const int t = i * 32 + lane;
        if (i * 32 >= tile) break;
        const int p = p0 + t < nnz ? (int)p0 + t : nnz - 1;  // past the end: the last entry again, not stored
        const int r = single ? r0 : b200sp::RowOfLane(rowPtr, m, r0, p, lane);
        sRow[t] = r;
        sCol[t] = cols[i];
        sDot[t] = 0.0f;
        if (!single) r0 = __shfl_sync(0xffffffffu, r, 31);
    }
    __syncwarp();
    TileDots<T, kBytes, kLanes, kSlabs, kNear, kBatch>(rows, ring, sRow, sCol, sDot, tile, lane);
    for (int t = lane; t < tile && p0 + t < nnz; t += 32) {
        float z = a * sDot[t];
        if (b != 0.0f) z += b * Load<T>(cVal + p0 + t);
        cVal[p0 + t] = Store<T>(z);
    }
}

float HalfBitsToFloat(uint16_t h) { return __half2float(__ushort_as_half(h)); }

float ReadScalar(const void *p, aclDataType computeType)  // sddmm_host.cpp:128-139
{
    if (computeType == ACL_FLOAT16) {
        uint16_t bits;
        __builtin_memcpy(&bits, p, sizeof(bits));
        return HalfBitsToFloat(bits);
    }
    float v;
    __builtin_memcpy(&v, p, sizeof(v));
    return v;
}

aclsparseStatus_t ValidateInputs(const aclsparseDnMatDescr *X, const aclsparseDnMatDescr *Y, const aclsparseSpMatDescr *C,
                                 aclsparseOperation_t opX, aclsparseOperation_t opY, aclDataType computeType,
                                 aclsparseSDDMMAlg_t alg)
{
    // descriptors (sddmm_host.cpp:209-232)
    if (X == nullptr || Y == nullptr || C == nullptr) return ACL_SPARSE_STATUS_INVALID_VALUE;
    if (C->format != ACL_SPARSE_FORMAT_CSR) return ACL_SPARSE_STATUS_MATRIX_TYPE_NOT_SUPPORTED;
    if (C->offsetType != C->indexType || C->offsetType != ACL_SPARSE_INDEX_32I) return ACL_SPARSE_STATUS_NOT_SUPPORTED;
    if (C->base != ACL_SPARSE_INDEX_BASE_ZERO) return ACL_SPARSE_STATUS_NOT_SUPPORTED;
    // operations (:194-207)
    if (opX != ACL_SPARSE_OP_NON_TRANSPOSE && opX != ACL_SPARSE_OP_TRANSPOSE) return ACL_SPARSE_STATUS_NOT_SUPPORTED;
    if (opY != ACL_SPARSE_OP_NON_TRANSPOSE && opY != ACL_SPARSE_OP_TRANSPOSE) return ACL_SPARSE_STATUS_NOT_SUPPORTED;
    // types and dimensions (:234-269)
    const bool f32 = X->valueType == ACL_FLOAT && Y->valueType == ACL_FLOAT && C->valueType == ACL_FLOAT &&
                     computeType == ACL_FLOAT;
    const bool f16 = X->valueType == ACL_FLOAT16 && Y->valueType == ACL_FLOAT16 && C->valueType == ACL_FLOAT16 &&
                     computeType == ACL_FLOAT16;
    if (!f32 && !f16) return ACL_SPARSE_STATUS_NOT_SUPPORTED;
    const int64_t m = C->rows, n = C->cols;
    int64_t k;
    if (opX == ACL_SPARSE_OP_NON_TRANSPOSE) {
        if (X->rows != m) return ACL_SPARSE_STATUS_INVALID_VALUE;
        k = X->cols;
    } else {
        if (X->cols != m) return ACL_SPARSE_STATUS_INVALID_VALUE;
        k = X->rows;
    }
    const bool yOk = opY == ACL_SPARSE_OP_NON_TRANSPOSE ? (Y->rows == k && Y->cols == n) : (Y->rows == n && Y->cols == k);
    if (!yOk) return ACL_SPARSE_STATUS_INVALID_VALUE;
    if (alg != ACL_SPARSE_SDDMM_ALG_DEFAULT) return ACL_SPARSE_STATUS_NOT_SUPPORTED;
    if (C->rows > INT32_MAX || C->cols > INT32_MAX || X->rows > INT32_MAX || X->cols > INT32_MAX ||
        Y->rows > INT32_MAX || Y->cols > INT32_MAX)
        return ACL_SPARSE_STATUS_NOT_SUPPORTED;
    // CSR data (:271-294)
    if (C->nnz > INT32_MAX) return ACL_SPARSE_STATUS_INVALID_VALUE;
    if (C->offsets == nullptr) return ACL_SPARSE_STATUS_INVALID_VALUE;
    if (C->nnz > 0 && (C->indices == nullptr || C->values == nullptr)) return ACL_SPARSE_STATUS_INVALID_VALUE;
    return ACL_SPARSE_STATUS_SUCCESS;
}

// sddmm_host.cpp:660-692
aclsparseStatus_t ValidateCall(aclsparseHandle_t handle, const aclsparseDnMatDescr *X, const aclsparseDnMatDescr *Y,
                               const aclsparseSpMatDescr *C, const void *alpha, const void *beta, void *buffer,
                               bool isPreprocess, aclsparseOperation_t opX, aclsparseOperation_t opY,
                               aclDataType computeType, aclsparseSDDMMAlg_t alg)
{
    if (handle == nullptr) return ACL_SPARSE_STATUS_HANDLE_IS_NULLPTR;
    const aclsparseStatus_t st = ValidateInputs(X, Y, C, opX, opY, computeType, alg);
    if (st != ACL_SPARSE_STATUS_SUCCESS) return st;
    if (alpha == nullptr || beta == nullptr) return ACL_SPARSE_STATUS_INVALID_VALUE;
    if (buffer == nullptr) return isPreprocess ? ACL_SPARSE_STATUS_INSUFFICIENT_RESOURCES : ACL_SPARSE_STATUS_INVALID_VALUE;
    return ACL_SPARSE_STATUS_SUCCESS;
}

// Whether the kernel may use the shared memory it wants on the current device: the attribute is set once per device.
template <auto kKernel> cudaError_t AllowSharedMemory(int bytes, int *device)
{
    static std::atomic<bool> done[64] = {};
    const cudaError_t got = cudaGetDevice(device);
    if (got != cudaSuccess || *device < 0 || *device >= 64) return cudaErrorInvalidDevice;
    if (done[*device].load(std::memory_order_relaxed)) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done[*device].store(true, std::memory_order_relaxed);
    return e;
}

template <typename T, int kBytes, int kLanes, int kSlabs, bool kNear, int kBatch, bool kOrdered, typename... Args>
int LaunchRowsShape(int nnz, int tile, cudaStream_t stream, Args... args)
{
    using Shape = SddmmShape<kBytes, kSlabs, kBatch, kOrdered>;
    int dev = 0;
    const cudaError_t e = AllowSharedMemory<SddmmRowsKernel<T, kBytes, kLanes, kSlabs, kNear, kBatch, kOrdered>>(Shape::kShared, &dev);
    if (e != cudaSuccess) return (int)e;
    const long long warps = ((long long)nnz + tile - 1) / tile;
    b200sp_note_launches(1);
    return (int)b200sp::LaunchChained(SddmmRowsKernel<T, kBytes, kLanes, kSlabs, kNear, kBatch, kOrdered>,
                                      (unsigned)((warps + Shape::kWarps - 1) / Shape::kWarps), 32 * Shape::kWarps, Shape::kShared,
                                      stream, args...);
}

// 300,000 rows of four entries, 16-byte copies past L1 and through it, us, by the size of Y: 9 columns, fp16, k = 16 (0.3 KB) 292 and
// 24, k = 200 (3.5 KB) 542 and 89, fp32, k = 300 (10.5 KB) 823 and 245; 100 columns, fp16, k = 64 (12.5 KB) 34 and 37, fp32,
// k = 64 (25 KB) 63 and 69; 1 M columns, fp16, k = 256, 16 M entries: 1140 and 1737.
constexpr long long kNearBytes = 12 << 10;

template <typename T, int kBytes>
int LaunchRows(const aclsparseSpMatDescr *C, const aclsparseDnMatDescr *X, const aclsparseDnMatDescr *Y, int k, Strides st,
               float alpha, float beta, const void *alphaDev, const void *betaDev, const TileOrder &order, cudaStream_t stream)
{
    const int nnz = (int)C->nnz;
    // pieces of a row, one more where they start in the middle of a word
    const long long pieces = kBytes == 2 ? ((long long)k + 1) / 2 + 1 : (long long)k * (long long)sizeof(T) / kBytes;
    // The longer the tile the longer the runs of copies in flight, as long as every SM gets some 16 warps.
    int tile = 32;
    while (tile < kSddmmTile && nnz / (2 * tile) >= 16 * b200sp_sm_count()) tile *= 2;
    // A Y of a few lines that all entries want is asked of a few slices of L2 by every SM at once: it comes through L1.
    const bool near = kBytes == 16 && (long long)C->cols * st.yj * (long long)sizeof(T) <= kNearBytes;
    auto launchAs = [&]<int kLanes, int kSlabs, bool kNear, int kBatch, bool kOrdered>() {
        const RowsOf rows{static_cast<const char *>(X->values), static_cast<const char *>(Y->values),
                          st.xi * (long long)sizeof(T), st.yj * (long long)sizeof(T), k};
        // Rows of more than 32 pieces are long enough work for a last wave that is nearly empty to show.  320,000 entries, fp32, tiles of 64 and
        // 32: k = 400 80 and 66 us, k = 512 68 and 58, fp16, k = 640 66 and 56; narrower rows lose (fp16, k = 80: 17.2 and 19.0).
        const long long room = (long long)SddmmShape<kBytes, kSlabs, kBatch>::kWarpsPerSm * b200sp_sm_count(), warps = nnz / kSddmmTile;
        const int entries = !kOrdered && kLanes * kSlabs > 32 && warps > room && warps < 3 * room ? 32 : tile;
        return LaunchRowsShape<T, kBytes, kLanes, kSlabs, kNear, kBatch, kOrdered>(
            nnz, entries, stream, static_cast<const int32_t *>(C->offsets), static_cast<const int32_t *>(C->indices),
            static_cast<T *>(C->values), rows, (int)C->rows, nnz, entries, alpha, beta, static_cast<const T *>(alphaDev),
            static_cast<const T *>(betaDev), order);
    };
    auto launchDeep = [&]<int kLanes, int kSlabs, int kBatch>() {
        if constexpr (kBytes == 16)
            if (near) return launchAs.template operator()<kLanes, kSlabs, true, kBatch, false>();
        return launchAs.template operator()<kLanes, kSlabs, false, kBatch, false>();
    };
    auto launch = [&]<int kLanes, int kSlabs>() {
        constexpr int kShort = kShortBatch<kBytes, kLanes, kSlabs>;
        if constexpr (kBytes == 16)
            if (order.tiles != nullptr && tile == kSddmmTile && !near && (order.near > 0 || kLanes * kSlabs <= kRowsPieces)) {
                if (order.near > 0) {
                    const int tiles = (nnz - 1) / kSddmmTile + 1;
                    b200sp_note_launches(1);
                    const cudaError_t e = b200sp::LaunchChained(SddmmOrderCheckKernel, (unsigned)((tiles + 255) / 256), 256, 0, stream, order.tiles,
                                                                order.place, tiles, order.ticket);
                    if (e != cudaSuccess) return (int)e;
                }
                return launchAs.template operator()<kLanes, kSlabs, false, kShort, true>();
            }
        const long long warps = (nnz + 31ll) / 32 / b200sp_sm_count();  // for every SM, with the shortest tiles
        if constexpr (kShort < 4)
            if (warps < SddmmShape<kBytes, kSlabs, 4>::kWarpsPerSm) return launchDeep.template operator()<kLanes, kSlabs, 4>();
        if constexpr (kShort < 2)
            if (warps < SddmmShape<kBytes, kSlabs, 2>::kWarpsPerSm) return launchDeep.template operator()<kLanes, kSlabs, 2>();
        return launchDeep.template operator()<kLanes, kSlabs, kShort>();
    };
    // Few lanes and several pieces each: a warp then works on more entries per instruction.  2.4 M entries, 16-byte pieces, us with 16 or 32
    // lanes of one piece, or 32 of two and four, and as here: 10 pieces 113 and 71, 16 109 and 83, 20 185 and 110, 24 183 and 111, 32
    // 183 and 131, 50 352 and 248, 80 576 and 371, 128 (fp16) 631 and 584.  Up to 8 pieces fewer lanes gain nothing.  Rows of 14 and 16 pieces start on
    // 32-byte sectors, which four lanes side by side fill: 84 and 83 us, by eight lanes 90 and 89; of 13 and 15: 94 and 101, by eight 91 and 92.
    if (pieces <= 4) return launch.template operator()<4, 1>();
    if (pieces <= 8) return launch.template operator()<8, 1>();
    if (pieces <= 12) return launch.template operator()<4, 3>();
    if (pieces <= 16) return pieces % 2 != 0 ? launch.template operator()<8, 2>() : launch.template operator()<4, 4>();
    if (pieces <= 24) return launch.template operator()<8, 3>();
    if (pieces <= 32) return launch.template operator()<8, 4>();
    if (pieces <= 48) return launch.template operator()<16, 3>();
    if (pieces <= 64) return launch.template operator()<16, 4>();
    if (pieces <= 96) return launch.template operator()<32, 3>();
    return launch.template operator()<32, 4>();
}

template <typename T>
int Launch(const aclsparseSpMatDescr *C, const aclsparseDnMatDescr *X, const aclsparseDnMatDescr *Y, int k, Strides st,
           float alpha, float beta, const void *alphaDev, const void *betaDev, const TileOrder &order, cudaStream_t stream)
{
    if (st.xk == 1 && st.yk == 1) {
        // the widest piece that every row starts and ends on
        const unsigned long long all = (unsigned long long)k * sizeof(T) | (unsigned long long)st.xi * sizeof(T) |
                                       (unsigned long long)st.yj * sizeof(T) | reinterpret_cast<uintptr_t>(X->values) |
                                       reinterpret_cast<uintptr_t>(Y->values);
        if (all % 16 == 0) return LaunchRows<T, 16>(C, X, Y, k, st, alpha, beta, alphaDev, betaDev, order, stream);
        if (all % 8 == 0) return LaunchRows<T, 8>(C, X, Y, k, st, alpha, beta, alphaDev, betaDev, order, stream);
        if (all % 4 == 0) return LaunchRows<T, 4>(C, X, Y, k, st, alpha, beta, alphaDev, betaDev, order, stream);
        if constexpr (sizeof(T) == 2)  // the covering words of the first rows start at the arrays
            if (reinterpret_cast<uintptr_t>(X->values) % 4 == 0 && reinterpret_cast<uintptr_t>(Y->values) % 4 == 0)
                return LaunchRows<T, 2>(C, X, Y, k, st, alpha, beta, alphaDev, betaDev, order, stream);
    }
    const long long chunks = (C->nnz + 31) / 32;
    const long long want = (chunks + 7) / 8;
    const long long cap = (long long)b200sp_sm_count() * 32;
    const unsigned grid = (unsigned)(want < cap ? want : cap);
    SddmmKernel<T><<<grid, 256, 0, stream>>>(
        static_cast<const int32_t *>(C->offsets), static_cast<const int32_t *>(C->indices), static_cast<T *>(C->values),
        static_cast<const T *>(X->values), static_cast<const T *>(Y->values), (int)C->rows, k, (long long)C->nnz, st,
        alpha, beta, static_cast<const T *>(alphaDev), static_cast<const T *>(betaDev));
    b200sp_note_launches(1);
    return (int)cudaGetLastError();
}

// Whether Preprocess writes an order of the tiles: rows of Y in whole 16-byte pieces side by side, and tiles enough.
bool MayOrder(const aclsparseDnMatDescr *Y, const aclsparseSpMatDescr *C, aclsparseOperation_t opY)
{
    const bool rows = (opY == ACL_SPARSE_OP_TRANSPOSE) == (Y->order == ACL_SPARSE_ORDER_ROW);
    const long long bytes = Y->valueType == ACL_FLOAT16 ? 2 : 4;
    return rows && Y->ld * bytes % 16 == 0 && C->nnz >= kOrderLeast;
}

// While another stream is being captured, waiting for one that is not, or loading a kernel, would end that capture with an error unless this
// thread says that it knows what it does.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
};

// pieces: the 16-byte pieces of a row of Y.
cudaError_t OrderTiles(const aclsparseDnMatDescr *Y, long long pieces, const aclsparseSpMatDescr *C, void *buffer, cudaStream_t stream,
                       b200sp::TileOrderPlan *plan)
{
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) {
        (void)cudaGetLastError();
        return cudaSuccess;  // a product without an order is as good, only slower
    }
    const RelaxedCapture relaxed;
    const OrderLayout L = OrderLayoutFor(C->nnz);
    char *p = static_cast<char *>(buffer);
    int *counts = reinterpret_cast<int *>(p + L.offCounts), *starts = counts + kOrderBuckets + 1;
    auto *bucket = reinterpret_cast<int16_t *>(p + L.offBucket);
    const long long rowBytes = Y->ld * (Y->valueType == ACL_FLOAT16 ? 2ll : 4ll);
    const bool mayBeNear = C->cols * rowBytes >= kOrderMinY && C->nnz >= (pieces <= kNearNarrow ? kNearLeast : kNearLeastWide);
    if (!mayBeNear && pieces > kRowsPieces) return cudaSuccess;
    auto *order = reinterpret_cast<int2 *>(p + L.offTiles);
    const auto *rowPtr = static_cast<const int32_t *>(C->offsets);
    plan->generation = b200sp::NoteBufferWrite(buffer);
    int near = 0;
    cudaError_t e = cudaSuccess;
    if (mayBeNear) {
        const int span = (int)std::min<long long>(kNearSpan / rowBytes, C->cols / 3);
        e = cudaMemsetAsync(counts, 0, sizeof(int) * (kOrderBuckets + 1), stream);
        if (e != cudaSuccess) return e;
        const long long want = (L.tiles + 7) / 8, cap = (long long)b200sp_sm_count() * 8;
        SddmmTileBucketsKernel<<<(unsigned)(want < cap ? want : cap), 256, 0, stream>>>(
            static_cast<const int32_t *>(C->indices), (int)C->nnz, (int)C->cols, span, L.tiles, bucket, counts);
        SddmmBucketStartsKernel<<<1, kOrderBuckets, 0, stream>>>(counts, starts);
        e = cudaMemcpyAsync(&near, starts + kOrderBuckets, sizeof(near), cudaMemcpyDeviceToHost, stream);
        if (e != cudaSuccess) return e;
        SddmmOrderTilesKernel<<<(unsigned)((L.tiles + 1023) / 1024), 256, 0, stream>>>(rowPtr, (int)C->rows, bucket, L.tiles, starts, order,
                                                                                       reinterpret_cast<int *>(p + L.offPlace));
        b200sp_note_launches(3);
        e = cudaGetLastError();
        // Not only for the number of near tiles: a product on another stream must not find the order changed after it has looked it over.
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess) return e;
        if (near * kNearShare < L.tiles) {
            if (pieces > kRowsPieces) return cudaSuccess;
            near = 0;
        }
    }
    if (near == 0) {  // nothing is waited for: a product compares the rows with the row offsets
        SddmmTileRowsKernel<<<(unsigned)((L.tiles + 255) / 256), 256, 0, stream>>>(rowPtr, (int)C->rows, L.tiles, order);
        b200sp_note_launches(1);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    plan->near = near;
    plan->nnz = C->nnz;
    plan->buffer = buffer;
    return cudaSuccess;
}

// The order that Preprocess left in the buffer, if it is still there and worth following.
TileOrder OrderOf(const aclsparseSpMatDescr *C, const void *buffer)
{
    b200sp::TileOrderPlan plan;
    {
        std::lock_guard<std::mutex> lock(C->sddmmMutex);
        plan = C->sddmm;
    }
    const OrderLayout L = OrderLayoutFor(C->nnz);
    if (plan.buffer == nullptr || plan.buffer != buffer || plan.nnz != C->nnz || plan.generation != b200sp::BufferGeneration(buffer))
        return {};
    static std::atomic<unsigned> products{0};
    unsigned ticket = products.fetch_add(1, std::memory_order_relaxed) + 1;
    if (ticket == 0) ticket = products.fetch_add(1, std::memory_order_relaxed) + 1;  // what every place holds at first
    const char *p = static_cast<const char *>(buffer);
    return {reinterpret_cast<const int2 *>(p + L.offTiles), reinterpret_cast<const int *>(p + L.offPlace), ticket, plan.near,
            (((unsigned long long)plan.near << 32) + (unsigned long long)L.tiles - 1) / (unsigned long long)L.tiles};
}

}  // namespace

extern "C" {

aclsparseStatus_t aclsparseSDDMMBufferSize(aclsparseHandle_t handle, aclsparseOperation_t opX, aclsparseOperation_t opY,
                                           const void *alpha, aclsparseConstDnMatDescr_t matX,
                                           aclsparseConstDnMatDescr_t matY, const void *beta, aclsparseSpMatDescr_t matC,
                                           aclDataType computeType, aclsparseSDDMMAlg_t alg, size_t *size)
{
    if (handle == nullptr) return ACL_SPARSE_STATUS_HANDLE_IS_NULLPTR;  // order of sddmm_host.cpp:487-505
    if (size == nullptr) return ACL_SPARSE_STATUS_INVALID_VALUE;
    if (alpha == nullptr || beta == nullptr) return ACL_SPARSE_STATUS_INVALID_VALUE;
    const aclsparseStatus_t st = ValidateInputs(matX, matY, matC, opX, opY, computeType, alg);
    if (st != ACL_SPARSE_STATUS_SUCCESS) return st;
    *size = MayOrder(matY, matC, opY) ? OrderLayoutFor(matC->nnz).total : 256;
    std::lock_guard<std::mutex> lock(matC->sddmmMutex);
    matC->sddmm.sized = (int64_t)*size;
    return ACL_SPARSE_STATUS_SUCCESS;
}

aclsparseStatus_t aclsparseSDDMMPreprocess(aclsparseHandle_t handle, aclsparseOperation_t opX, aclsparseOperation_t opY,
                                           const void *alpha, aclsparseConstDnMatDescr_t matX,
                                           aclsparseConstDnMatDescr_t matY, const void *beta, aclsparseSpMatDescr_t matC,
                                           aclDataType computeType, aclsparseSDDMMAlg_t alg, void *buffer)
{
    const aclsparseStatus_t st = ValidateCall(handle, matX, matY, matC, alpha, beta, buffer, true, opX, opY, computeType, alg);
    if (st != ACL_SPARSE_STATUS_SUCCESS) return st;
    b200sp::TileOrderPlan plan;  // without an order
    {
        std::lock_guard<std::mutex> lock(matC->sddmmMutex);
        plan.sized = matC->sddmm.sized;
        matC->sddmm = plan;
    }
    if (!MayOrder(matY, matC, opY) || plan.sized < (int64_t)OrderLayoutFor(matC->nnz).total) return ACL_SPARSE_STATUS_SUCCESS;
    if (reinterpret_cast<uintptr_t>(buffer) % alignof(int2) != 0) return ACL_SPARSE_STATUS_SUCCESS;  // any address is accepted
    if (b200sp::HoldsPlan(buffer)) return ACL_SPARSE_STATUS_SUCCESS;
    const int64_t k = opX == ACL_SPARSE_OP_TRANSPOSE ? matX->rows : matX->cols;
    if (OrderTiles(matY, (k * (matY->valueType == ACL_FLOAT16 ? 2 : 4) + 15) / 16, matC, buffer, handle->stream, &plan) != cudaSuccess) {
        B200SP_LOGE("aclsparseSDDMMPreprocess: analysis failed");
        return ACL_SPARSE_STATUS_EXECUTION_FAILED;
    }
    if (plan.buffer != nullptr) {
        std::lock_guard<std::mutex> lock(matC->sddmmMutex);
        plan.sized = matC->sddmm.sized;
        matC->sddmm = plan;
    }
    return ACL_SPARSE_STATUS_SUCCESS;
}

aclsparseStatus_t aclsparseSDDMM(aclsparseHandle_t handle, aclsparseOperation_t opX, aclsparseOperation_t opY,
                                 const void *alpha, aclsparseConstDnMatDescr_t matX, aclsparseConstDnMatDescr_t matY,
                                 const void *beta, aclsparseSpMatDescr_t matC, aclDataType computeType,
                                 aclsparseSDDMMAlg_t alg, void *buffer)
{
    const aclsparseStatus_t st = ValidateCall(handle, matX, matY, matC, alpha, beta, buffer, false, opX, opY, computeType, alg);
    if (st != ACL_SPARSE_STATUS_SUCCESS) return st;
    if (matC->nnz == 0 || matC->rows == 0) return ACL_SPARSE_STATUS_SUCCESS;
    const bool xT = opX == ACL_SPARSE_OP_TRANSPOSE, yT = opY == ACL_SPARSE_OP_TRANSPOSE;
    const bool xRow = matX->order == ACL_SPARSE_ORDER_ROW, yRow = matY->order == ACL_SPARSE_ORDER_ROW;
    const int k = (int)(xT ? matX->rows : matX->cols);
    Strides s;
    // stored X is (m x k) or, transposed, (k x m); element (row, col) sits at row * ld + col (row-major) or
    // row + col * ld (column-major)
    const bool xContigK = xT ? !xRow : xRow;  // k runs along the contiguous direction
    s.xi = xContigK ? matX->ld : 1;
    s.xk = xContigK ? 1 : matX->ld;
    const bool yContigK = yT ? yRow : !yRow;  // stored Y is (k x n) or, transposed, (n x k)
    s.yk = yContigK ? 1 : matY->ld;
    s.yj = yContigK ? matY->ld : 1;
    const bool host = handle->pointerMode == ACL_SPARSE_POINTER_MODE_HOST;
    const float a = host ? ReadScalar(alpha, computeType) : 0.0f;
    const float b = host ? ReadScalar(beta, computeType) : 0.0f;
    const void *aDev = host ? nullptr : alpha;
    const void *bDev = host ? nullptr : beta;
    const TileOrder order = OrderOf(matC, buffer);
    const int rc = computeType == ACL_FLOAT16
                       ? Launch<__half>(matC, matX, matY, k, s, a, b, aDev, bDev, order, handle->stream)
                       : Launch<float>(matC, matX, matY, k, s, a, b, aDev, bDev, order, handle->stream);
    if (rc != 0) {
        B200SP_LOGE("aclsparseSDDMM: kernel launch failed (cuda error %d)", rc);
        return ACL_SPARSE_STATUS_EXECUTION_FAILED;
    }
    return ACL_SPARSE_STATUS_SUCCESS;
}

}  // extern "C"
