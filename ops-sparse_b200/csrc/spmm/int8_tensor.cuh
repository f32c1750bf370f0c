// int8 products whose A is dense enough for the tensor cores (pruned weights): included by spmm_kernels.cu.
//
// A CTA computes 128 rows of C by up to 128 columns with tcgen05.mma (kind::i8, accumulators in tensor memory).  The CTAs of
// the same rows are a cluster: together they first write those rows of A out as dense rows of bytes, in a workspace that stays in
// L2, and then read them back, with B, in swizzled tiles.  B is read as it lies: its rows hold consecutive columns of C, which
// the tensor core takes as an "MN-major" operand.  Sums of integers may be regrouped, so the result is that of every other int8
// kernel, bit for bit (wrapping 32-bit sums).
//   - Only rows whose columns ascend, without repetition, can be written out (a repeated column would want the sum of its
//     values in one byte).  The analysis admits no others, and every entry is still compared with the one before it: a
//     row that fails is marked, and its outputs are summed entry by entry instead.
//   - Tiles of 128 columns of A and as many rows of B come through seven stages of shared memory by TMA, requested by one thread; another
//     starts the products.
// 4096 x 4096 at one tenth, N = 512: 69 us with the lane groups of SpmmFastKernel, 24 here: every SM fetches 1.1 MB from L2, at least 9.4 us
// at the 62 bytes per clock that it gets; before that the rows are written out and the cluster meets, and the tensor cores
// work in 19 % of the cycles.
// Writing the rows of A straight into the swizzled tiles, by every CTA for itself, took 68 us (some hundred
// instructions per row and step), tiles by cp.async, which wants a proxy fence before every step, 28 us.
// Every wait is bounded, as in the row-stream kernel.  After one that ran out the CTA sums its part of C entry by entry, straight from
// A and B: no output is lost, and none comes from shared or tensor memory that a copy or a product may still be writing.
#pragma once

constexpr int kTcRows = 128;                // rows of a CTA: the lanes of tensor memory
constexpr int kTcCols = 128;                // columns of C of a CTA at most: the bytes of a swizzled row of B
constexpr int kTcDepth = 128;               // columns of A (rows of B) per stage
constexpr int kTcThreads = 512;
constexpr int kTcWarps = kTcThreads / 32;
constexpr int kTcCluster = 4;               // CTAs that share the rows of A at most; twice as many where there are few rows
constexpr int kTcStages = 7;
constexpr int kTcTileBytes = kTcRows * kTcDepth;                     // of A, and of B: rows of 128 bytes
constexpr int kTcSmem = 2 * kTcStages * kTcTileBytes + 1024;         // tiles start on multiples of 1024 bytes
constexpr int kTcPitch = kTcCols + 4;       // of the sums in shared memory
constexpr long long kTcMaxK = 12288;        // every warp has a row of A, written out, in the stages' shared memory
constexpr long long kTcMaxDense = 4ll << 30;  // bytes of A written out
static_assert(kTcMaxK * kTcWarps <= 2 * kTcStages * kTcTileBytes);
static_assert(kTcRows * kTcPitch * 4 <= 2 * kTcStages * kTcTileBytes);

// Columns of A as written out, and the bytes of that and of a mark per row.
inline long long DenseCols(long long k) { return (k + kTcDepth - 1) / kTcDepth * kTcDepth; }
inline size_t DenseBytes(long long m, long long k) { return AlignUp((size_t)m * (size_t)DenseCols(k), 256) + AlignUp((size_t)m, 256); }

// Whether the columns of every row ascend without repetition.
__global__ void __launch_bounds__(256) SpmmAscendingKernel(const int32_t *__restrict__ rowPtr, const int32_t *__restrict__ colInd,
                                                           int rows, int32_t *notAscending)
{
    const int lane = threadIdx.x & 31;
    bool bad = false;
    for (long long r = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += (long long)gridDim.x * 8) {
        const int s = rowPtr[r], len = rowPtr[r + 1] - s;
        // unsigned, from the row's start: a row may end at the last entry that 31 bits count
        for (unsigned i = lane; i + 1 < (unsigned)len; i += 32) bad |= colInd[s + i] >= colInd[s + i + 1];
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicExch(notAscending, 1);
}

struct TcArgs {
    const int32_t *rowPtr, *colInd;
    const int8_t *val, *B;
    unsigned char *dense, *odd;    // A written out, and marks of the rows that could not be
    int32_t *C;
    int m, n, chunks;              // chunks: steps of kTcDepth columns of A
    int cols, colTiles, firstCol;  // columns of C of a CTA: 32, 64 or 128; CTAs of the cluster; first column of all
    long long ldb, cRow, cCol;     // element (r, j) of C lies at r * cRow + j * cCol
    int cVectors;                  // rows of C take 16 bytes at a time
    ScalarsI sc;
    long long waitCycles;
    unsigned extraTx;              // bytes expected on every barrier beyond those copied (0 outside the wait test)
};

__device__ __forceinline__ void TcAlloc(uint32_t *out, uint32_t columns)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(SmemAddr(out)), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void TcFree(uint32_t at, uint32_t columns)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(at), "r"(columns) : "memory");
}
// Shared-memory matrix descriptor: rows of 128, 64 or 32 bytes swizzled over their whole width, groups of eight side by side.
// A: rows of the matrix along 128 bytes of its columns; B: rows of B along the CTA's columns of C.
__device__ __forceinline__ uint64_t TcDescriptor(uint32_t at, uint32_t rowBytes)
{
    const uint64_t group = 8 * rowBytes >> 4, swizzle = rowBytes == 128 ? 2 : rowBytes == 64 ? 4 : 6;
    return (uint64_t)((at & 0x3ffff) >> 4) | group << 16 | group << 32 | 1ull << 46 | swizzle << 61;
}
__device__ __forceinline__ void TcMma(uint32_t d, uint64_t a, uint64_t b, uint32_t instr, bool add)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(instr), "r"((uint32_t)add)
                 : "memory");
}
__device__ __forceinline__ void TcCommit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(SmemAddr(bar)) : "memory");
}
__device__ __forceinline__ void TcLoad16(uint32_t at, int32_t (&v)[16])
{
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(at));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = (int32_t)r[i];
}
__device__ __forceinline__ void TcCopyTile(uint32_t dst, const CUtensorMap *map, int x, int y, uint64_t *bar)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(map), "r"(x), "r"(y), "r"(SmemAddr(bar))
                 : "memory");
}

// Up to kTcWindows windows of 32 entries of a row, all requested before the first is looked at.  4 windows: 27.2 us, 8: 24.4, 16: 24.2 for
// the product above; 15.3, 15.0 and 17.7 for 3000 rows of 100 entries.
constexpr int kTcWindows = 8;
struct TcEntries {
    uint32_t col[kTcWindows];
    int8_t val[kTcWindows];
    // len: entries from `from` on.  Lengths are compared, not positions: from + 32 * h + lane may not fit 31 bits.
    __device__ __forceinline__ void Request(const TcArgs &a, int from, int len, int lane)
    {
#pragma unroll
        for (int h = 0; h < kTcWindows; ++h) {
            const int i = 32 * h + lane;
            col[h] = 0x80000000u + i;  // past the end: ascending too, and in no row
            val[h] = 0;
            if (i < len) {
                col[h] = (uint32_t)__ldg(a.colInd + from + i);
                val[h] = __ldg(a.val + from + i);
            }
        }
    }
    // Writes them into the row; true if one is not above the one before it (least: what the first is at least).
    __device__ __forceinline__ bool Write(unsigned char *sRow, int width, uint32_t &least, int lane) const
    {
        bool bad = false;
#pragma unroll
        for (int h = 0; h < kTcWindows; ++h) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, col[h], 1) + 1;
            bad |= col[h] < (lane == 0 ? least : up);
            least = __shfl_sync(0xffffffffu, col[h], 31) + 1;
            if (col[h] < (uint32_t)width) reinterpret_cast<int8_t *>(sRow)[col[h]] = val[h];
        }
        return bad;
    }
};

// Row `row` of A as bytes, through a row of zeros in shared memory; its first entries are in hand.
__device__ __forceinline__ void TcExpandRow(const TcArgs &a, int row, int from, int len, const TcEntries &first, unsigned char *sRow,
                                            int lane)
{
    const int width = a.chunks * kTcDepth;
    uint4 *const sPieces = reinterpret_cast<uint4 *>(sRow);
    for (int i = lane; i < width / 16; i += 32) sPieces[i] = make_uint4(0, 0, 0, 0);
    __syncwarp();
    uint32_t least = 0;
    bool bad = first.Write(sRow, width, least, lane);
    for (int left = len - 32 * kTcWindows; left > 0; left -= 32 * kTcWindows) {
        TcEntries more;
        more.Request(a, from + (len - left), left, lane);
        bad |= more.Write(sRow, width, least, lane);
    }
    bad = __any_sync(0xffffffffu, bad);
    __syncwarp();  // bytes of other lanes are read from here on: votes order no memory
    uint4 *const out = reinterpret_cast<uint4 *>(a.dense + (long long)row * width);
    for (int i = lane; i < width / 16; i += 32) out[i] = sPieces[i];
    if (lane == 0) a.odd[row] = bad;
    __syncwarp();
}

// One element of A * B, entry by entry.
__device__ __forceinline__ int32_t TcSum(const TcArgs &a, int row, int col)
{
    int32_t sum = 0;
    for (int p = a.rowPtr[row]; p < a.rowPtr[row + 1]; ++p)
        sum += (int32_t)a.val[p] * (int32_t)a.B[(long long)a.colInd[p] * a.ldb + col];
    return sum;
}

__global__ void __launch_bounds__(kTcThreads, 1) SpmmInt8TensorKernel(const TcArgs a, const __grid_constant__ CUtensorMap mapA,
                                                                      const __grid_constant__ CUtensorMap mapB)
{
    extern __shared__ unsigned char sRaw[];
    __shared__ uint64_t sFull[kTcStages], sEmpty[kTcStages], sDone;
    __shared__ uint32_t sTmem;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t base = (SmemAddr(sRaw) + 1023u) & ~1023u;
    unsigned char *const tiles = sRaw + (base - SmemAddr(sRaw));
    if (warp == 0) TcAlloc(&sTmem, kTcCols);
    if (tid == 0) {
        for (int s = 0; s < kTcStages; ++s) {
            MbarInit(sFull + s, 1);
            MbarInit(sEmpty + s, 1);
        }
        MbarInit(&sDone, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    b200sp::WaitForPrevious();
    const int rank = blockIdx.x % a.colTiles;
    const int row0 = (int)(blockIdx.x / a.colTiles) * kTcRows;
    const int n0 = a.firstCol + rank * a.cols;
    {  // lane t has the start and the length of the warp's t-th row; two rows at a time
        unsigned char *const sRow = tiles + warp * a.chunks * kTcDepth;
        const int first = rank * kTcWarps + warp, step = a.colTiles * kTcWarps;  // rows of the tile: first, first + step, ...
        const int own = row0 + first + lane * step;
        const bool some = first + lane * step < kTcRows && own < a.m;
        const int ownFrom = some ? __ldg(a.rowPtr + own) : 0, ownLen = some ? __ldg(a.rowPtr + own + 1) - ownFrom : 0;
        for (int t = 0; first + t * step < kTcRows && row0 + first + t * step < a.m; t += 2) {
            const int row = row0 + first + t * step;
            const int from0 = __shfl_sync(0xffffffffu, ownFrom, t), len0 = __shfl_sync(0xffffffffu, ownLen, t);
            const int from1 = __shfl_sync(0xffffffffu, ownFrom, t + 1), len1 = __shfl_sync(0xffffffffu, ownLen, t + 1);
            TcEntries e0, e1;
            e0.Request(a, from0, len0, lane);
            e1.Request(a, from1, len1, lane);
            TcExpandRow(a, row, from0, len0, e0, sRow, lane);
            if (first + (t + 1) * step < kTcRows && row + step < a.m) TcExpandRow(a, row + step, from1, len1, e1, sRow, lane);
        }
    }
    // What was stored, here and by the rest of the cluster, is read, and the shared memory written, by TMA from here on.
    asm volatile("fence.proxy.async;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    asm volatile("fence.proxy.async;" ::: "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sTmem;
    // marks of the rows this warp will write (lane t: its t-th), asked for before they are wanted
    const int markRow = row0 + warp + lane * kTcWarps;
    const unsigned odd = __ballot_sync(0xffffffffu, lane < kTcRows / kTcWarps && markRow < a.m && __ldcg(a.odd + markRow) != 0);

    bool failed = false;
    int asked = 0;  // of the requesting thread: steps whose tiles it asked for
    if (tid == 0) {
        for (; asked < a.chunks; ++asked) {
            const int s = asked % kTcStages, use = asked / kTcStages;
            if (use > 0 && !MbarWait(sEmpty + s, (uint32_t)(use - 1) & 1u, a.waitCycles)) {
                failed = true;
                break;
            }
            const uint32_t tile = base + s * 2 * kTcTileBytes;
            MbarExpectTx(sFull + s, kTcTileBytes + a.cols * kTcDepth + a.extraTx);
            TcCopyTile(tile, &mapA, asked * kTcDepth, row0, sFull + s);
            TcCopyTile(tile + kTcTileBytes, &mapB, n0, asked * kTcDepth, sFull + s);
        }
    } else if (tid == 32) {
        // 32-bit sums, signed 8-bit operands, B MN-major
        const uint32_t instr = 2u << 4 | 1u << 7 | 1u << 10 | 1u << 16 | (uint32_t)(a.cols >> 3) << 17 | (uint32_t)(kTcRows >> 4) << 24;
        for (int c = 0; c < a.chunks; ++c) {
            const int s = c % kTcStages;
            if (!MbarWait(sFull + s, (uint32_t)(c / kTcStages) & 1u, a.waitCycles)) {
                failed = true;
                break;
            }
            const uint32_t tile = base + s * 2 * kTcTileBytes;
#pragma unroll
            for (int i = 0; i < kTcDepth / 32; ++i)
                TcMma(tmem, TcDescriptor(tile + i * 32, kTcDepth), TcDescriptor(tile + kTcTileBytes + i * 32 * a.cols, a.cols), instr,
                      c > 0 || i > 0);
            TcCommit(sEmpty + s);
        }
        TcCommit(&sDone);  // when every product started here is complete, also after a failure
    }
    __syncwarp();
    if (!MbarWait(&sDone, 0, 4 * a.waitCycles)) failed = true;  // longer than the waits above may take one after the other
    failed = __syncthreads_or(failed) != 0;
    const int32_t alpha = a.sc.Alpha(), beta = a.sc.Beta();
    const int live = min(a.cols, a.n - n0);  // columns
    if (failed && tid == 0) {
        for (int c = asked > kTcStages ? asked - kTcStages : 0; c < asked; ++c)  // copies on their way: a bounded chance to land
            (void)MbarWait(sFull + c % kTcStages, (uint32_t)(c / kTcStages) & 1u, a.waitCycles);
    }
    if (!failed) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // The sums go through shared memory (the stages are done with), so that rows of C are written whole.
        const int quarter = warp & 3;  // a warp reads the lanes of tensor memory that are its rank modulo four
        int32_t *const sSums = reinterpret_cast<int32_t *>(tiles);
        for (int j0 = (warp >> 2) * 16; j0 < a.cols; j0 += kTcThreads / 128 * 16) {
            int32_t acc[16];
            TcLoad16(tmem + ((uint32_t)quarter << 21) + j0, acc);
            int4 *const to = reinterpret_cast<int4 *>(sSums + (quarter * 32 + lane) * kTcPitch + j0);
#pragma unroll
            for (int i = 0; i < 4; ++i) to[i] = make_int4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
        }
        __syncthreads();
        const bool plain = alpha == 1 && beta == 0;
        for (int r = warp; r < kTcRows && row0 + r < a.m; r += kTcWarps) {
            const int row = row0 + r;
            int32_t *const sums = sSums + r * kTcPitch;
            if (odd >> (r / kTcWarps) & 1) {
                for (int j = lane; j < live; j += 32) sums[j] = TcSum(a, row, n0 + j);
                __syncwarp();
            }
            if (a.cCol != 1) continue;
            int32_t *const out = a.C + row * a.cRow + n0;
            if (a.cVectors) {
                const int j = lane * 4;
                if (j + 4 <= live) {
                    const int4 v = *reinterpret_cast<const int4 *>(sums + j);
                    if (plain) {
                        __stcs(reinterpret_cast<int4 *>(out + j), v);
                        continue;
                    }
                    int4 old = make_int4(0, 0, 0, 0);
                    if (beta != 0) old = __ldcs(reinterpret_cast<const int4 *>(out + j));
                    __stcs(reinterpret_cast<int4 *>(out + j),
                           make_int4(Finish<int32_t>(v.x, alpha, beta, &old.x), Finish<int32_t>(v.y, alpha, beta, &old.y),
                                     Finish<int32_t>(v.z, alpha, beta, &old.z), Finish<int32_t>(v.w, alpha, beta, &old.w)));
                } else {
                    for (int i = j; i < live; ++i) out[i] = Finish<int32_t>(sums[i], alpha, beta, out + i);
                }
            } else {
                for (int j = lane; j < live; j += 32) out[j] = Finish<int32_t>(sums[j], alpha, beta, out + j);
            }
        }
        if (a.cCol != 1) {  // columns of C: lanes along the rows
            __syncthreads();
            for (int j = warp; j < live; j += kTcWarps) {
                int32_t *const out = a.C + (n0 + j) * a.cCol;
                for (int r = lane; r < kTcRows && row0 + r < a.m; r += 32) {
                    int32_t *const at = out + (row0 + r) * a.cRow;
                    *at = Finish<int32_t>(sSums[r * kTcPitch + j], alpha, beta, at);
                }
            }
        }
    } else {
        for (int r = warp; r < kTcRows && row0 + r < a.m; r += kTcWarps) {
            for (int j = lane; j < live; j += 32) {
                int32_t *const at = a.C + (row0 + r) * a.cRow + (n0 + j) * a.cCol;
                *at = Finish<int32_t>(TcSum(a, row0 + r, n0 + j), alpha, beta, at);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) TcFree(tmem, kTcCols);
}
