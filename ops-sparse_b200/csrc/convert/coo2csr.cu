// aclsparseXcoo2csr: sorted COO row indices -> CSR row offsets.
// Checks and their order follow the reference host layer (sparse/coo2csr/arch35/coo2csr_host.cpp:38-78);
// the reference counts the entries of every row and prefix-sums the counts, which for the sorted input the
// API requires is the same as csrRowPtr[i] = base + |{k : cooRowInd[k] < i + base}|.  Here one thread per
// output looks that position up by binary search: one pass, no workspace, no atomics.
#include <climits>
#include <cstdint>

#include <cuda_runtime.h>

#include "b200sp_kernels.h"
#include "common/chained.cuh"
#include "common/internal.h"
#include "common/rows.cuh"

namespace {

// Bound by the latency of the probes: 256 rows share one bracket, so that a thread's search covers their entries only
// (31 M entries, 1 M rows: 38 us with a search of the whole array per row, 35 now).
__global__ void __launch_bounds__(256) Coo2CsrKernel(const int *__restrict__ cooRowInd, int nnz, int m,
                                                     int *__restrict__ csrRowPtr, int base)
{
    b200sp::WaitForPrevious();
    for (long long i0 = (long long)blockIdx.x * 256; i0 <= m; i0 += (long long)gridDim.x * 256)
        b200sp::OffsetsOfSorted(cooRowInd, nnz, i0, m, base, base, csrRowPtr);
}

}  // namespace

extern "C" aclsparseStatus_t aclsparseXcoo2csr(aclsparseHandle_t handle, const int *cooRowInd, int nnz, int m,
                                               int *csrRowPtr, aclsparseIndexBase_t idxBase)
{
    if (handle == nullptr) return ACL_SPARSE_STATUS_HANDLE_IS_NULLPTR;
    if (nnz < 0) return ACL_SPARSE_STATUS_INVALID_VALUE;
    if (nnz == INT32_MAX && idxBase == ACL_SPARSE_INDEX_BASE_ONE) return ACL_SPARSE_STATUS_INVALID_VALUE;  // nnz + 1 overflows
    if (m < 0) return ACL_SPARSE_STATUS_INVALID_VALUE;
    if (nnz > 0 && m == 0) return ACL_SPARSE_STATUS_INVALID_VALUE;
    if (idxBase != ACL_SPARSE_INDEX_BASE_ZERO && idxBase != ACL_SPARSE_INDEX_BASE_ONE)
        return ACL_SPARSE_STATUS_INVALID_VALUE;
    if (nnz > 0 && cooRowInd == nullptr) return ACL_SPARSE_STATUS_INVALID_VALUE;
    if (csrRowPtr == nullptr) return ACL_SPARSE_STATUS_INVALID_VALUE;

    const long long want = ((long long)m + 1 + 255) / 256;
    const long long cap = (long long)b200sp_sm_count() * 32;
    const cudaError_t e =
        b200sp::LaunchChained(Coo2CsrKernel, (unsigned)(want < cap ? want : cap), 256, 0, handle->stream, cooRowInd, nnz, m,
                              csrRowPtr, idxBase == ACL_SPARSE_INDEX_BASE_ONE ? 1 : 0);
    b200sp_note_launches(1);
    if (e != cudaSuccess) {
        B200SP_LOGE("aclsparseXcoo2csr: kernel launch failed (%s)", cudaGetErrorString(e));
        return ACL_SPARSE_STATUS_EXECUTION_FAILED;
    }
    return ACL_SPARSE_STATUS_SUCCESS;
}
