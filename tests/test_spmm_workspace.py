"""CPU: when aclsparseSpMMGetBufferSize asks for room to write a dense int8 A out for the tensor cores."""
from __future__ import annotations

from ctypes import byref, c_int64, c_size_t, c_void_p

import pytest

FAKE = c_void_p(0x1000)  # sizes only: nothing is read


def extra_bytes(pkg, m, k, nnz, n, order="row"):
    """Bytes of the buffer beyond those of the analysis."""
    L, S = pkg.lib(), pkg
    A, B, C, size = c_void_p(), c_void_p(), c_void_p(), c_size_t()
    col = order == "col"
    assert L.aclsparseCreateCsr(byref(A), m, k, nnz, FAKE, FAKE, FAKE, S.ACL_SPARSE_INDEX_32I, S.ACL_SPARSE_INDEX_32I, 0, S.ACL_INT8) == 0
    layout = S.ACL_SPARSE_ORDER_COL if col else S.ACL_SPARSE_ORDER_ROW
    assert L.aclsparseCreateDnMat(byref(B), k, n, k if col else n, FAKE, S.ACL_INT8, layout) == 0
    assert L.aclsparseCreateDnMat(byref(C), m, n, m if col else n, FAKE, S.ACL_INT32, layout) == 0
    handle = c_void_p()
    assert L.aclsparseSpMMGetBufferSize(handle, 0, 0, None, A, B, None, C, S.ACL_INT32, 0, byref(size)) == 0
    L.b200sp_spmm_plan_bytes.argtypes, L.b200sp_spmm_plan_bytes.restype = [c_int64] * 3, c_size_t
    extra = size.value - L.b200sp_spmm_plan_bytes(m, nnz, n)
    assert L.aclsparseDestroySpMat(A) == 0 and L.aclsparseDestroyDnMat(B) == 0 and L.aclsparseDestroyDnMat(C) == 0
    return extra


# one twelfth full as a matrix, but not as rows of 128 bytes; full enough, but a tile has too little work; wider, the same
@pytest.mark.parametrize("m,k,mean,n", [(2000000, 1, 1, 64), (10000000, 12, 1, 16), (1000000, 16, 4, 64), (500000, 64, 16, 64),
                                        (200000, 128, 11, 64), (200000, 128, 16, 64), (100000, 256, 38, 64), (100000, 512, 77, 32)])
def test_thin_matrices_stay_sparse(pkg, m, k, mean, n):
    assert extra_bytes(pkg, m, k, m * mean, n) == 0


@pytest.mark.parametrize("m,k,mean,n,order", [(4096, 4096, 410, 512, "row"), (40000, 2000, 300, 16, "row"), (100000, 1024, 154, 128, "row"),
                                              (100000, 512, 77, 128, "row"), (100000, 512, 154, 16, "row"), (30000, 512, 76, 100, "col")])
def test_dense_matrices_have_room(pkg, m, k, mean, n, order):
    assert extra_bytes(pkg, m, k, m * mean, n, order) >= m * k


def test_no_more_than_four_gigabytes(pkg):
    assert extra_bytes(pkg, 500000, 8192, 500000 * 1000, 64) >= 500000 * 8192
    assert extra_bytes(pkg, 600000, 8192, 600000 * 1000, 64) == 0
