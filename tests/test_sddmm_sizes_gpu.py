"""GPU: aclsparseSDDMM at the widths and entry counts where its row kernel changes (lanes and pieces of a row, several
turns, odd fp16 widths, ends of a warp's tile of entries)."""
from __future__ import annotations

import numpy as np
import pytest

from test_sddmm_gpu import dense_operand, golden, run_sddmm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("pad", [0, 1])  # 1: rows that start on any element
@pytest.mark.parametrize("k", [1, 2, 3, 4, 7, 8, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 256, 257, 511, 512, 513, 1024, 1100])
def test_widths(pkg, handle, device, k, pad, dtype):
    rng = np.random.default_rng(k)
    check(pkg, handle, device, rng, rng.integers(0, 9, 90), k, pad, dtype)


# pieces of 16 bytes in a row on either side of every change of lanes per row and pieces per lane
@pytest.mark.parametrize("pieces", [4, 5, 8, 9, 12, 13, 15, 16, 17, 24, 25, 32, 33, 48, 49, 64, 65, 96, 97, 128, 129])
@pytest.mark.parametrize("dtype", ["f32", "f16"])
def test_pieces(pkg, handle, device, pieces, dtype):
    rng = np.random.default_rng(pieces)
    check(pkg, handle, device, rng, rng.integers(0, 9, 90), pieces * (4 if dtype == "f32" else 8), 0, dtype)


# one to four entries a batch, tiles of 32 and 64 entries: every shape at entry counts on either side of where they change, which depends
# on the shared memory of a shape; pieces of 16, 8, 4 and 2 bytes
@pytest.mark.parametrize("nnz", [18944, 37889, 75777, 151553, 260003])
@pytest.mark.parametrize("dtype,k", [("f16", 32), ("f16", 64), ("f16", 80), ("f16", 104), ("f16", 112), ("f16", 192), ("f16", 256), ("f16", 384),
                                     ("f32", 256), ("f16", 768), ("f32", 512), ("f32", 600), ("f16", 20), ("f16", 36), ("f16", 100), ("f16", 204),
                                     ("f16", 300), ("f16", 500), ("f16", 18), ("f32", 129), ("f16", 23), ("f16", 401)])
def test_entries_in_flight(pkg, handle, device, dtype, k, nnz):
    rng = np.random.default_rng(nnz + k)
    check(pkg, handle, device, rng, np.bincount(rng.integers(0, 9000, nnz), minlength=9000), k, 0, dtype)


@pytest.mark.parametrize("nnz", [1, 3, 4, 5, 31, 32, 33, 63, 64, 65, 129, 148 * 16 * 128 + 1])  # the last: tiles of 64 entries
def test_entry_counts(pkg, handle, device, nnz):
    rng = np.random.default_rng(nnz)
    lengths = np.bincount(rng.integers(0, 50, nnz), minlength=50)
    check(pkg, handle, device, rng, lengths, 24, 0, "f16")


@pytest.mark.parametrize("dtype,k,n", [("f32", 64, 47), ("f32", 64, 48), ("f32", 64, 49), ("f16", 16, 9), ("f16", 1024, 6), ("f16", 1024, 7)])
def test_few_rows_of_y(pkg, handle, device, dtype, k, n):
    """Y up to 12 KB comes through L1, a larger one past it."""
    rng = np.random.default_rng(n)
    check(pkg, handle, device, rng, rng.integers(0, 9, 90), k, 0, dtype, n)


def check(pkg, handle, device, rng, lengths, k, pad, dtype, n=300):
    m = lengths.size
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    ci = rng.integers(0, n, rp[-1]).astype(np.int32)
    X, xs, ldx = dense_operand(rng, m, k, "row", pad, dtype)
    Yt, ys, ldy = dense_operand(rng, n, k, "row", pad, dtype)
    c0 = rng.uniform(-1.0, 1.0, ci.size).astype(np.float32)
    if dtype == "f16":
        c0 = c0.astype(np.float16).astype(np.float32)
    got = run_sddmm(pkg, handle, device, rp, ci, c0, (xs, m, k, ldx), (ys, n, k, ldy), 1.5, -0.5, m, n, False, True,
                    "row", "row", dtype)
    want, scale = golden(rp, ci, c0, X, np.ascontiguousarray(Yt.T), 1.5, -0.5)
    tol = 1e-5 * scale + 1e-30 if dtype == "f32" else 2e-3 * scale + np.abs(want) * 2.0 ** -11 + 2.0 ** -25
    assert np.all(np.abs(got - want) <= tol)


def test_odd_rows_of_two_gigabytes(pkg, handle, device):
    """A width whose bytes do not fit 31 bits: an element at either end of the row and one in the middle count."""
    import torch
    from ops_sparse_b200 import api
    from ctypes import addressof, c_uint16, c_void_p
    k = (1 << 30) + 1
    X, Y = (make(1, k, dtype=torch.float16, device=device) for make in (torch.zeros, torch.ones))
    X[0, 0], X[0, k // 2], X[0, k - 1] = 2, 3, 5
    C = api.CsrMatrix(torch.tensor([0, 1], dtype=torch.int32, device=device), torch.zeros(1, dtype=torch.int32, device=device),
                      torch.full((1,), 4.0, dtype=torch.float16, device=device), 1, 1)
    dX, dY = api.DnMat.row_major(X), api.DnMat.row_major(Y)
    alpha, beta = (c_uint16(int(np.float16(v).view(np.uint16))) for v in (1.0, 0.5))
    buf = torch.empty(256, dtype=torch.uint8, device=device)
    pkg.check(pkg.lib().aclsparseSDDMM(handle.raw, 0, pkg.ACL_SPARSE_OP_TRANSPOSE, c_void_p(addressof(alpha)), dX.raw, dY.raw,
                                       c_void_p(addressof(beta)), C.raw, pkg.ACL_FLOAT16, 0, c_void_p(buf.data_ptr())),
              "aclsparseSDDMM")
    assert C.values.item() == 12.0
