"""GPU: aclsparseSpMM on a B that is copied into the analysed buffer (columns contiguous): where there is room for the copy,
and who may use it."""
from __future__ import annotations

import threading
from ctypes import byref, c_size_t, c_void_p

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

M, K, N, PER_ROW = 3000, 2500, 40, 24  # more than a wave of short rows, every B row read often: worth a copy


class Case:
    """A matrix and products with several column-major B; every sum is a whole number below 2^11, so any order is exact."""

    def __init__(self, device, seed=0, matrices=1):
        from ops_sparse_b200 import api
        rng = np.random.default_rng(seed)
        rp = np.arange(M + 1, dtype=np.int32) * PER_ROW
        ci = rng.integers(0, K, M * PER_ROW).astype(np.int32)
        val = rng.integers(-3, 4, ci.size).astype(np.float16)
        up = lambda a: torch.from_numpy(a).to(device)
        self.A = api.CsrMatrix(up(rp), up(ci), up(val), M, K)
        dense = np.zeros((M, K))
        np.add.at(dense, (np.repeat(np.arange(M), PER_ROW), ci), val.astype(np.float64))
        self.B, self.C, self.want = [], [], []
        for _ in range(matrices):
            b = rng.integers(-3, 4, (K, N)).astype(np.float16)
            self.B.append(api.DnMat(up(np.ascontiguousarray(b.T)), K, N, K, "col"))
            self.C.append(api.DnMat(torch.zeros(N, M, dtype=torch.float16, device=device), M, N, M, "col"))
            self.want.append((dense @ b.astype(np.float64)).T)
        self.row_major_B = api.DnMat(torch.zeros(K, N, dtype=torch.float16, device=device), K, N, N, "row")

    def right(self, i, C=None):
        return np.array_equal((C or self.C[i]).values.cpu().numpy().astype(np.float64), self.want[i])


def preprocess(pkg, handle, case, buffer):
    p = lambda t: c_void_p(t.data_ptr())
    assert pkg.lib().aclsparseSpMMPreprocess(handle.raw, 0, 0, None, case.A.raw, case.B[0].raw, None, case.C[0].raw,
                                             pkg.ACL_FLOAT, 0, p(buffer)) == 0


def test_buffer_sized_for_another_layout(pkg, handle, device):
    """A buffer sized with a row-major B has no room for a copy: nothing is written behind it."""
    from ops_sparse_b200 import api
    case = Case(device)
    copied = api.spmm_buffer_size(handle, case.A, case.B[0], case.C[0])
    size = api.spmm_buffer_size(handle, case.A, case.row_major_B, case.C[0])
    assert copied - size >= K * N * 2
    arena = torch.full((copied + 4096,), 0x5A, dtype=torch.uint8, device=device)
    preprocess(pkg, handle, case, arena[:size])
    api.spmm(handle, case.A, case.B[0], case.C[0], 1.0, 0.0, buffer=arena[:size])
    assert case.right(0)
    assert bool((arena[size:] == 0x5A).all())


def test_buffer_on_any_word(pkg, handle, device):
    """A buffer that does not start on a 16-byte boundary holds the plan, but no copy."""
    from ops_sparse_b200 import api
    case = Case(device)
    size = api.spmm_buffer_size(handle, case.A, case.B[0], case.C[0])
    buffer = torch.empty(size + 4, dtype=torch.uint8, device=device)[4:]
    preprocess(pkg, handle, case, buffer)
    api.spmm(handle, case.A, case.B[0], case.C[0], 1.0, 0.0, buffer=buffer)
    assert case.right(0)
