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


@pytest.fixture()
def shared(pkg, handle, device):
    """A matrix analysed once, four B, and a graph of the product with the last of them."""
    from ops_sparse_b200 import api
    case = Case(device, seed=1, matrices=4)
    buffer = torch.empty(api.spmm_buffer_size(handle, case.A, case.B[0], case.C[0]), dtype=torch.uint8, device=device)
    preprocess(pkg, handle, case, buffer)
    return case, buffer


def test_products_on_two_streams(pkg, handle, device, shared):
    """Products that share the buffer may overlap: each uses its own B."""
    from ops_sparse_b200 import api
    case, buffer = shared
    handles = [api.Handle(torch.cuda.Stream()) for _ in range(3)]
    for _ in range(20):
        for c in case.C:
            c.values.zero_()
        torch.cuda.synchronize()
        for i, h in enumerate(handles):
            for _ in range(3):
                api.spmm(h, case.A, case.B[i], case.C[i], 1.0, 0.0, buffer=buffer)
        torch.cuda.synchronize()
        assert all(case.right(i) for i in range(3))
    for h in handles:
        h.close()


def test_products_of_two_threads(pkg, handle, device, shared):
    """The copy and its product stay together when threads enqueue on one stream."""
    from ops_sparse_b200 import api
    case, buffer = shared
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        h = api.Handle(stream)
        with torch.cuda.stream(stream):
            for _ in range(200):
                api.spmm(h, case.A, case.B[i], case.C[i], 1.0, 0.0, buffer=buffer)
                wrong.append(not case.right(i))
        h.close()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(wrong) == 600 and not any(wrong)


def test_graph_beside_a_product(pkg, handle, device, shared):
    """A recorded product may be launched beside others that share the buffer."""
    from ops_sparse_b200 import api
    case, buffer = shared
    record, beside = torch.cuda.Stream(), torch.cuda.Stream()
    h = api.Handle(record)
    api.spmm(h, case.A, case.B[3], case.C[3], 1.0, 0.0, buffer=buffer)  # what is created at first use must exist
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=record):
        api.spmm(h, case.A, case.B[3], case.C[3], 1.0, 0.0, buffer=buffer)
    for _ in range(20):
        for c in case.C:
            c.values.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(beside):
            graph.replay()
        for i in range(3):
            api.spmm(h, case.A, case.B[i], case.C[i], 1.0, 0.0, buffer=buffer)
        torch.cuda.synchronize()
        assert all(case.right(i) for i in range(4))
    del graph
    h.close()
