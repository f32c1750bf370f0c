"""GPU: int8 SpMM on the tensor cores, at the edges of its tiles, clusters and launches, and on rows it may not write out."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def pattern(rng, m, k, entries):
    """Ascending columns; rows of about `entries` among empty and full ones."""
    lengths = np.where(rng.random(m) < 0.05, rng.choice([0, 1, k], m), np.minimum(entries + rng.integers(-5, 6, m), k))
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.permutation(k)[:n]) for n in lengths]).astype(np.int32)
    return rp, ci, rng.integers(-128, 128, ci.size).astype(np.int8)


class Product:
    def __init__(self, pkg, handle, device, rng, m, k, n, entries, order, align=0, ascending=True, pad=0):
        from ops_sparse_b200 import api
        self.handle, self.shape, self.order = handle, (m, k, n), order
        self.rp, self.ci, self.val = pattern(rng, m, k, entries)
        self.B = rng.integers(-128, 128, (k, n)).astype(np.int8)
        self.C = rng.integers(-1000, 1000, (m, n)).astype(np.int32)
        if not ascending:  # one row of many
            r = m // 2
            self.ci[self.rp[r]:self.rp[r + 1]] = self.ci[self.rp[r]:self.rp[r + 1]][::-1]
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(device)
        stored = (lambda a: a) if order == "row" else (lambda a: a.T)
        self.A = api.CsrMatrix(dev(self.rp), dev(self.ci), dev(self.val), m, k)
        padded = np.pad(stored(self.B), ((0, 0), (0, pad)), constant_values=99)  # rows (columns) of B further apart
        self.dB = api.DnMat(dev(padded), k, n, (n if order == "row" else k) + pad, order)
        self.dC = api.DnMat(dev(stored(self.C)), m, n, n if order == "row" else m, order)
        size = api.spmm_buffer_size(handle, self.A, self.dB, self.dC)
        assert size >= m * k  # room for A as it is written out
        self.buffer = torch.empty(size + 256, dtype=torch.uint8, device=device)[align:]
        pkg.check(pkg.lib().aclsparseSpMMPreprocess(handle.raw, 0, 0, None, self.A.raw, self.dB.raw, None, self.dC.raw, pkg.ACL_INT32, 0,
                                                    ctypes.c_void_p(self.buffer.data_ptr())), "aclsparseSpMMPreprocess")

    def run(self, alpha, beta, handle=None):
        from ops_sparse_b200 import api
        api.spmm(handle or self.handle, self.A, self.dB, self.dC, alpha, beta, buffer=self.buffer)
        torch.cuda.synchronize()
        m, k, n = self.shape
        got = self.dC.values.cpu().numpy()
        return got.reshape(m, n) if self.order == "row" else got.reshape(n, m).T

    def want(self, alpha, beta, ci=None):
        import scipy.sparse
        m, k, n = self.shape
        A = scipy.sparse.csr_matrix((self.val.astype(np.int64), self.ci if ci is None else ci, self.rp), shape=(m, k))
        exact = alpha * (A @ self.B.astype(np.int64)) + beta * self.C.astype(np.int64)
        return np.clip(exact, -2 ** 31, 2 ** 31 - 1).astype(np.int32)


# columns of A on either side of a step and the most a row may have; one to eight column tiles of 32, 64 and 128, several launches;
# last rows and columns of a tile
@pytest.mark.parametrize("m,k,n,entries,order", [
    (4100, 128, 130, 60, "row"), (4097, 129, 132, 60, "col"), (1000, 257, 300, 120, "col"), (220, 12288, 112, 1200, "col"),
    (2000, 512, 256, 256, "row"), (5000, 700, 64, 350, "row"), (20000, 320, 32, 180, "row"), (1700, 400, 1100, 100, "col"),
    (1500, 200, 1030, 100, "row"), (1280, 1000, 512, 200, "row"), (2049, 900, 24, 700, "col"), (257, 3000, 136, 1000, "col"),
])
@pytest.mark.parametrize("alpha,beta", [(1, 0), (70000, -3)])
def test_edges(pkg, handle, device, m, k, n, entries, order, alpha, beta):
    p = Product(pkg, handle, device, np.random.default_rng(m + k + n), m, k, n, entries, order)
    assert np.array_equal(p.run(alpha, beta), p.want(alpha, beta))


def test_rows_that_ascend_no_longer(pkg, handle, device):
    """Columns written over in place after the analysis: repeated and unordered ones are summed entry by entry."""
    p = Product(pkg, handle, device, np.random.default_rng(5), 1500, 600, 150, 270, "col")
    ci = p.ci.copy()
    for i, r in enumerate((0, 3, 127, 128, 700, 1499)):
        row = ci[p.rp[r]:p.rp[r + 1]]
        if i % 2 and row.size > 257:
            row[255] = row[256]  # across two requests
        else:
            row[:] = row[::-1]
    p.A.col_ind.copy_(torch.from_numpy(ci))
    assert np.array_equal(p.run(2, -1), p.want(2, -1, ci))


@pytest.mark.parametrize("m,k,n,entries,order", [(9001, 100, 64, 60, "col"), (9001, 127, 40, 80, "col"), (9401, 64, 256, 50, "row")])
def test_fewer_columns_than_a_step(pkg, handle, device, m, k, n, entries, order):
    p = Product(pkg, handle, device, np.random.default_rng(k), m, k, n, entries, order)
    assert np.array_equal(p.run(2, -1), p.want(2, -1))


@pytest.mark.parametrize("m,k,n,entries,order,pad", [(2000, 512, 256, 256, "row", 16), (2000, 512, 256, 256, "row", 5), (1500, 600, 150, 270, "col", 3)])
def test_wider_leading_dimension(pkg, handle, device, m, k, n, entries, order, pad):
    p = Product(pkg, handle, device, np.random.default_rng(pad), m, k, n, entries, order, pad=pad)
    assert np.array_equal(p.run(2, -1), p.want(2, -1))


def test_rows_that_never_ascended(pkg, handle, device):
    """The analysis finds a row that descends: lane groups."""
    p = Product(pkg, handle, device, np.random.default_rng(12), 1500, 600, 150, 270, "col", ascending=False)
    assert np.array_equal(p.run(2, -1), p.want(2, -1))


def test_replaced_column_array(pkg, handle, device):
    """Other arrays drop the plan, which is analysed again in the product or, for the products after it, by a Preprocess."""
    p = Product(pkg, handle, device, np.random.default_rng(13), 1500, 600, 150, 270, "col")
    columns = p.A.col_ind.clone()
    p.A.col_ind.zero_()
    L = pkg.lib()
    pointer = lambda t: ctypes.c_void_p(t.data_ptr())
    pkg.check(L.aclsparseCsrSetPointers(p.A.raw, pointer(p.A.row_ptr), pointer(columns), pointer(p.A.values)), "aclsparseCsrSetPointers")
    assert np.array_equal(p.run(1, 0), p.want(1, 0))
    pkg.check(L.aclsparseSpMMPreprocess(p.handle.raw, 0, 0, None, p.A.raw, p.dB.raw, None, p.dC.raw, pkg.ACL_INT32, 0, pointer(p.buffer)),
              "aclsparseSpMMPreprocess")
    assert np.array_equal(p.run(3, 0), p.want(3, 0))


def test_in_a_graph(pkg, handle, device):
    """A captured product leaves the shared buffer alone and gives the same, also with other values and beside later ones."""
    from ops_sparse_b200 import api
    p = Product(pkg, handle, device, np.random.default_rng(14), 1500, 600, 150, 270, "col")
    assert np.array_equal(p.run(1, 0), p.want(1, 0))
    record = torch.cuda.Stream()
    recorder = api.Handle(record)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=record):
        api.spmm(recorder, p.A, p.dB, p.dC, 3, 0, buffer=p.buffer)
    p.val = np.roll(p.val, 1)
    p.A.values.copy_(torch.from_numpy(p.val))
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(p.dC.values.cpu().numpy().reshape(150, 1500).T, p.want(3, 0))
    assert np.array_equal(p.run(5, 0), p.want(5, 0))
    del graph
    recorder.close()


@pytest.mark.parametrize("align", [4, 8])
def test_buffer_on_any_word(pkg, handle, device, align):
    p = Product(pkg, handle, device, np.random.default_rng(6), 1500, 600, 150, 270, "col", align)
    assert np.array_equal(p.run(2, -1), p.want(2, -1))


def test_second_stream(pkg, handle, device):
    """The first product's stream may write A into the shared buffer, a product on another reads it as it lies."""
    from ops_sparse_b200 import api
    p = Product(pkg, handle, device, np.random.default_rng(8), 1500, 600, 150, 270, "col")
    assert np.array_equal(p.run(1, 0), p.want(1, 0))
    other = api.Handle(torch.cuda.Stream())
    assert np.array_equal(p.run(3, 0, other), p.want(3, 0))
    other.close()


@pytest.mark.parametrize("order,n", [("col", 150), ("row", 256), ("row", 150)])  # rows of 16-byte pieces: from 96 M products on
def test_wait_that_runs_out(pkg, handle, device, order, n):
    """A few bytes more expected than are copied, two milliseconds to wait for them: C is whole all the same, entry by entry."""
    L = pkg.lib()
    L.b200sp_spmm_stream_wait_test.argtypes = [ctypes.c_longlong, ctypes.c_uint]
    L.b200sp_spmm_stream_wait_test.restype = None
    p = Product(pkg, handle, device, np.random.default_rng(9), 1500, 600, n, 270, order)
    start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    try:
        L.b200sp_spmm_stream_wait_test(1 << 22, 16)
        start.record()
        got = p.run(3, -2)
        end.record()
        end.synchronize()
    finally:
        L.b200sp_spmm_stream_wait_test(0, 0)
    assert start.elapsed_time(end) > 1.0  # it did wait
    assert np.array_equal(got, p.want(3, -2))
    assert L.b200sp_spmm_stream_error() == 0
    p.dC.values.copy_(torch.from_numpy(np.ascontiguousarray(p.C if order == "row" else p.C.T)))
    assert np.array_equal(p.run(3, -2), p.want(3, -2))
