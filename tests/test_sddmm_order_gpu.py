"""GPU: SDDMM on a Y that L2 does not hold, where Preprocess leaves an order of the tiles in the buffer: the same bits as without
one, whatever became of the pattern and the buffer since."""
from __future__ import annotations

from ctypes import addressof, byref, c_float, c_size_t, c_uint16, c_void_p

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


class Case:
    """Rows of 16 to 30,000 entries among short ones; a last tile that is not full."""

    def __init__(self, pkg, handle, device, dtype, k, seed=0, nnz=(1 << 20) + 77, cols=0):
        from ops_sparse_b200 import api
        self.pkg, self.handle, self.device = pkg, handle, device
        half = dtype == "f16"
        self.cols, tdt = cols or (100 << 20) // (k * (2 if half else 4)) + 3, torch.float16 if half else torch.float32
        rng = np.random.default_rng(seed)
        lengths = np.concatenate([[30000, 16, 1, 0, 2000, 64, 63, 65], rng.integers(100, 3000, 300), rng.integers(0, 9, 40000)])
        lengths = rng.permutation(lengths[np.cumsum(lengths) < nnz])
        lengths[-1] += nnz - lengths.sum()
        self.m, self.nnz, self.k = lengths.size, nnz, k
        self.row_ptr = torch.from_numpy(np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)).to(device)
        gen = torch.Generator(device=device).manual_seed(seed + 1)
        key = torch.repeat_interleave(torch.arange(self.m, device=device), torch.from_numpy(lengths).to(device)) * self.cols
        self.col_ind = (torch.sort(key + torch.randint(self.cols, (nnz,), generator=gen, device=device)).values - key).to(torch.int32)
        self.rows = key // self.cols
        self.X = torch.randn((self.m, k), generator=gen, device=device).to(tdt)
        self.Y = torch.randn((self.cols, k), generator=gen, device=device).to(tdt)
        self.c0 = torch.randn(nnz, generator=gen, device=device).to(tdt)
        self.C = api.CsrMatrix(self.row_ptr, self.col_ind, self.c0.clone(), self.m, self.cols)
        self.dX, self.dY = api.DnMat.row_major(self.X), api.DnMat.row_major(self.Y)
        word = (lambda v: c_uint16(int(np.float16(v).view(np.uint16)))) if half else c_float
        self.keep = word(0.75), word(-0.5)
        a, b = (c_void_p(addressof(w)) for w in self.keep)
        self.args = (handle.raw, pkg.ACL_SPARSE_OP_NON_TRANSPOSE, pkg.ACL_SPARSE_OP_TRANSPOSE, a, self.dX.raw, self.dY.raw, b,
                     self.C.raw, pkg.ACL_FLOAT16 if half else pkg.ACL_FLOAT, 0)

    def buffer(self):
        size = c_size_t()
        self.pkg.check(self.pkg.lib().aclsparseSDDMMBufferSize(*self.args, byref(size)), "size")
        return torch.full((size.value,), 255, dtype=torch.uint8, device=self.device)

    def preprocess(self, buf):
        self.pkg.check(self.pkg.lib().aclsparseSDDMMPreprocess(*self.args, c_void_p(buf.data_ptr())), "preprocess")

    def product(self, buf):
        self.C.values.copy_(self.c0)
        self.pkg.check(self.pkg.lib().aclsparseSDDMM(*self.args, c_void_p(buf.data_ptr())), "product")
        torch.cuda.synchronize()
        return self.C.values.clone()

    def check(self, got):
        """|error| <= (k + 3) eps32 sum |x y| and the rounding of the result, against 64 bits."""
        rel = 2.0 ** -11 if got.dtype == torch.float16 else 2.0 ** -24
        for s in range(0, self.nnz, 1 << 18):
            p = slice(s, s + (1 << 18))
            x, y = self.X[self.rows[p]].double(), self.Y[self.col_ind[p].long()].double()
            want = 0.75 * (x * y).sum(1) - 0.5 * self.c0[p].double()
            scale = 0.75 * (x * y).abs().sum(1) + 0.5 * self.c0[p].double().abs()
            err = (got[p].double() - want).abs()
            assert bool((err <= (self.k + 3) * 2.0 ** -24 * scale + rel * want.abs() + 1e-7).all())


# one and several turns over k, pieces of 16 bytes; one and two warps a CTA; and 8-byte pieces, which have no ordered form
@pytest.mark.parametrize("dtype,k", [("f16", 256), ("f16", 64), ("f16", 520), ("f32", 128), ("f32", 600), ("f16", 100)])
def test_order(pkg, handle, device, dtype, k):
    case = Case(pkg, handle, device, dtype, k)
    plain = case.product(torch.empty(256, dtype=torch.uint8, device=device))  # never preprocessed: no order
    case.check(plain)
    buf = case.buffer()
    assert (buf.numel() > 256) == (k != 100)
    assert torch.equal(case.product(buf), plain)    # of the right size, but not preprocessed
    case.preprocess(buf)
    assert torch.equal(case.product(buf), plain)
    other = torch.empty(256, dtype=torch.uint8, device=device)
    assert torch.equal(case.product(other), plain)  # another buffer than the one with the order


# a Y that L2 holds, one that comes through L1, and a matrix too small for an order
@pytest.mark.parametrize("cols,nnz", [(5000, (1 << 18) + 1), (60, 1 << 18), (5000, (1 << 18) - 1), (5000, 1_000_003)])
@pytest.mark.parametrize("dtype,k", [("f16", 64), ("f32", 256), ("f16", 384)])
def test_rows_of_tiles(pkg, handle, device, dtype, k, cols, nnz):
    case = Case(pkg, handle, device, dtype, k, nnz=nnz, cols=cols)
    plain = case.product(torch.empty(256, dtype=torch.uint8, device=device))
    case.check(plain)
    buf = case.buffer()
    assert (buf.numel() > 256) == (nnz >= 1 << 18)
    case.preprocess(buf)
    assert torch.equal(case.product(buf), plain)


def test_pattern_and_buffer_that_change(pkg, handle, device):
    case = Case(pkg, handle, device, "f16", 128)
    buf = case.buffer()
    case.preprocess(buf)
    want = case.product(buf)
    # the same descriptor, another pattern of as many entries, written in place: the rows the order names are wrong now
    later = Case(pkg, handle, device, "f16", 128, seed=7)
    assert later.m == case.m
    plain = later.product(torch.empty(256, dtype=torch.uint8, device=device))
    kept = case.row_ptr.clone(), case.col_ind.clone(), case.X.clone(), case.Y.clone(), case.c0.clone()
    for mine, its in ((case.row_ptr, later.row_ptr), (case.col_ind, later.col_ind), (case.X, later.X), (case.Y, later.Y),
                      (case.c0, later.c0)):
        mine.copy_(its)
    assert torch.equal(case.product(buf), plain)
    for mine, its in zip((case.row_ptr, case.col_ind, case.X, case.Y, case.c0), kept):
        mine.copy_(its)
    # another matrix is preprocessed into the buffer: this one's order is gone
    fewer = Case(pkg, handle, device, "f16", 128, seed=9, nnz=(1 << 20) + 5)
    fewer.buffer()
    fewer.preprocess(buf)
    assert torch.equal(case.product(buf), want)
    # in a graph, from a side stream
    case.preprocess(buf)
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream(device)
    with torch.cuda.graph(graph, stream=stream):
        assert pkg.lib().aclsparseSetStream(handle.raw, c_void_p(stream.cuda_stream)) == 0
        try:
            case.pkg.check(pkg.lib().aclsparseSDDMM(*case.args, c_void_p(buf.data_ptr())), "product")
        finally:
            assert pkg.lib().aclsparseSetStream(handle.raw, c_void_p(handle.stream.cuda_stream)) == 0
    case.C.values.copy_(case.c0)
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(case.C.values, want)


# rows of 32 pieces and of 33; Y above 96 MB with too few entries for near tiles, by the width of the rows
@pytest.mark.parametrize("dtype,k,cols,nnz,written", [("f16", 256, 5000, 1 << 18, True), ("f16", 264, 5000, 1 << 18, False), ("f32", 1024, 5000, 300_000, False),
                                                      ("f32", 136, 0, (1 << 19) - 1, False), ("f32", 136, 0, 1 << 19, True), ("f16", 64, 0, 1 << 19, True)])
def test_where_an_order_pays(pkg, handle, device, dtype, k, cols, nnz, written):
    case = Case(pkg, handle, device, dtype, k, nnz=nnz, cols=cols)
    plain = case.product(torch.empty(256, dtype=torch.uint8, device=device))
    buf = case.buffer()
    untouched = buf.clone()
    case.preprocess(buf)
    torch.cuda.synchronize()
    assert (not torch.equal(buf, untouched)) == written
    assert torch.equal(case.product(buf), plain)


@pytest.mark.parametrize("cols,launches", [(5000, 1), (0, 3)])  # the rows of the tiles; an order of them
def test_launches_of_preprocess(pkg, handle, device, cols, launches):
    """Where no tile can be near, one kernel, which does not wait and does not read the columns: those may not be there yet."""
    case = Case(pkg, handle, device, "f16", 128, cols=cols)
    plain = case.product(torch.empty(256, dtype=torch.uint8, device=device))
    buf = case.buffer()
    before = pkg.lib().b200sp_kernel_launches()
    case.preprocess(buf)
    assert pkg.lib().b200sp_kernel_launches() - before == launches
    assert torch.equal(case.product(buf), plain)


@pytest.mark.parametrize("cols", [0, 5000])
@pytest.mark.parametrize("shift", [1, 2, 4, 8, 16])
def test_buffer_at_any_address(pkg, handle, device, shift, cols):
    case = Case(pkg, handle, device, "f16", 128, cols=cols)
    plain = case.product(torch.empty(256, dtype=torch.uint8, device=device))
    whole = torch.full((case.buffer().numel() + 16,), 255, dtype=torch.uint8, device=device)
    buf = whole[shift:shift + whole.numel() - 16]
    case.preprocess(buf)
    torch.cuda.synchronize()
    assert bool((buf == 255).all()) == (shift % 8 != 0)  # no order where its entries would not be aligned
    assert torch.equal(case.product(buf), plain)


@pytest.mark.parametrize("cols", [0, 5000])
@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_preprocess_while_another_stream_is_captured(pkg, handle, device, mode, cols):
    """Nothing of it goes into the graph and the capture goes on, as when Preprocess launched nothing."""
    case = Case(pkg, handle, device, "f16", 128, cols=cols)
    plain = case.product(torch.empty(256, dtype=torch.uint8, device=device))
    buf, data = case.buffer(), torch.ones(1000, device=device)
    graph, stream, mine = torch.cuda.CUDAGraph(), torch.cuda.Stream(device), torch.cuda.Stream(device)
    torch.cuda.synchronize()
    assert pkg.lib().aclsparseSetStream(handle.raw, c_void_p(mine.cuda_stream)) == 0
    try:
        with torch.cuda.graph(graph, stream=stream, capture_error_mode=mode):
            data.add_(1)
            case.preprocess(buf)
            data.add_(1)
    finally:
        assert pkg.lib().aclsparseSetStream(handle.raw, c_void_p(handle.stream.cuda_stream)) == 0
    graph.replay()
    torch.cuda.synchronize()
    assert bool((data == 3).all())
    assert torch.equal(case.product(buf), plain)


def test_threads(pkg, handle, device):
    """One thread preprocesses the matrix again and again, into two buffers in turn; others run products of it on the same stream."""
    import threading
    case = Case(pkg, handle, device, "f16", 128, nnz=1 << 20)
    plain = case.product(torch.empty(256, dtype=torch.uint8, device=device))
    buf, other, failed, done = case.buffer(), case.buffer(), [], threading.Event()

    def products():
        torch.cuda.set_device(device)
        while not done.is_set():
            for b in (buf, other):
                if pkg.lib().aclsparseSDDMM(*case.args, c_void_p(b.data_ptr())):
                    failed.append(1)

    case.keep[1].value = 0  # beta: every product writes the same
    zero = case.product(torch.empty(256, dtype=torch.uint8, device=device))
    threads = [threading.Thread(target=products) for _ in range(2)]
    for t in threads:
        t.start()
    for i in range(60):
        case.preprocess((buf, other)[i % 2])
        size = c_size_t()
        pkg.check(pkg.lib().aclsparseSDDMMBufferSize(*case.args, byref(size)), "size")
    done.set()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed
    assert torch.equal(case.C.values, zero)
    assert not torch.equal(zero, plain)


@pytest.mark.parametrize("cols", [0, 5000])
@pytest.mark.parametrize("dtype", ["f16", "f32"])
@pytest.mark.parametrize("x,y", [("row", "row"), ("turned", "row"), ("row", "turned"), ("turned", "turned"), ("other", "row")])
def test_layouts_leading_dimensions_and_device_scalars(pkg, handle, device, dtype, x, y, cols):
    """The operands as stored rows, as columns of a turned matrix (the same memory), and an X whose rows do not lie together."""
    from ops_sparse_b200 import api
    case = Case(pkg, handle, device, dtype, 128, cols=cols)
    k, tdt, keep, scalars = case.k, case.X.dtype, [], []

    def operand(a, how, pad):
        rows = a.shape[0]
        store = torch.full((rows, k + pad), float("nan"), dtype=tdt, device=device)
        store[:, :k] = a
        if how == "other":
            store = a.t().contiguous()
            mat = api.DnMat(store, rows, k, rows, "col")
        else:
            mat = api.DnMat(store, rows, k, k + pad, "row") if how == "row" else api.DnMat(store, k, rows, k + pad, "col")
        keep.append((store, mat))
        return mat
    X, Y = operand(case.X, x, 8), operand(case.Y, y, 16)
    opx = pkg.ACL_SPARSE_OP_TRANSPOSE if x == "turned" else pkg.ACL_SPARSE_OP_NON_TRANSPOSE
    opy = pkg.ACL_SPARSE_OP_NON_TRANSPOSE if y == "turned" else pkg.ACL_SPARSE_OP_TRANSPOSE
    plain_args = case.args
    case.args = (handle.raw, opx, opy, plain_args[3], X.raw, Y.raw, *plain_args[6:])
    plain = case.product(torch.empty(256, dtype=torch.uint8, device=device))
    case.check(plain)
    buf = case.buffer()
    case.preprocess(buf)
    assert torch.equal(case.product(buf), plain)
    scalars = [torch.tensor([v], dtype=tdt, device=device) for v in (0.75, -0.5)]
    case.args = (*case.args[:3], c_void_p(scalars[0].data_ptr()), *case.args[4:6], c_void_p(scalars[1].data_ptr()), *case.args[7:])
    handle.set_pointer_mode_device(True)
    try:
        assert torch.equal(case.product(buf), plain)
    finally:
        handle.set_pointer_mode_device(False)
