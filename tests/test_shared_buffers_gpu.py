"""GPU: one buffer that several operations are given, one after the other: none trusts what another has written over."""
from __future__ import annotations

from ctypes import addressof, byref, c_float, c_size_t, c_void_p

import numpy as np
import pytest
import torch

from test_sddmm_order_gpu import Case

pytestmark = pytest.mark.gpu


def at(t):
    return c_void_p(t.data_ptr())


class Writer:
    """A library call that writes its buffer: `bytes` it wants, `write(buf)`."""

    def __init__(self, pkg, handle, case, kind):
        self.pkg, self.L, self.handle, self.kind = pkg, pkg.lib(), handle, kind
        h, m, n, nnz, size = handle.raw, case.m, case.cols, case.nnz, c_size_t()
        rp, self.ci = case.row_ptr, case.col_ind.clone()
        if kind == "csr2csc":
            self.val = torch.rand(nnz, device=case.device)
            self.out = [torch.empty(nnz, device=case.device), *(torch.empty(s, dtype=torch.int32, device=case.device) for s in (n + 1, nnz))]
            self.args = (h, m, n, nnz, at(self.val), at(rp), at(self.ci), *map(at, self.out), pkg.ACL_FLOAT, 1, 0, 0)
            pkg.check(self.L.aclsparseCsr2cscEx2_bufferSize(*self.args, byref(size)), "size")
        elif kind == "csrsort":
            self.descr, self.P = c_void_p(), torch.arange(nnz, dtype=torch.int32, device=case.device)
            pkg.check(self.L.aclsparseCreateMatDescr(byref(self.descr)), "descr")
            self.args = (h, m, n, nnz, self.descr, at(rp), at(self.ci), at(self.P))
            pkg.check(self.L.aclsparseXcsrsort_bufferSizeExt(h, m, n, nnz, at(rp), at(self.ci), byref(size)), "size")
        else:
            from ops_sparse_b200 import api
            self.A = api.CsrMatrix(rp, self.ci, torch.rand(nnz, device=case.device), m, n)
            self.x, self.y = (api.DnVec(torch.rand(s, device=case.device)) for s in (n, m))
            self.args = (0, self.A.raw, self.x.raw, self.y.raw, self.y.raw, pkg.ACL_FLOAT, 2)
            self.descr = c_void_p()
            pkg.check(self.L.aclsparseSpMVOp_bufferSize(h, *self.args, byref(size)), "size")
        self.bytes = size.value

    def write(self, buf):
        if self.kind == "csr2csc":
            status = self.L.aclsparseCsr2cscEx2(*self.args, at(buf))
        elif self.kind == "csrsort":
            status = self.L.aclsparseXcsrsort(*self.args, at(buf))
        else:
            status = self.L.aclsparseSpMVOp_createDescr(self.handle.raw, byref(self.descr), *self.args, at(buf))
        self.pkg.check(status, self.kind)

    def close(self):
        if self.kind == "csrsort":
            self.L.aclsparseDestroyMatDescr(self.descr)
        elif self.kind == "spmvop":
            self.L.aclsparseSpMVOp_destroyDescr(self.descr)


@pytest.mark.parametrize("kind", ["csr2csc", "csrsort", "spmvop"])
def test_sddmm_order_written_over(pkg, handle, device, kind):
    case = Case(pkg, handle, device, "f16", 128)
    writer = Writer(pkg, handle, case, kind)
    plain = case.product(torch.empty(256, dtype=torch.uint8, device=device))
    buf = torch.empty(max(case.buffer().numel(), writer.bytes), dtype=torch.uint8, device=device)
    case.preprocess(buf)
    writer.write(buf)
    assert torch.equal(case.product(buf), plain)
    writer.close()


@pytest.mark.parametrize("kind", ["csr2csc", "csrsort", "spmvop"])
def test_spmv_plan_written_over(pkg, handle, device, kind):
    from ops_sparse_b200 import api
    case = Case(pkg, handle, device, "f32", 4, nnz=300_000, cols=50_000)
    writer = Writer(pkg, handle, case, kind)
    val, x = torch.rand(case.nnz, device=device), torch.rand(case.cols, device=device)
    A, dx, dy = api.CsrMatrix(case.row_ptr, case.col_ind, val, case.m, case.cols), api.DnVec(x), api.DnVec(torch.empty(case.m, device=device))
    size = api.spmv_preprocess(handle, A, dx, dy).numel()
    buf = torch.empty(max(size, writer.bytes), dtype=torch.uint8, device=device)
    null = c_void_p()
    pkg.check(pkg.lib().aclsparseSpMVPreprocess(handle.raw, 0, null, A.raw, dx.raw, null, dy.raw, pkg.ACL_FLOAT, 0, at(buf)), "preprocess")
    writer.write(buf)
    api.spmv(handle, A, dx, dy, 1.0, 0.0, buffer=buf)
    torch.cuda.synchronize()
    want = torch.zeros(case.m, dtype=torch.float64, device=device).index_add(0, case.rows, val.double() * x.double()[case.col_ind.long()])
    count = torch.bincount(case.rows, minlength=case.m)
    # all terms are positive: (additions + 3) half ulps of the sum
    assert bool(((dy.values.double() - want).abs() <= (count + 3) * 2.0 ** -24 * want).all())
    writer.close()


@pytest.mark.parametrize("kind", ["csr2csc", "csrsort", "spmvop", "spmv"])
def test_row_order_of_spmvop_written_over(pkg, handle, device, kind):
    from ops_sparse_b200 import api
    case = Case(pkg, handle, device, "f32", 4, nnz=300_000, cols=50_000)
    A = api.CsrMatrix(case.row_ptr, case.col_ind, torch.rand(case.nnz, device=device), case.m, case.cols)
    x, y, z = (api.DnVec(torch.rand(s, device=device)) for s in (case.cols, case.m, case.m))
    fewer = Case(pkg, handle, device, "f32", 4, seed=5, nnz=200_000, cols=50_000)
    other = Writer(pkg, handle, fewer, "csrsort" if kind == "spmv" else kind)
    args, null, size, descr, plan = (0, A.raw, x.raw, y.raw, z.raw, pkg.ACL_FLOAT, 2), c_void_p(), c_size_t(), c_void_p(), c_void_p()
    pkg.check(pkg.lib().aclsparseSpMVOp_bufferSize(handle.raw, *args, byref(size)), "size")
    buf = torch.empty(max(size.value, other.bytes, api.spmv_buffer_size(handle, A, x, y)), dtype=torch.uint8, device=device)
    pkg.check(pkg.lib().aclsparseSpMVOp_createDescr(handle.raw, byref(descr), *args, at(buf)), "descr")
    pkg.check(pkg.lib().aclsparseSpMVOp_createPlan(handle.raw, descr, byref(plan), None, 0), "plan")
    if kind == "spmv":
        pkg.check(pkg.lib().aclsparseSpMVPreprocess(handle.raw, 0, null, A.raw, x.raw, null, y.raw, pkg.ACL_FLOAT, 0, at(buf)), "preprocess")
    else:
        other.write(buf)
    a, b = c_float(1.0), c_float(0.0)
    pkg.check(pkg.lib().aclsparseSpMVOp(handle.raw, plan, c_void_p(addressof(a)), c_void_p(addressof(b)), x.raw, y.raw, z.raw), "product")
    torch.cuda.synchronize()
    terms = A.values.double() * x.values.double()[case.col_ind.long()]
    want = torch.zeros(case.m, dtype=torch.float64, device=device).index_add(0, case.rows, terms)
    # compensated sums of positive terms
    assert bool(((z.values.double() - want).abs() <= 8 * 2.0 ** -24 * want).all())
    pkg.lib().aclsparseSpMVOp_destroyPlan(plan)
    pkg.lib().aclsparseSpMVOp_destroyDescr(descr)
    other.close()


def foreign(kind, buf, kept, gen):
    """Bytes that no call of the library wrote."""
    n, words = buf.numel(), buf[: buf.numel() // 8 * 8].view(torch.int32)
    if kind == "zeros":
        buf.zero_()
    elif kind == "ones":
        buf.fill_(255)
    elif kind == "noise":
        buf.random_(0, 256, generator=gen)
    elif kind == "small numbers":  # many are tiles
        words.random_(0, 20000, generator=gen)
    elif kind == "shifted":  # every entry is one, but of another place
        buf.copy_(kept.roll(8))
    elif kind == "half":  # what was there, up to the middle; the end of the order is another one's
        buf[n // 2:].random_(0, 256, generator=gen)
    elif kind == "swapped":  # two entries of the order in each other's place
        words[-200:] = words[-200:].flip(0)
    else:  # single words
        at = torch.randint(words.numel(), (50,), generator=gen, device=buf.device)
        words[at] = words[at] + 1


@pytest.mark.parametrize("kind", ["zeros", "ones", "noise", "small numbers", "shifted", "half", "swapped", "words"])
@pytest.mark.parametrize("cols", [0, 5000])  # with near tiles, and the rows of the tiles alone
def test_sddmm_order_written_over_by_others(pkg, handle, device, cols, kind):
    """Straight into the memory, and into that of a product that a graph repeats: with beta, so that a tile done twice shows."""
    case = Case(pkg, handle, device, "f16", 128, cols=cols)
    plain = case.product(torch.empty(256, dtype=torch.uint8, device=device))
    buf = case.buffer()
    case.preprocess(buf)
    assert torch.equal(case.product(buf), plain)
    kept, gen = buf.clone(), torch.Generator(device=device).manual_seed(3)
    for _ in range(2):
        foreign(kind, buf, kept, gen)
        kept = buf.clone()
        assert torch.equal(case.product(buf), plain)
        assert torch.equal(buf, kept)  # the product only reads it
    case.preprocess(buf)
    kept = buf.clone()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream(device)
    with torch.cuda.graph(graph, stream=stream):
        assert pkg.lib().aclsparseSetStream(handle.raw, c_void_p(stream.cuda_stream)) == 0
        try:
            pkg.check(pkg.lib().aclsparseSDDMM(*case.args, at(buf)), "product")
        finally:
            assert pkg.lib().aclsparseSetStream(handle.raw, c_void_p(handle.stream.cuda_stream)) == 0
    foreign(kind, buf, kept, gen)
    for _ in range(2):  # the second time on the order again
        case.C.values.copy_(case.c0)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(case.C.values, plain)
        buf.copy_(kept)


@pytest.mark.parametrize("dtype", ["f32", "f16"])  # a y of 16 bits accumulates in the buffer
def test_sddmm_leaves_the_buffer_of_a_transposed_product_alone(pkg, handle, device, dtype):
    """What was preprocessed for the transposed product, and may be 256 bytes, stays refused for the plain one."""
    from ops_sparse_b200 import api
    case = Case(pkg, handle, device, "f16", 128, nnz=300_000, cols=5000)
    tdt = torch.float16 if dtype == "f16" else torch.float32
    A = api.CsrMatrix(case.row_ptr, case.col_ind, torch.rand(case.nnz, device=device).to(tdt), case.m, case.cols)
    x, y = (api.DnVec(torch.rand(s, device=device).to(tdt)) for s in (case.m, case.cols))
    buf, L, null, T = case.buffer(), pkg.lib(), c_void_p(), pkg.ACL_SPARSE_OP_TRANSPOSE
    assert buf.numel() >= 4 * case.cols
    pkg.check(L.aclsparseSpMVPreprocess(handle.raw, T, null, A.raw, x.raw, null, y.raw, pkg.ACL_FLOAT, 0, at(buf)), "plan")
    a, b = c_float(1.0), c_float(0.0)
    scalars = c_void_p(addressof(a)), c_void_p(addressof(b))
    for _ in range(2):  # the second time after a product
        torch.cuda.synchronize()
        kept = buf.clone()
        case.preprocess(buf)
        torch.cuda.synchronize()
        assert torch.equal(buf, kept)
        status = L.aclsparseSpMV(handle.raw, 0, scalars[0], A.raw, y.raw, scalars[1], x.raw, pkg.ACL_FLOAT, 0, at(buf))
        assert status == pkg.ACL_SPARSE_STATUS_INVALID_VALUE
        pkg.check(L.aclsparseSpMV(handle.raw, T, scalars[0], A.raw, x.raw, scalars[1], y.raw, pkg.ACL_FLOAT, 0, at(buf)), "product")


@pytest.mark.parametrize("kind", ["spmv", "spmm", "spmvop"])
def test_sddmm_leaves_the_plans_of_others_alone(pkg, handle, device, kind):
    from ops_sparse_b200 import api
    case = Case(pkg, handle, device, "f16", 128, nnz=300_000, cols=5000)
    plain = case.product(torch.empty(256, dtype=torch.uint8, device=device))
    A = api.CsrMatrix(case.row_ptr, case.col_ind, torch.rand(case.nnz, device=device), case.m, case.cols)
    null, descr, size = c_void_p(), c_void_p(), c_size_t()
    x, y = (api.DnVec(torch.rand(s, device=device)) for s in (case.cols, case.m))
    B, out = (api.DnMat.row_major(torch.rand((s, 16), device=device)) for s in (case.cols, case.m))
    need = {"spmv": lambda: api.spmv_preprocess(handle, A, x, y).numel(), "spmm": lambda: api.spmm_preprocess(handle, A, B, out).numel(),
            "spmvop": lambda: 4 * case.m + 4096}[kind]()
    buf = torch.full((max(case.buffer().numel(), need),), 255, dtype=torch.uint8, device=device)
    L = pkg.lib()
    if kind == "spmv":
        pkg.check(L.aclsparseSpMVPreprocess(handle.raw, 0, null, A.raw, x.raw, null, y.raw, pkg.ACL_FLOAT, 0, at(buf)), "plan")
    elif kind == "spmm":
        pkg.check(L.aclsparseSpMMPreprocess(handle.raw, 0, 0, null, A.raw, B.raw, null, out.raw, pkg.ACL_FLOAT, 0, at(buf)), "plan")
    else:
        args = (0, A.raw, x.raw, y.raw, y.raw, pkg.ACL_FLOAT, 2)
        pkg.check(L.aclsparseSpMVOp_bufferSize(handle.raw, *args, byref(size)), "size")
        assert size.value <= need
        pkg.check(L.aclsparseSpMVOp_createDescr(handle.raw, byref(descr), *args, at(buf)), "plan")
    kept = buf.clone()
    case.preprocess(buf)
    assert torch.equal(buf, kept)
    assert torch.equal(case.product(buf), plain)
    if kind == "spmm":  # a product with a plan waits for nothing, so a graph may hold it
        graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream(device)
        with torch.cuda.graph(graph, stream=stream):
            assert L.aclsparseSetStream(handle.raw, c_void_p(stream.cuda_stream)) == 0
            try:
                api.spmm(handle, A, B, out, 1.0, 0.0, buffer=buf)
            finally:
                assert L.aclsparseSetStream(handle.raw, c_void_p(handle.stream.cuda_stream)) == 0
    A.close()  # nobody needs the plan any more
    if kind == "spmvop":
        L.aclsparseSpMVOp_destroyDescr(descr)
    case.preprocess(buf)
    torch.cuda.synchronize()
    assert not torch.equal(buf, kept)
    assert torch.equal(case.product(buf), plain)
