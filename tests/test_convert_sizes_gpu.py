"""GPU: csrsort and csr2csc where their kernels change hands, bit for bit against the golden restatement."""
from __future__ import annotations

from ctypes import byref, c_size_t, c_void_p

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def P(t):
    return c_void_p(t.data_ptr())


@pytest.mark.parametrize("columns", ["even", "clusters", "one value"])
def test_csrsort_row_kernels(pkg, handle, device, oracle, columns):
    """Both sides of every row length at which another kernel takes over; columns that fill the buckets of the
    shared-memory sort evenly, and columns that do not (the radix passes behind it)."""
    L = pkg.lib()
    rng = np.random.default_rng(len(columns))
    edges = [32, 256, 2048, 8192, 16384]
    lengths = np.array([0, 1] + [e + d for e in edges for d in (0, 1)] + [700, 5000, 12000, 3, 0])
    m, n, nnz = lengths.size, 1 << 21, int(lengths.sum())
    rp = np.zeros(m + 1, np.int32)
    rp[1:] = np.cumsum(lengths)
    if columns == "even":
        ci = rng.integers(0, n, nnz)
    elif columns == "clusters":  # a few dense stretches far apart, duplicates among them
        ci = rng.choice([0, 5, 70000, 1 << 20, n - 900], nnz) + rng.integers(0, 800, nnz)
    else:
        ci = np.full(nnz, 77)
    ci = ci.astype(np.int32)
    p0 = rng.permutation(nnz).astype(np.int32)
    want_ci, want_p = oracle.csrsort(rp, ci, p0, 0)
    d_rp, d_ci, d_p = (torch.from_numpy(a).to(device) for a in (rp, ci, p0))
    descr, size = c_void_p(), c_size_t()
    assert L.aclsparseCreateMatDescr(byref(descr)) == 0
    assert L.aclsparseXcsrsort_bufferSizeExt(handle.raw, m, n, nnz, P(d_rp), P(d_ci), byref(size)) == 0
    buf = torch.full((size.value,), 0x5A, dtype=torch.uint8, device=device)
    assert L.aclsparseXcsrsort(handle.raw, m, n, nnz, descr, P(d_rp), P(d_ci), P(d_p), P(buf)) == 0
    torch.cuda.synchronize()
    assert np.array_equal(d_ci.cpu().numpy(), want_ci)
    assert np.array_equal(d_p.cpu().numpy(), want_p)
    assert L.aclsparseDestroyMatDescr(descr) == 0


@pytest.mark.parametrize("m,n,nnz", [
    (50, 1, 300), (3000, 1024, 2047), (3000, 1025, 2048), (7, 1 << 20, 2049),   # one pass, two, the edges of a tile
    (3000, (1 << 20) + 1, 5000),                                                # three passes
    (5_000_000, 1 << 20, 20000),                                                # two, rows too many to share a word
    (100_000, 900, 2049), (100_000, (1 << 20) + 1, 5000), (3_000_000, 700, 20000),  # empty rows, a few and many per entry
    (70000, 40000, 1 << 20), (70000, 40000, (1 << 20) + 1), (9, 700, 3_000_000),  # small tiles, large ones, long rows
])
@pytest.mark.parametrize("base", [0, 1])
def test_csr2csc_passes_and_tiles(pkg, handle, device, oracle, m, n, nnz, base):
    L, S = pkg.lib(), pkg
    rng = np.random.default_rng(m + n + nnz)
    rp = np.concatenate([[0], np.sort(rng.integers(0, nnz + 1, m - 1)), [nnz]]).astype(np.int32) + base
    ci = (np.minimum(rng.integers(0, n, nnz), rng.integers(0, n, nnz))).astype(np.int32) + base
    raw = rng.integers(0, 1 << 32, nnz, dtype=np.uint64).astype(np.uint32)
    want_cp, want_ri, want_raw = oracle.csr2csc(m, n, rp, ci, raw, base)
    d_rp, d_ci, d_v = (torch.from_numpy(a).to(device) for a in (rp, ci, raw.view(np.int32)))
    o_v, o_ri = torch.empty_like(d_v), torch.empty_like(d_ci)
    o_cp = torch.full((n + 1,), -3, dtype=torch.int32, device=device)
    size = c_size_t()
    args = (handle.raw, m, n, nnz, P(d_v), P(d_rp), P(d_ci), P(o_v), P(o_cp), P(o_ri), S.ACL_FLOAT, 1, base, 0)
    assert L.aclsparseCsr2cscEx2_bufferSize(*args, byref(size)) == 0
    buf = torch.full((size.value,), 0x5A, dtype=torch.uint8, device=device)
    assert L.aclsparseCsr2cscEx2(*args, P(buf)) == 0
    torch.cuda.synchronize()
    assert np.array_equal(o_cp.cpu().numpy(), want_cp)
    assert np.array_equal(o_ri.cpu().numpy(), want_ri)
    assert np.array_equal(o_v.cpu().numpy().view(np.uint32), want_raw)


def test_csr2csc_few_entries_in_many_rows(pkg, handle, device):
    """Rows without entries are searched, not walked through: 50 M of them around 1000 entries took 88 ms when a CTA went
    through all rows of its tile, and take 0.04 ms."""
    L, S = pkg.lib(), pkg
    m, n, nnz = 50_000_000, 1_000_000, 1000
    rows = torch.arange(nnz, dtype=torch.int64, device=device) * (m // nnz) + 17
    d_rp = torch.searchsorted(rows, torch.arange(m + 1, device=device)).to(torch.int32)
    cols = torch.randperm(n, generator=torch.Generator().manual_seed(5))[:nnz]
    d_ci = cols.to(device=device, dtype=torch.int32)
    d_v = torch.arange(nnz, dtype=torch.float32, device=device)
    o_v, o_ri = torch.empty_like(d_v), torch.empty_like(d_ci)
    o_cp = torch.empty(n + 1, dtype=torch.int32, device=device)
    size = c_size_t()
    args = (handle.raw, m, n, nnz, P(d_v), P(d_rp), P(d_ci), P(o_v), P(o_cp), P(o_ri), S.ACL_FLOAT, 1, 0, 0)
    assert L.aclsparseCsr2cscEx2_bufferSize(*args, byref(size)) == 0
    buf = torch.empty(size.value, dtype=torch.uint8, device=device)
    start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    assert L.aclsparseCsr2cscEx2(*args, P(buf)) == 0
    start.record()
    assert L.aclsparseCsr2cscEx2(*args, P(buf)) == 0
    end.record()
    torch.cuda.synchronize()
    order = torch.argsort(d_ci)
    assert torch.equal(o_ri, rows[order].to(torch.int32)) and torch.equal(o_v, d_v[order])
    assert torch.equal(o_cp[1:] - o_cp[:-1], torch.bincount(d_ci, minlength=n).to(torch.int32))
    assert start.elapsed_time(end) < 20.0  # ms
