"""GPU: aclsparseSpMV without an analysed buffer where its kernels change hands, against the CPU golden."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mean", [2, 12, 40, 100, 300])  # one per width of the lane groups
@pytest.mark.parametrize("vt,ot", [("f32", "f32"), ("bf16", "bf16"), ("i32", "i32")])
@pytest.mark.parametrize("own_buffer", [False, True])
def test_row_lengths_around_every_limit(handle, device, oracle, mean, vt, ot, own_buffer):
    """Rows on both sides of a lane group's, a warp's and a segment's limit; twice, so that what the first product left
    behind is met by the second."""
    from ops_sparse_b200 import api, synth
    rng = np.random.default_rng(mean)
    edges = [16 * g for g in (2, 4, 8, 16, 32)] + [1024, 8192, 16384]
    lengths = np.concatenate([rng.integers(0, 2 * mean + 1, 5000), [e + d for e in edges for d in (0, 1)], [0, 40000]])
    rng.shuffle(lengths)
    m, n = lengths.size, 60000
    whole = vt == "i32"
    A = synth.csr_from_lengths(rng, lengths, n, (lambda r, k: r.integers(-9, 10, k)) if whole else synth.normal)
    x = rng.integers(-9, 10, n).astype(np.int32) if whole else oracle.to_storage(rng.standard_normal(n).astype(np.float32), vt)
    y = rng.integers(-9, 10, m).astype(np.int32) if whole else oracle.to_storage(rng.standard_normal(m).astype(np.float32), ot)
    val = A.values.astype(np.int32) if whole else oracle.to_storage(A.values, vt)
    alpha, beta = (2, -3) if whole else (1.5, -0.5)
    dA = helpers.make_csr(device, A.row_ptr, A.col_ind, val, vt, m, n)
    dx = api.DnVec(helpers.to_device(x, vt, device))
    for _ in range(2):
        dy = api.DnVec(helpers.to_device(y, ot, device))
        buf = torch.full((api.spmv_buffer_size(handle, dA, dx, dy),), 0x5A, dtype=torch.uint8, device=device) if own_buffer else None
        api.spmv(handle, dA, dx, dy, alpha, beta, buffer=buf)
        torch.cuda.synchronize()
        got = helpers.to_host(dy.values, ot)
        if whole:
            prod = val.astype(np.int64) * x[A.col_ind].astype(np.int64)
            total = np.concatenate([[0], np.cumsum(prod)])
            want = alpha * (total[A.row_ptr[1:]] - total[A.row_ptr[:-1]]) + beta * y.astype(np.int64)
            assert np.array_equal(got, want.astype(np.int32))
            continue
        f = lambda a, t: oracle.from_storage(a, t).astype(np.float64)
        prod = f(val, vt) * f(x, vt)[A.col_ind]
        add = lambda p: np.diff(np.concatenate([[0.0], np.cumsum(p)])[A.row_ptr])
        want, scale = alpha * add(prod) + beta * f(y, ot), abs(alpha) * add(np.abs(prod)) + np.abs(beta * f(y, ot))
        if ot == "bf16":  # the one rounding of the result, 8 bits
            scale = scale + np.abs(want) * 2.0 ** -8 / helpers.TOL[vt]
        helpers.assert_rowwise(f(got, ot), want, scale + 1e-12, helpers.TOL[vt], f"unplanned {vt} mean {mean}")


@pytest.mark.parametrize("items", [1 << 18, (1 << 18) + 1, 1 << 23, (1 << 23) + 1])
def test_tile_sizes_of_the_entry_point_without_scratch(pkg, device, oracle, items):
    """rows + entries at which the tiles change size; rows that span tiles, empty rows, a ragged last tile."""
    from ctypes import c_float, c_int, c_int64, c_void_p
    rng = np.random.default_rng(items)
    m, n = items // 40, 50000
    nnz = items - m
    rp = np.concatenate([[0], np.sort(rng.integers(0, nnz + 1, m - 1)), [nnz]]).astype(np.int32)
    rp[m // 2:m // 2 + m // 50] = rp[m // 2]  # a long row after a stretch of empty ones
    ci = rng.integers(0, n, nnz).astype(np.int32)
    val, x, y = (rng.standard_normal(k).astype(np.float32) for k in (nnz, n, m))
    f = pkg.lib().b200sp_spmv_f32_noalloc
    f.restype, f.argtypes = c_int, [c_void_p] * 5 + [c_int64] * 3 + [c_float] * 2 + [c_void_p]
    d = [torch.from_numpy(a).to(device) for a in (rp, ci, val, x, y)]
    assert f(*(c_void_p(t.data_ptr()) for t in d), m, n, nnz, 1.5, -0.5,
             c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    want = oracle.spmv(rp, ci, val, x, y, 1.5, -0.5)
    scale = 1.5 * oracle.spmv_abs_rowsum(rp, ci, val, x) + 0.5 * np.abs(y) + 1e-12
    helpers.assert_rowwise(d[4].cpu().numpy().astype(np.float64), want.astype(np.float64), scale, helpers.TOL["f32"], "tiles")


def whole_case(device, seed):
    """An int32 matrix with listed rows of one and of several segments, and the product of it, on the GPU and exact."""
    from ops_sparse_b200 import api, synth
    rng = np.random.default_rng(seed)
    lengths = np.concatenate([rng.integers(0, 9, 3000), [1025, 8193, 20000] * 3])
    rng.shuffle(lengths)
    m, n = lengths.size, 30000
    A = synth.csr_from_lengths(rng, lengths, n, lambda r, k: r.integers(-9, 10, k))
    val, x, y = A.values.astype(np.int32), rng.integers(-9, 10, n).astype(np.int32), rng.integers(-9, 10, m).astype(np.int32)
    total = np.concatenate([[0], np.cumsum(val.astype(np.int64) * x[A.col_ind])])
    want = (2 * (total[A.row_ptr[1:]] - total[A.row_ptr[:-1]]) - y).astype(np.int32)
    dA = helpers.make_csr(device, A.row_ptr, A.col_ind, val, "i32", m, n)
    return dA, api.DnVec(helpers.to_device(x, "i32", device)), lambda: api.DnVec(helpers.to_device(y, "i32", device)), want


@pytest.mark.parametrize("offset", [0, 4])  # bytes from an aligned address: any word will do
def test_scratch_with_anything_in_it(pkg, handle, device, offset):
    """The list may hold whatever an unfinished product, or one of another matrix, left there."""
    from ctypes import Structure, byref, c_float, c_int, c_int32, c_int64, c_size_t, c_void_p
    from ops_sparse_b200 import api

    class Scalars(Structure):  # b200spScalars
        _fields_ = [("alpha_f", c_float), ("beta_f", c_float), ("alpha_i", c_int32), ("beta_i", c_int32),
                    ("alpha_dev", c_void_p), ("beta_dev", c_void_p)]
    dA, dx, make_y, want = whole_case(device, 1)
    rows_bytes, launch = pkg.lib().b200sp_spmv_rows_bytes, pkg.lib().b200sp_spmv_rows_launch
    rows_bytes.restype, rows_bytes.argtypes = c_size_t, [c_int64]
    launch.restype = c_int
    launch.argtypes = [c_void_p] * 5 + [c_int64] * 2 + [c_void_p] + [c_int] * 3 + [c_void_p] * 3
    ptr = lambda t: c_void_p(t.data_ptr())
    i32 = 3  # B200SP_I32
    dB, dv, make_w, other = whole_case(device, 2)
    bytes_ = max(rows_bytes(dA.nnz), rows_bytes(dB.nnz)) + offset
    for fill in (0x00, 0x5A, 0xFF):
        scratch = torch.full((bytes_,), fill, dtype=torch.uint8, device=device)[offset:]
        state = torch.full((2,), 0x5A5A5A5A, dtype=torch.int32, device=device)
        for M, dense, make, result in ((dA, dx, make_y, want), (dB, dv, make_w, other), (dA, dx, make_y, want)):
            dy = make()
            assert launch(ptr(M.row_ptr), ptr(M.col_ind), ptr(M.values), ptr(dense.values), ptr(dy.values), M.rows, M.nnz,
                          byref(Scalars(alpha_i=2, beta_i=-1)), i32, i32, i32, ptr(scratch), ptr(state),
                          c_void_p(handle.stream.cuda_stream)) == 0
            assert np.array_equal(helpers.to_host(dy.values, "i32"), result)
    dy = make_y()  # and through the interface, with a buffer of that alignment
    buf = torch.full((api.spmv_buffer_size(handle, dA, dx, dy) + offset,), 0x5A, dtype=torch.uint8, device=device)[offset:]
    api.spmv(handle, dA, dx, dy, 2, -1, buffer=buf)
    assert np.array_equal(helpers.to_host(dy.values, "i32"), want)


def test_handle_that_changes_its_stream(pkg, handle, device):
    """Products without a buffer share the handle's workspace; in order, whatever the stream, each finds its own list."""
    from ctypes import c_void_p
    from ops_sparse_b200 import api
    cases = [whole_case(device, seed) for seed in range(3)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    results = []
    for i in range(12):
        dA, dx, make_y, want = cases[i % 3]
        dy = make_y()
        torch.cuda.synchronize()
        s, before = streams[i % 2], streams[(i + 1) % 2]
        s.wait_stream(before)
        assert pkg.lib().aclsparseSetStream(handle.raw, c_void_p(s.cuda_stream)) == 0
        api.spmv(handle, dA, dx, dy, 2, -1)
        results.append((dy, want))
    torch.cuda.synchronize()
    for dy, want in results:
        assert np.array_equal(helpers.to_host(dy.values, "i32"), want)
