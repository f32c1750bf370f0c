"""GPU: SpMM with B rows of 512 and 1024 bytes, on either side of the rules that choose the row stream, the rows a warp of it
takes, and whether units of long rows are CTAs of its grid."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from test_spmm_gpu import check_compact, compact_case, run_spmm

pytestmark = pytest.mark.gpu

KINDS = [("bf16", "f32", 256), ("f16", "f16", 256), ("f32", "f32", 128), ("f32", "f32", 256), ("bf16", "bf16", 512)]
# the last rows for SpmmFastKernel and the first for the stream; two, four and eight rows a warp, the last warp with one row
ROWS = [16383, 16384, 28417, 56833]


def product(handle, device, oracle, lengths, k, vt, ot, n):
    rng = np.random.default_rng(lengths.size + n)
    m = lengths.size
    rp, ci, val, B, C = compact_case(oracle, rng, m, k, n, lengths, vt, ot, 1.5, -0.5)
    got = run_spmm(handle, device, rp, ci, val, vt, B, C, ot, m, k, n, n, n, 1.5, -0.5).reshape(m, n)
    check_compact(oracle, rp, ci, val, B, C, vt, ot, 1.5, -0.5, got, f"{vt}->{ot} n={n} m={m}")
    if vt == "f32":
        gold = oracle.spmm_f32_layout(m, n, rp, ci, val, B, n, True, False, C, n, True, 1.5, -0.5)
    else:
        gold = oracle.spmm_16(rp, ci, val, B, C, 1.5, -0.5, vt, ot)
    short = lengths <= 1024
    assert np.array_equal(got[short].view(np.uint8), np.asarray(gold).reshape(m, n)[short].view(np.uint8))


@pytest.mark.parametrize("m", ROWS)
@pytest.mark.parametrize("vt,ot,n", KINDS)
def test_rows(handle, device, oracle, vt, ot, n, m):
    """Rows of 0 to 6 entries, one of exactly a batch of copies, of a chunk of lookups, and of one more, first and last."""
    lengths = np.random.default_rng(m).integers(0, 7, m)
    lengths[[0, 1, 2, 3, m - 2, m - 1]] = [8, 9, 32, 0, 33, 64]
    product(handle, device, oracle, lengths, 3000, vt, ot, n)


@pytest.mark.parametrize("m", [16383, 20011])
@pytest.mark.parametrize("vt,ot,n", KINDS)
def test_long_rows(handle, device, oracle, vt, ot, n, m):
    """Rows above 1024 entries and a B of more than 96 MB: units of their own kernel, and of the stream's grid; units of one
    entry, of a request, a chunk and one more."""
    k = (100 << 20) // (n * (4 if vt == "f32" else 2)) + 1
    lengths = np.random.default_rng(m).integers(0, 5, m)
    lengths[[0, 5, m // 2, m - 1]] = [1025, 1024, 3000, 1500]
    product(handle, device, oracle, lengths, k, vt, ot, n)


def test_skewed_rows(handle, device, oracle):
    """More than a thousandth of the rows above four times the mean: SpmmFastKernel, which sums those apart."""
    lengths = np.random.default_rng(3).integers(0, 5, 20000)
    lengths[::500] = 200
    product(handle, device, oracle, lengths, 3000, "bf16", "f32", 256)


def streams(pkg, A):
    on = ctypes.c_int32()
    assert pkg.lib().b200spSpMMToRowStream(A.raw, ctypes.byref(on)) == 0
    return bool(on.value)


def planned(handle, device, rp, ci, val, B, C, vt, ot, m, k, n, ldb=0, ldc=0):
    """Descriptors and an analysed buffer; rows of B and C `ldb` and `ldc` elements apart, NaN between them."""
    import helpers
    from ops_sparse_b200 import api

    def stored(a, kind, ld):
        wide = torch.full((a.shape[0], ld or n), float("nan"), dtype=helpers.TORCH_OF[kind], device=device)
        wide[:, :n] = helpers.to_device(a, kind, device).view(a.shape[0], n)
        return wide
    A = helpers.make_csr(device, rp, ci, val, vt, m, k)
    dB = api.DnMat(stored(B, vt, ldb), k, n, ldb or n, "row")
    dC = api.DnMat(stored(C, ot, ldc), m, n, ldc or n, "row")
    return A, dB, dC, api.spmm_preprocess(handle, A, dB, dC)


@pytest.mark.parametrize("vt,ot,n", KINDS)
def test_beta_zero_and_device_scalars(pkg, handle, device, oracle, vt, ot, n):
    """Rows with and without entries: beta = 0 reads no NaN of C, on the host and on the device; device scalars give the host's bits."""
    from ops_sparse_b200 import api
    m, k, rng = 16384, 3000, np.random.default_rng(n)
    lengths = rng.integers(0, 7, m)
    lengths[[0, 5, m - 1]] = [0, 40, 0]
    rp, ci, val, B, C = compact_case(oracle, rng, m, k, n, lengths, vt, ot, 1.5, -0.5)
    A, dB, dC, buf = planned(handle, device, rp, ci, val, B, C, vt, ot, m, k, n)
    assert streams(pkg, A)
    start = dC.values.clone()
    bits = lambda: dC.values.clone().view(torch.uint8)
    api.spmm(handle, A, dB, dC, 1.5, -0.5, buffer=buf)
    torch.cuda.synchronize()
    with_beta = bits()
    dC.values.zero_()
    api.spmm(handle, A, dB, dC, 1.5, 0.0, buffer=buf)
    torch.cuda.synchronize()
    without = bits()
    dC.values.fill_(float("nan"))
    api.spmm(handle, A, dB, dC, 1.5, 0.0, buffer=buf)
    torch.cuda.synchronize()
    assert torch.equal(bits(), without)
    handle.set_pointer_mode_device(True)
    try:
        for beta, begin, want in ((-0.5, start, with_beta), (0.0, torch.full_like(start, float("nan")), without)):
            dC.values.copy_(begin)
            a, b = (torch.tensor(v, dtype=torch.float32, device=device) for v in (1.5, beta))
            api.spmm(handle, A, dB, dC, a, b, buffer=buf)
            torch.cuda.synchronize()
            assert torch.equal(bits(), want)
    finally:
        handle.set_pointer_mode_device(False)


@pytest.mark.parametrize("m,on", [(262143, False), (262144, True)])
def test_many_skewed_rows(pkg, handle, device, oracle, m, on):
    """A thousandth of the rows above four times the mean: the stream takes them from 262,144 rows on."""
    from ops_sparse_b200 import api
    rng, k, n = np.random.default_rng(4), 3000, 256
    lengths = rng.integers(0, 3, m)
    lengths[::500] = 200
    rp, ci, val, B, C = compact_case(oracle, rng, m, k, n, lengths, "bf16", "f32", 1.5, 0.0)
    A, dB, dC, buf = planned(handle, device, rp, ci, val, B, C, "bf16", "f32", m, k, n)
    assert streams(pkg, A) == on
    api.spmm(handle, A, dB, dC, 1.5, 0.0, buffer=buf)
    torch.cuda.synchronize()
    gold = oracle.spmm_16(rp, ci, val, B, C, 1.5, 0.0, "bf16", "f32")
    assert np.array_equal(dC.values.cpu().numpy().view(np.uint8), np.asarray(gold).reshape(m, n).view(np.uint8))


@pytest.mark.parametrize("vt,ot,n", KINDS)
def test_long_rows_beside_and_in_the_stream(pkg, handle, device, oracle, vt, ot, n):
    """The same matrix with one empty row more: units in a kernel of their own and in the stream's grid, the same bits, twice, with rows of B
    and C that lie apart."""
    from ops_sparse_b200 import api
    m, rng = 16383, np.random.default_rng(n)
    k = (100 << 20) // (n * (4 if vt == "f32" else 2)) + 1
    lengths = rng.integers(0, 5, m)
    lengths[[0, 5, m // 2, m - 1]] = [1025, 1024, 1500, 5000]
    rp, ci, val, B, C = compact_case(oracle, rng, m, k, n, lengths, vt, ot, 1.5, -0.5)
    vec = 4 if vt == "f32" else 8
    results = []
    for rows, ldb, ldc in ((m, 0, 0), (m + 1, 0, 0), (m + 1, n + vec, n + 2 * vec), (m, n + 3 * vec, n + vec)):
        rp2, C2 = np.append(rp, rp[-1:]) if rows > m else rp, np.append(C, C[:1], axis=0) if rows > m else C
        A, dB, dC, buf = planned(handle, device, rp2, ci, val, B, C2, vt, ot, rows, k, n, ldb, ldc)
        assert streams(pkg, A) == (rows > m)
        info = (ctypes.c_int32 * 4)()
        assert pkg.lib().b200spSpMMPlanInfo(A.raw, info) == 0 and info[1] > 0
        start = dC.values.clone()
        for _ in range(2):
            dC.values.copy_(start)
            api.spmm(handle, A, dB, dC, 1.5, -0.5, buffer=buf)
            torch.cuda.synchronize()
            results.append(dC.values[:m, :n].contiguous().view(torch.uint8).clone())
            assert bool(dC.values[:, n:].isnan().all())
    assert all(torch.equal(r, results[0]) for r in results)


def test_wait_that_runs_out_and_recovery(pkg, handle, device, oracle):
    """As test_spmm_gpu's, on a product that goes to the stream without the test's hook, too, and has units of long rows."""
    from ops_sparse_b200 import ACL_FLOAT, api
    L = pkg.lib()
    L.b200sp_spmm_stream_wait_test.argtypes = [ctypes.c_longlong, ctypes.c_uint]
    L.b200sp_spmm_stream_wait_test.restype = None
    m, n, rng = 16384, 256, np.random.default_rng(3)
    k = (100 << 20) // (2 * n) + 1
    lengths = rng.integers(0, 4, m)
    lengths[[7, 9000]] = [3000, 1025]
    rp, ci, val, B, C = compact_case(oracle, rng, m, k, n, lengths, "bf16", "f32", 1.0, 1.0)
    A, dB, dC, buf = planned(handle, device, rp, ci, val, B, C, "bf16", "f32", m, k, n)
    assert streams(pkg, A)
    assert L.b200sp_spmm_stream_error() == 0
    start = dC.values.clone()
    api.spmm(handle, A, dB, dC, 1.0, 1.0, buffer=buf)
    torch.cuda.synchronize()
    want = dC.values.clone()
    dC.values.copy_(start)
    try:
        L.b200sp_spmm_stream_wait_test(1 << 20, 16)
        api.spmm(handle, A, dB, dC, 1.0, 1.0, buffer=buf)
        torch.cuda.synchronize()
        assert L.b200sp_spmm_stream_error() == 1
        short = torch.from_numpy(lengths <= 1024).to(device)
        assert torch.equal(dC.values[short], start[short])
    finally:
        L.b200sp_spmm_stream_wait_test(0, 0)
    args = (handle.raw, 0, 0, None, A.raw, dB.raw, None, dC.raw, ACL_FLOAT, 0, api._ptr(buf))
    assert L.aclsparseSpMMPreprocess(*args) == pkg.ACL_SPARSE_STATUS_EXECUTION_FAILED
    assert L.aclsparseSpMMPreprocess(*args) == 0
    assert streams(pkg, A)
    dC.values.copy_(start)
    api.spmm(handle, A, dB, dC, 1.0, 1.0, buffer=buf)
    torch.cuda.synchronize()
    assert L.b200sp_spmm_stream_error() == 0
    assert torch.equal(dC.values, want)


def test_no_wait_ran_out(pkg, device):  # last in this file: of all products above but those that were told to
    torch.cuda.synchronize()
    assert pkg.lib().b200sp_spmm_stream_error() == 0
