"""GPU: SpMM at the row lengths and widths where its kernels change (rows summed apart from their neighbours, rows cut
every 1024 entries, 64-byte slices of B, repacked layouts)."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse
import torch

from test_spmm_gpu import check_compact, compact_case, run_spmm

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 1023, 1024, 1025, 2048, 2049, 9000]
# one lane to several tiles of 32 per row of B, whole and ragged 64-byte slices and 16-byte pieces
WIDTHS = [1, 4, 5, 8, 12, 16, 31, 40, 64, 100, 136, 300]


def case(oracle, vt, ot, n, filler):
    rng = np.random.default_rng(n + filler)
    # few rows: every row above 16 entries is a unit; more: those above 64, or above four times the mean
    extra = 300 if filler == 3 else 148 * 512 // max(n, 16) + 1
    lengths = rng.permutation(np.concatenate([EDGES, np.full(extra, filler)]))
    m, k = lengths.size, 9000
    return m, k, *compact_case(oracle, rng, m, k, n, lengths, vt, ot, 1.5, -0.5)


@pytest.mark.parametrize("vt,ot", [("f32", "f32"), ("f16", "f16"), ("bf16", "bf16"), ("bf16", "f32")])
@pytest.mark.parametrize("order", ["row", "col"])
@pytest.mark.parametrize("n", WIDTHS)
@pytest.mark.parametrize("filler", [3, 30])
def test_row_lengths(handle, device, oracle, filler, n, order, vt, ot):
    """The golden's bits for rows of up to 1024 entries, its tolerance for the others."""
    if n == 1 and filler != 3:
        filler = 4  # rows enough for the SMs are many here
    m, k, rp, ci, val, B, C = case(oracle, vt, ot, n, filler)
    stored = (lambda a: a) if order == "row" else (lambda a: np.ascontiguousarray(a.T))
    ldb, ldc = (n, n) if order == "row" else (k, m)
    got = run_spmm(handle, device, rp, ci, val, vt, stored(B), stored(C), ot, m, k, n, ldb, ldc, 1.5, -0.5,
                   b_order=order, c_order=order)
    got = got.reshape(m, n) if order == "row" else np.ascontiguousarray(got.reshape(n, m).T)
    check_compact(oracle, rp, ci, val, B, C, vt, ot, 1.5, -0.5, got, f"{vt}->{ot} n={n} {order} filler={filler}")
    if vt == "f32":
        gold = oracle.spmm_f32_layout(m, n, rp, ci, val, B, n, True, False, C, n, True, 1.5, -0.5)
    else:
        gold = oracle.spmm_16(rp, ci, val, B, C, 1.5, -0.5, vt, ot)
    short = np.diff(rp) <= 1024
    assert np.array_equal(got[short].view(np.uint8), np.asarray(gold).reshape(m, n)[short].view(np.uint8))


@pytest.mark.parametrize("n", [3, 16, 150])
def test_compensated_sums(handle, device, oracle, n):
    from ops_sparse_b200 import ACL_SPARSE_SPMM_CSR_FP32_HIGH_PRECISION_ALG as KAHAN
    m, k, rp, ci, val, B, C = case(oracle, "f32", "f32", n, 5)
    got = run_spmm(handle, device, rp, ci, val, "f32", B, C, "f32", m, k, n, n, n, 1.5, -0.5, alg=KAHAN).reshape(m, n)
    exact = 1.5 * np.stack([val[s:e].astype(np.float64) @ B[ci[s:e]].astype(np.float64) for s, e in zip(rp, rp[1:])]) - 0.5 * C
    scale = 1.5 * oracle.spmm_abs_sum(rp, ci, val, B, "f32") + np.abs(0.5 * C)
    # compensated: 2 eps and a term in eps^2 n per unit, plus the rounding of at most nine units' sums and of the epilogue
    assert np.all(np.abs(got - exact) <= 16 * 2.0 ** -24 * scale + 1e-30)


@pytest.mark.parametrize("order", ["row", "col"])
@pytest.mark.parametrize("n", [1, 8, 16, 17, 32, 33, 64, 100, 300])
@pytest.mark.parametrize("filler", [3, 60, 200])
def test_int8(handle, device, oracle, filler, n, order):
    rng = np.random.default_rng(n + filler)
    lengths = rng.permutation(np.concatenate([EDGES, np.full(300 if filler == 3 else 148 * 512 // max(n, 16) + 1, filler)]))
    m, k = lengths.size, 2500
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    ci = rng.integers(0, k, rp[-1]).astype(np.int32)
    val = rng.integers(-128, 128, rp[-1]).astype(np.int8)
    B = rng.integers(-128, 128, (k, n)).astype(np.int8)
    C = rng.integers(-1000, 1000, (m, n)).astype(np.int32)
    stored = (lambda a: a) if order == "row" else (lambda a: np.ascontiguousarray(a.T))
    ldb, ldc = (n, n) if order == "row" else (k, m)
    got = run_spmm(handle, device, rp, ci, val, "i8", stored(B), stored(C), "i32", m, k, n, ldb, ldc, 2, -1,
                   b_order=order, c_order=order)
    got = got.reshape(m, n) if order == "row" else got.reshape(n, m).T
    import scipy.sparse
    A = scipy.sparse.csr_matrix((val.astype(np.int64), ci, rp), shape=(m, k))
    assert np.array_equal(got, (2 * (A @ B.astype(np.int64)) - C).astype(np.int32))


@pytest.mark.parametrize("order", ["row", "col"])
@pytest.mark.parametrize("vt,ot", [("f32", "f32"), ("f16", "f16"), ("i8", "i32")])
@pytest.mark.parametrize("m,k,entries", [(4000, 4000, 1), (4000, 4000, 4), (4000, 4000, 5), (40_000, 1666, 1), (40_000, 1667, 1)])
def test_rows_of_a_few_entries(handle, device, oracle, m, k, entries, vt, ot, order):
    """Both sides of the rule that gives such rows a thread per output: entries of a row, columns of B, uses of a row of B."""
    rng = np.random.default_rng(m + k + entries)
    lengths = np.full(m, entries)
    for n in (1, 3, 4, 5, 8, 9, 10, 11, 12, 13, 16, 17):
        if vt == "i8":
            rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
            ci = rng.integers(0, k, rp[-1]).astype(np.int32)
            val, B = (rng.integers(-128, 128, shape).astype(np.int8) for shape in (ci.size, (k, n)))
            C = rng.integers(-1000, 1000, (m, n)).astype(np.int32)
            alpha, beta = 2, -1
        else:
            alpha, beta = 1.5, -0.5
            rp, ci, val, B, C = compact_case(oracle, rng, m, k, n, lengths, vt, ot, alpha, beta)
        stored = (lambda a: a) if order == "row" else (lambda a: np.ascontiguousarray(a.T))
        ldb, ldc = (n, n) if order == "row" else (k, m)
        got = run_spmm(handle, device, rp, ci, val, vt, stored(B), stored(C), ot, m, k, n, ldb, ldc, alpha, beta,
                       b_order=order, c_order=order)
        got = got.reshape(m, n) if order == "row" else np.ascontiguousarray(got.reshape(n, m).T)
        if vt == "i8":
            want = 2 * np.add.reduceat(val.astype(np.int64)[:, None] * B[ci].astype(np.int64), rp[:-1]) - C
            assert np.array_equal(got, want.astype(np.int32))
            continue
        if vt == "f32":
            gold = oracle.spmm_f32_layout(m, n, rp, ci, val, B, n, True, False, C, n, True, alpha, beta)
        else:
            gold = oracle.spmm_16(rp, ci, val, B, C, alpha, beta, vt, ot)
        assert np.array_equal(got.view(np.uint8), np.asarray(gold).reshape(m, n).view(np.uint8))


@pytest.mark.parametrize("order", ["row", "col"])
@pytest.mark.parametrize("vt,ot,n", [("f32", "f32", 16), ("f16", "f16", 37), ("bf16", "f32", 64), ("f32", "f32", 64), ("bf16", "bf16", 120)])
def test_rows_in_order_of_their_lengths(handle, device, oracle, vt, ot, n, order):
    """Rows enough for CTAs of 32 that take them by length (4 to 16 lanes a row): the golden's bits, ties and empty rows among them."""
    rng = np.random.default_rng(n)
    m, k = 4 * 32 * 148 + 13, 3000
    lengths = rng.integers(0, 12, m)
    lengths[64:128] = 7                      # CTAs of equal rows
    lengths[rng.integers(0, m, 200)] = 100   # rows summed apart
    rp, ci, val, B, C = compact_case(oracle, rng, m, k, n, lengths, vt, ot, 1.5, -0.5)
    stored = (lambda a: a) if order == "row" else (lambda a: np.ascontiguousarray(a.T))
    ldb, ldc = (n, n) if order == "row" else (k, m)
    got = run_spmm(handle, device, rp, ci, val, vt, stored(B), stored(C), ot, m, k, n, ldb, ldc, 1.5, -0.5,
                   b_order=order, c_order=order)
    got = got.reshape(m, n) if order == "row" else np.ascontiguousarray(got.reshape(n, m).T)
    if vt == "f32":
        gold = oracle.spmm_f32_layout(m, n, rp, ci, val, B, n, True, False, C, n, True, 1.5, -0.5)
    else:
        gold = oracle.spmm_16(rp, ci, val, B, C, 1.5, -0.5, vt, ot)
    assert np.array_equal(got.view(np.uint8), np.asarray(gold).reshape(m, n).view(np.uint8))


# lanes a row and what the kernel is asked for beside: compensated sums, B by words, C in rows of any width, scalars on the device
@pytest.mark.parametrize("vt,ot,m,k,n,most,kind", [
    ("f32", "f32", 18957, 3000, 32, 40, "plain"), ("f32", "f32", 18957, 3000, 32, 40, "kahan"),
    ("f32", "f32", 28423, 90000, 37, 40, "plain"), ("f16", "f16", 28423, 90000, 74, 40, "plain"), ("f32", "f32", 18957, 60000, 21, 40, "kahan"),
    ("f16", "f16", 18957, 3000, 32, 40, "plain"), ("bf16", "bf16", 5003, 3000, 24, 40, "device"), ("f32", "f32", 5003, 3000, 16, 140, "plain"),
    ("f32", "f32", 5003, 3000, 13, 140, "kahan"), ("bf16", "f32", 18957, 3000, 64, 40, "wide"), ("f32", "f32", 28423, 3000, 64, 40, "device"),
])
def test_uneven_rows_in_order_of_their_lengths(handle, device, oracle, vt, ot, m, k, n, most, kind):
    """The rules' own ranges: four lanes from 8 (64) entries on, more lanes from 1700 entries for every SM on; the golden's bits."""
    from ops_sparse_b200 import ACL_SPARSE_SPMM_CSR_FP32_HIGH_PRECISION_ALG as KAHAN
    rng = np.random.default_rng(n)
    lengths = rng.integers(0, most + 1, m)
    lengths[64:128] = most // 2              # CTAs of equal rows
    lengths[128:160] = 0                     # ... and of empty ones
    rp, ci, val, B, C = compact_case(oracle, rng, m, k, n, lengths, vt, ot, 1.5, -0.5)
    ldc = n + 1 if kind == "wide" else n
    stored = np.zeros((m, ldc), C.dtype)
    stored[:, :n] = C
    alpha, beta = 1.5, -0.5
    if kind == "device":
        handle.set_pointer_mode_device(True)
        alpha, beta = (torch.tensor(v, dtype=torch.float32, device=device) for v in (1.5, -0.5))
    got = run_spmm(handle, device, rp, ci, val, vt, B, stored, ot, m, k, n, n, ldc, alpha, beta, alg=KAHAN if kind == "kahan" else 0)
    got = got.reshape(m, ldc)
    assert not got[:, n:].any()
    got = np.ascontiguousarray(got[:, :n])
    if kind == "kahan":
        exact = 1.5 * np.asarray(scipy.sparse.csr_matrix((val.astype(np.float64), ci, rp), shape=(m, k)) @ B.astype(np.float64)) - 0.5 * C
        scale = 1.5 * oracle.spmm_abs_sum(rp, ci, val, B, vt) + 0.5 * np.abs(C)
        # products one rounding, compensated sums two, alpha, beta and the last sum one each
        assert np.all(np.abs(got - exact) <= 6 * 2.0 ** -24 * scale)
        return
    if vt == "f32":
        gold = oracle.spmm_f32_layout(m, n, rp, ci, val, B, n, True, False, C, n, True, 1.5, -0.5)
    else:
        gold = oracle.spmm_16(rp, ci, val, B, C, 1.5, -0.5, vt, ot)
    assert np.array_equal(got.view(np.uint8), np.asarray(gold).reshape(m, n).view(np.uint8))


@pytest.mark.parametrize("n", [17, 32, 48, 64])
@pytest.mark.parametrize("m,outliers", [(500, 0), (9471, 0), (9473, 0), (9473, 7)])  # few rows; enough; enough with a few long ones
def test_int8_rows_that_are_waited_for(handle, device, oracle, m, n, outliers):
    rng = np.random.default_rng(m + n)
    k = 2000
    lengths = rng.integers(0, 40, m)
    lengths[rng.integers(0, m, outliers)] = 900
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    ci = rng.integers(0, k, rp[-1]).astype(np.int32)
    val, B = (rng.integers(-128, 128, shape).astype(np.int8) for shape in (rp[-1], (k, n)))
    C = rng.integers(-1000, 1000, (m, n)).astype(np.int32)
    got = run_spmm(handle, device, rp, ci, val, "i8", B, C, "i32", m, k, n, n, n, 3, -2)
    assert np.array_equal(got.reshape(-1), oracle.spmm_i8(m, n, rp, ci, val, B, n, True, False, C, n, True, 3, -2))
