"""GPU: SpMM with B rows of 512 and 1024 bytes, on either side of the rules that choose the row stream, the rows a warp of it
takes, and whether units of long rows are CTAs of its grid."""
from __future__ import annotations

import numpy as np
import pytest

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
