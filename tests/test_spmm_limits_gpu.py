"""GPU: SpMM on matrices of as many entries as 32-bit offsets count: no position after the last entry may wrap."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

MOST = 2 ** 31 - 1


def product(handle, device, lengths, k, n, value, out, columns, tail):
    """C of a matrix whose entries are zero but for those of the last `tail` rows, and what those rows give."""
    from ops_sparse_b200 import api
    m = lengths.size
    rp = np.concatenate([[0], np.cumsum(lengths)])
    assert rp[-1] == MOST
    rng = np.random.default_rng(1)
    first = int(rp[m - tail])
    last = rng.integers(-8, 9, MOST - first).astype(np.int8)  # whole numbers: every sum is exact
    B = rng.integers(-8, 9, (k, n)).astype(np.int8)
    val = torch.zeros(MOST, dtype=value, device=device)
    val[first:] = torch.from_numpy(last).to(device).to(value)
    A = api.CsrMatrix(torch.from_numpy(rp.astype(np.int32)).to(device), columns, val, m, k)
    dB = api.DnMat(torch.from_numpy(B).to(device).to(value), k, n, n, "row")
    dC = api.DnMat(torch.full((m, n), 3, dtype=out, device=device), m, n, n, "row")
    buffer = api.spmm_preprocess(handle, A, dB, dC)
    api.spmm(handle, A, dB, dC, 1, 0, buffer=buffer)
    torch.cuda.synchronize()
    assert not dC.values[:m - tail].any()
    ci = columns[first:].cpu().numpy()
    want = np.stack([last[s:e].astype(np.int64) @ B[ci[s:e]].astype(np.int64)
                     for s, e in zip(rp[m - tail:-1] - first, rp[m - tail + 1:] - first)])
    assert np.array_equal(dC.values[m - tail:].cpu().numpy(), want)


def test_short_rows_at_the_end(handle, device):
    """Eight lanes a row: short and empty rows end the matrix in one warp with long ones."""
    lengths = np.full(2099203, 1023, dtype=np.int64)
    lengths[-16:] = [1000, 5, 1017, 0, 1020, 9, 8, 1, 1022, 7, 1021, 0, 33, 1019, 0, 3]
    while (over := int(lengths.sum()) - MOST) != 0:
        lengths[:-16][:abs(over)] -= 1 if over > 0 else -1
    product(handle, device, lengths, 64, 32, torch.float32, torch.float32,
            torch.arange(64, dtype=torch.int32, device=device).repeat(MOST // 64 + 1)[:MOST], 16)


def test_int8_rows_written_out_at_the_end(handle, device):
    """Full rows of the widest A that goes to the tensor cores, the last one in the middle of a request."""
    k = 12288
    lengths = np.full(MOST // k + 1, k, dtype=np.int64)
    lengths[-1] = MOST - k * (lengths.size - 1)
    product(handle, device, lengths, k, 16, torch.int8, torch.int32,
            torch.arange(k, dtype=torch.int32, device=device).repeat(lengths.size)[:MOST], 3)
