"""GPU: planned aclsparseSpMV whose long rows are summed against blocks of x held in shared memory."""
from __future__ import annotations

import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

BLOCK = 32768  # columns of x that a CTA holds


# long rows and blocks for which 8, 32 and 256 lanes share the piece of a row inside a block
@pytest.mark.parametrize("longs,cols", [(2000, 8 * BLOCK), (5000, BLOCK), (100, BLOCK - 5)])
@pytest.mark.parametrize("vt,ot", [("f32", "f32"), ("f16", "f32")])
@pytest.mark.parametrize("shift", [0, 1])  # 1: col_ind and values off the 16-byte boundary, entry by entry
def test_rows_do_not_meet_columns_they_lack(handle, device, oracle, longs, cols, vt, ot, shift):
    """The first column of every block holds an infinity or a NaN and no row has an entry there."""
    import torch
    from ops_sparse_b200 import api
    rng = np.random.default_rng(longs)
    lengths = np.concatenate([rng.integers(512, 700, longs), rng.integers(0, 40, 300)])
    rng.shuffle(lengths)
    m, nnz = lengths.size, int(lengths.sum())
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    row = np.repeat(np.arange(m), lengths)
    ci = rng.integers(1, cols, nnz)
    ci += ci % BLOCK == 0
    ci = np.minimum(ci, cols - 1)
    ci = (np.sort(row * cols + ci) - row * cols).astype(np.int32)
    assert not np.any(ci % BLOCK == 0)
    val, x = (oracle.to_storage(rng.standard_normal(k).astype(np.float32), vt) for k in (nnz, cols))
    f = lambda a: oracle.from_storage(a, vt).astype(np.float64)
    prod = f(val) * f(x)[ci]
    want, scale = np.bincount(row, prod, m), np.bincount(row, np.abs(prod), m)
    marks = np.where(np.arange(0, cols, BLOCK) // BLOCK % 2 == 0, np.inf, np.nan).astype(np.float32)
    x[::BLOCK] = oracle.to_storage(marks, vt)
    d_ci = torch.zeros(nnz + 1, dtype=torch.int32, device=device)[shift:shift + nnz]
    d_val = torch.zeros(nnz + 1, dtype=helpers.TORCH_OF[vt], device=device)[shift:shift + nnz]
    d_ci.copy_(torch.from_numpy(ci))
    d_val.copy_(helpers.to_device(val, vt, device))
    dA = api.CsrMatrix(torch.from_numpy(rp).to(device), d_ci, d_val, m, cols)
    dx, dy = api.DnVec(helpers.to_device(x, vt, device)), api.DnVec(torch.empty(m, device=device))
    buf = api.spmv_preprocess(handle, dA, dx, dy)
    api.spmv(handle, dA, dx, dy, 1.0, 0.0, buffer=buf)
    got = dy.values.cpu().numpy().astype(np.float64)
    helpers.assert_rowwise(got, want, scale + 1e-12, helpers.TOL[vt], f"{longs} long rows, {cols} columns, {vt}")
