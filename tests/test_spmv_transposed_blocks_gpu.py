"""GPU: transposed aclsparseSpMV with so few columns that every SM adds up a y of its own: one column, the most that fit and one
more, in every type, with entries for one and for several chunks a warp and a last one that is not full."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vt,ot", [("f32", "f32"), ("f16", "f32"), ("bf16", "bf16"), ("i32", "i32")])
@pytest.mark.parametrize("cols,nnz", [(1, 70_001), (33, 200_003), (4096, 1_300_001), (49152, 4_000_037), (49153, 4_000_037)])
def test_few_columns(handle, device, cols, nnz, vt, ot):
    from ops_sparse_b200 import ACL_SPARSE_OP_TRANSPOSE, api
    rng = np.random.default_rng(cols)
    lengths = np.concatenate([[nnz // 3, 0, 0, 257], rng.integers(0, 40, nnz // 30)])
    lengths[-1] += nnz - int(lengths.sum())
    assert lengths[-1] >= 0
    m = lengths.size
    gen = torch.Generator(device=device).manual_seed(cols)
    rp = torch.from_numpy(np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)).to(device)
    ci = torch.randint(cols, (nnz,), generator=gen, device=device, dtype=torch.int32)
    whole = vt == "i32"
    draw = (lambda n: torch.randint(-9, 10, (n,), generator=gen, device=device, dtype=torch.int32)) if whole else (
        lambda n: torch.randn(n, generator=gen, device=device))
    val, x = (draw(n).to(helpers.TORCH_OF[vt]) for n in (nnz, m))
    y = draw(cols).to(helpers.TORCH_OF[ot])
    alpha, beta = (2, -1) if whole else (1.5, -0.5)
    wide = torch.int64 if whole else torch.float64
    rows = torch.repeat_interleave(torch.arange(m, device=device), torch.from_numpy(lengths).to(device))
    terms = alpha * val.to(wide) * x.to(wide)[rows]
    want = (beta * y.to(wide)).index_add(0, ci.long(), terms)
    scale = (abs(beta) * y.to(wide).abs()).index_add(0, ci.long(), terms.abs())
    A = api.CsrMatrix(rp, ci, val, m, cols)
    dx, dy = api.DnVec(x), api.DnVec(y.clone())
    buf = api.spmv_preprocess(handle, A, dx, dy, ACL_SPARSE_OP_TRANSPOSE)
    api.spmv(handle, A, dx, dy, alpha, beta, op=ACL_SPARSE_OP_TRANSPOSE, buffer=buf)
    torch.cuda.synchronize()
    if whole:
        assert torch.equal(dy.values.long(), want)
        return
    # fp32 additions in any order: (additions + 3) half ulps of the sum of magnitudes, and the rounding of a 16-bit result
    count = torch.bincount(ci.long(), minlength=cols).double()
    bound = (count + 3) * 2.0 ** -24 * scale + (2.0 ** -8 * want.abs() if ot == "bf16" else 0)
    assert bool(((dy.values.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("vt,ot", [("f32", "f32"), ("i32", "i32")])
@pytest.mark.parametrize("cols", [1, 30, 395, 1000])
@pytest.mark.parametrize("nnz", [30_011, 65_536, 65_537, 200_003, 600_007])  # CTAs with one chunk, with a chunk for every warp, and between
def test_columns_that_many_entries_share(handle, device, cols, nnz, vt, ot):
    from ops_sparse_b200 import ACL_SPARSE_OP_TRANSPOSE, api
    gen = torch.Generator(device=device).manual_seed(nnz + cols)
    m = (nnz + 9) // 10
    rp = torch.arange(m + 1, device=device).mul_(10).clamp_max_(nnz).to(torch.int32)
    ci = torch.randint(cols, (nnz,), generator=gen, device=device, dtype=torch.int32)
    ci[torch.rand(nnz, generator=gen, device=device) < 0.5] = cols // 2
    draw = lambda n: torch.randint(-9, 10, (n,), generator=gen, device=device, dtype=torch.int32).to(helpers.TORCH_OF[vt])  # sums below 2^24: exact
    val, x, y = draw(nnz), draw(m), draw(cols)
    rows = torch.arange(nnz, device=device) // 10
    want = (-y.to(torch.int64)).index_add(0, ci.long(), 2 * val.to(torch.int64) * x.to(torch.int64)[rows])
    A = api.CsrMatrix(rp, ci, val, m, cols)
    dx, dy = api.DnVec(x), api.DnVec(y.clone())
    buf = api.spmv_preprocess(handle, A, dx, dy, ACL_SPARSE_OP_TRANSPOSE)
    api.spmv(handle, A, dx, dy, 2, -1, op=ACL_SPARSE_OP_TRANSPOSE, buffer=buf)
    torch.cuda.synchronize()
    assert int(want.abs().max()) < 1 << 23
    assert torch.equal(dy.values.long(), want)
