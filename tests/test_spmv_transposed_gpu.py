"""GPU: transposed aclsparseSpMV (scatter by chunks of entries) on row patterns that its row lookup has to get right."""
from __future__ import annotations

import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

PATTERNS = {
    "one entry each": lambda rng: np.ones(3000, np.int64),
    "mostly empty": lambda rng: (rng.random(200_000) < 0.01).astype(np.int64) * rng.integers(1, 5, 200_000),
    "empty stretches": lambda rng: np.concatenate([[3], np.zeros(70, np.int64), [300, 0, 1], np.zeros(33, np.int64), [40] * 31]),
    "33 rows a step": lambda rng: np.tile([1] * 31 + [0, 0, 2], 40),
    "long and short": lambda rng: np.concatenate([[5000], rng.integers(0, 3, 500), [256, 255, 257, 1]]),
    "a single row": lambda rng: np.array([777]),
    # the offsets are searched where a chunk of 256 entries spans more than 1024 rows
    "a long stretch inside a chunk": lambda rng: np.concatenate([[5] * 30, np.zeros(300_000, np.int64), [7] * 40]),
    "around the limit": lambda rng: np.concatenate([[100, *[0] * k, 200] for k in range(1019, 1028)]),
    "one row in a hundred": lambda rng: (rng.random(300_000) < 0.01).astype(np.int64),
}


@pytest.mark.parametrize("name", sorted(PATTERNS))
@pytest.mark.parametrize("copies", [1, 200])  # 200: several chunks per warp
def test_rows_of_every_entry(handle, device, name, copies):
    """int32, so exact: every entry must meet the x of its own row."""
    from ops_sparse_b200 import ACL_SPARSE_OP_TRANSPOSE, api
    rng = np.random.default_rng(len(name))
    base = PATTERNS[name](rng)
    lengths = np.tile(base, max(1, min(copies, 12_000_000 // max(int(base.sum()), base.size))))
    m, n, nnz = lengths.size, 4096, int(lengths.sum())
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    ci = rng.integers(0, n, nnz).astype(np.int32)
    val, x, y = (rng.integers(-9, 10, k).astype(np.int32) for k in (nnz, m, n))
    dA = helpers.make_csr(device, rp, ci, val, "i32", m, n)
    dx, dy = api.DnVec(helpers.to_device(x, "i32", device)), api.DnVec(helpers.to_device(y, "i32", device))
    buf = api.spmv_preprocess(handle, dA, dx, dy, ACL_SPARSE_OP_TRANSPOSE)
    api.spmv(handle, dA, dx, dy, 2, -1, op=ACL_SPARSE_OP_TRANSPOSE, buffer=buf)
    want = -y.astype(np.int64)
    want += 2 * np.bincount(ci, weights=val.astype(np.float64) * np.repeat(x, lengths), minlength=n).astype(np.int64)
    assert np.array_equal(helpers.to_host(dy.values, "i32"), want.astype(np.int32))
