"""GPU: planned aclsparseSpMV on banded matrices (every row short and near its neighbours), against the CPU golden."""
from __future__ import annotations

import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 127, 128, 129, 4097])  # around the 128 rows a CTA stages
@pytest.mark.parametrize("vt,ot", [("f32", "f32"), ("f16", "f32"), ("bf16", "bf16"), ("i32", "i32")])
@pytest.mark.parametrize("beta", [0, 1])
def test_banded_rows(handle, device, oracle, m, vt, ot, beta):
    """Rows of 8 to 32 entries (and a few empty ones) on a band; the last row ends at an odd offset."""
    from ops_sparse_b200 import api
    rng = np.random.default_rng(m)
    n = m + 40
    lengths = rng.integers(8, 33, m)
    lengths[rng.random(m) < 0.02] = 0
    lengths[-1] = 9
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    ci = np.concatenate([r + np.sort(rng.choice(40, k, replace=False)) for r, k in enumerate(lengths)]).astype(np.int32)
    whole = vt == "i32"
    make = (lambda k, t: rng.integers(-9, 10, k).astype(np.int32)) if whole else \
        (lambda k, t: oracle.to_storage(rng.standard_normal(k).astype(np.float32), t))
    val, x, y = make(rp[-1], vt), make(n, vt), make(m, ot)
    dA = helpers.make_csr(device, rp, ci, val, vt, m, n)
    dx, dy = api.DnVec(helpers.to_device(x, vt, device)), api.DnVec(helpers.to_device(y, ot, device))
    buf = api.spmv_preprocess(handle, dA, dx, dy)
    alpha = 2 if whole else 1.5
    api.spmv(handle, dA, dx, dy, alpha, beta, buffer=buf)
    got = helpers.to_host(dy.values, ot)
    row = np.repeat(np.arange(m), lengths)
    if whole:
        want = np.zeros(m, np.int64)
        np.add.at(want, row, val.astype(np.int64) * x[ci])
        assert np.array_equal(got, (alpha * want + beta * y).astype(np.int32))
        return
    f = lambda a, t: oracle.from_storage(a, t).astype(np.float64)
    prod, want, scale = f(val, vt) * f(x, vt)[ci], np.zeros(m), np.zeros(m)
    np.add.at(want, row, prod)
    np.add.at(scale, row, np.abs(prod))
    want, scale = alpha * want + beta * f(y, ot), alpha * scale + np.abs(beta * f(y, ot))
    if ot == "bf16":  # the one rounding of the result, 8 bits
        scale = scale + np.abs(want) * 2.0 ** -8 / helpers.TOL[vt]
    helpers.assert_rowwise(f(got, ot), want, scale + 1e-12, helpers.TOL[vt], f"banded {vt} m={m}")
