"""GPU: SpMM into a C of any layout: one kernel reads C, eight elements at a time, and one does not; beta on the host or the device."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from test_spmm_gpu import check_compact, compact_case, run_spmm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vt,ot", [("f32", "f32"), ("f16", "f16"), ("bf16", "f32")])
@pytest.mark.parametrize("n", [3, 7, 33, 40, 100])  # fewer elements than eight a lane, remainders, several tiles
@pytest.mark.parametrize("m", [37, 9001])
def test_layouts_and_scalars(handle, device, oracle, m, n, vt, ot):
    from ops_sparse_b200 import api
    rng = np.random.default_rng(m + n)
    k, alpha, beta = 3000, 1.5, -0.5
    rp, ci, val, B, C = compact_case(oracle, rng, m, k, n, rng.integers(0, 50, m), vt, ot, alpha, beta)
    flip = lambda a: np.ascontiguousarray(a.T)
    row = run_spmm(handle, device, rp, ci, val, vt, B, C, ot, m, k, n, n, n, alpha, beta).reshape(m, n)
    check_compact(oracle, rp, ci, val, B, C, vt, ot, alpha, beta, row, f"{vt} n={n} m={m}")
    col = run_spmm(handle, device, rp, ci, val, vt, flip(B), flip(C), ot, m, k, n, k, m, alpha, beta, b_order="col", c_order="col")
    assert np.array_equal(flip(col.reshape(n, m)).view(np.uint8), row.view(np.uint8))
    # beta on the device, not 0 and 0, into a C of NaN where nothing may be read
    import helpers
    A = helpers.make_csr(device, rp, ci, val, vt, m, k)
    nan = np.full_like(C, 0x7FFF) if ot != "f32" else np.full_like(C, np.nan)
    zero = run_spmm(handle, device, rp, ci, val, vt, B, nan, ot, m, k, n, n, n, alpha, 0.0).reshape(m, n)
    for order, b, stored, want in (("row", beta, C, row), ("col", beta, C, row), ("row", 0.0, nan, zero), ("col", 0.0, nan, zero)):
        put = (lambda a: a) if order == "row" else flip
        dB = api.DnMat(helpers.to_device(put(B), vt, device), k, n, n if order == "row" else k, order)
        dC = api.DnMat(helpers.to_device(put(stored), ot, device), m, n, n if order == "row" else m, order)
        buf = api.spmm_preprocess(handle, A, dB, dC)
        handle.set_pointer_mode_device(True)
        try:
            api.spmm(handle, A, dB, dC, *(torch.tensor(v, dtype=torch.float32, device=device) for v in (alpha, b)), buffer=buf)
            torch.cuda.synchronize()
        finally:
            handle.set_pointer_mode_device(False)
        got = helpers.to_host(dC.values, ot).reshape((m, n) if order == "row" else (n, m))
        assert np.array_equal((got if order == "row" else flip(got)).view(np.uint8), want.view(np.uint8)), (order, b)


@pytest.mark.parametrize("vt,ot", [("f32", "f32"), ("f16", "f16"), ("bf16", "f32")])
@pytest.mark.parametrize("n", [59, 60, 95, 96, 119, 120, 191, 192])  # fifteen sixteenths of a tile's columns; rows of 384 bytes
def test_either_side_of_the_rule(handle, device, oracle, n, vt, ot):
    test_layouts_and_scalars(handle, device, oracle, 9001, n, vt, ot)
