"""GPU: SpMVOp at the row lengths where its kernels change the number of lanes of a row."""
from __future__ import annotations

import numpy as np
import pytest

from test_spmv_op_gpu import check, run_op

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 2, 3, 4, 5, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 2500]


@pytest.mark.parametrize("offsets,base", [("i32", 0), ("i64", 1)])
@pytest.mark.parametrize("alg", [1, 2])
@pytest.mark.parametrize("filler", [2, 5, 20, 50, 100, 300])  # the mean length: 2 to 32 lanes per row, skewed or not
def test_row_lengths(pkg, handle, device, oracle, filler, alg, offsets, base):
    rng = np.random.default_rng(filler)
    lengths = rng.permutation(np.concatenate([EDGES, np.full(777, filler)])).astype(np.int64)
    k = 5000
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    ci = rng.integers(0, k, rp[-1]).astype(np.int32)
    val, x, y = (rng.uniform(-1.0, 1.0, s).astype(np.float32) for s in (int(rp[-1]), k, lengths.size))
    got = run_op(pkg, handle, device, rp, ci, val, x, y, 1.5, -0.5, k, offsets=offsets, base=base, alg=alg, runs=2)
    check(oracle, got, rp, ci, val, x, y, 1.5, -0.5, f"filler {filler} alg {alg}")


@pytest.mark.parametrize("offsets,base", [("i32", 0), ("i64", 1)])
@pytest.mark.parametrize("rows", [0, 3000, 60000])  # of 20 entries: all rows long ones; most entries in long rows; few
def test_rows_that_the_grid_would_wait_for(pkg, handle, device, oracle, rows, offsets, base):
    """Both sides of the lengths from which a row has a CTA of its own beside the grid (1024, 4096), and a wider one (16384)."""
    rng = np.random.default_rng(rows)
    outliers = [e + d for e in (1024, 2048, 4096, 8192, 16384) for d in (-1, 0, 1)] + [100_000]
    lengths = rng.permutation(np.concatenate([outliers, np.full(rows, 20)])).astype(np.int64)
    k = 5000
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    ci = rng.integers(0, k, rp[-1]).astype(np.int32)
    val, x, y = (rng.uniform(-1.0, 1.0, s).astype(np.float32) for s in (int(rp[-1]), k, lengths.size))
    got = run_op(pkg, handle, device, rp, ci, val, x, y, 1.5, -0.5, k, offsets=offsets, base=base, alg=2, runs=2)
    check(oracle, got, rp, ci, val, x, y, 1.5, -0.5, f"{rows} rows of 20")
