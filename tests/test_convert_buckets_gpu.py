"""GPU: csr2csc by buckets of columns, bit for bit: buckets that are empty, just fit into shared memory, just do not, and hold nearly
everything; every value size."""
from __future__ import annotations

from ctypes import byref, c_size_t, c_void_p

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def P(t):
    return c_void_p(t.data_ptr())


# 40,000 columns and 1.5 M entries: buckets of 512 columns, 19,200 entries on average
N, NNZ, WIDTH = 40_000, 1_500_003, 512


def columns(kind, rng):
    if kind == "even":
        return rng.integers(0, N, NNZ)
    if kind == "edges":  # 32,768 in a bucket, 32,769 in the next, one in the last, none in some, tiles that are full and not
        sizes = {3: 32768, 4: 32769, 5: 40960, 6: 8192 * 9 + 1, 78: 1}
        parts = [b * WIDTH + rng.integers(0, min(WIDTH, N - b * WIDTH), k) for b, k in sizes.items()]
        rest = NNZ - sum(sizes.values())
        parts.append((20 + rng.integers(0, 50, rest)) * WIDTH + rng.integers(0, WIDTH, rest))
        return rng.permutation(np.concatenate(parts))
    hub = rng.random(NNZ) < 0.95  # one bucket with nearly everything, most of it in one column
    return np.where(hub, np.where(rng.random(NNZ) < 0.5, 7 * WIDTH + 11, 7 * WIDTH + rng.integers(0, WIDTH, NNZ)), rng.integers(0, N, NNZ))


@pytest.mark.parametrize("bits", [0, 8, 16, 32])
@pytest.mark.parametrize("kind", ["even", "edges", "hub"])
@pytest.mark.parametrize("base", [0, 1])
def test_buckets(pkg, handle, device, kind, bits, base):
    L, S = pkg.lib(), pkg
    rng = np.random.default_rng(len(kind))
    m = 70_000
    rp = np.concatenate([[0], np.sort(rng.integers(0, NNZ + 1, m - 1)), [NNZ]]).astype(np.int32)
    ci = columns(kind, rng).astype(np.int32)
    val = rng.integers(0, 1 << max(bits, 1), NNZ, dtype=np.uint64).astype({0: np.uint8, 8: np.uint8, 16: np.uint16, 32: np.uint32}[bits])
    order = np.argsort(ci, kind="stable")
    rows = np.repeat(np.arange(m), np.diff(rp))
    acl, action = {0: (S.ACL_FLOAT, 0), 8: (S.ACL_INT8, 1), 16: (S.ACL_FLOAT16, 1), 32: (S.ACL_FLOAT, 1)}[bits]
    d_rp, d_ci = (torch.from_numpy(a + np.int32(base)).to(device) for a in (rp, ci))
    d_v = torch.from_numpy(val.view({1: np.int8, 2: np.int16, 4: np.int32}[val.itemsize])).to(device)
    o_v, o_ri = torch.zeros_like(d_v), torch.empty_like(d_ci)
    o_cp = torch.full((N + 1,), -3, dtype=torch.int32, device=device)
    size = c_size_t()
    args = (handle.raw, m, N, NNZ, P(d_v), P(d_rp), P(d_ci), P(o_v), P(o_cp), P(o_ri), acl, action, base, 0)
    assert L.aclsparseCsr2cscEx2_bufferSize(*args, byref(size)) == 0
    buf = torch.full((size.value,), 0x5A, dtype=torch.uint8, device=device)
    for _ in range(2):
        assert L.aclsparseCsr2cscEx2(*args, P(buf)) == 0
    torch.cuda.synchronize()
    want_cp = np.concatenate([[0], np.cumsum(np.bincount(ci, minlength=N))]) + base
    assert np.array_equal(o_cp.cpu().numpy(), want_cp)
    assert np.array_equal(o_ri.cpu().numpy(), rows[order] + base)
    if bits:
        assert np.array_equal(o_v.cpu().numpy(), d_v.cpu().numpy()[order])
