"""What the library is timed on: the work its users have it do, through its public entry points.

A case is a dict of plain values.  `listed()` names the fixed ones, `draw(rng)` gives one more of the same ranges,
`prepare(case, seed)` makes what a user's program holds before the call (inputs on the GPU, descriptors, analysed
buffers), `run(state)` is one pass, `work(case)` the bytes and operations a pass cannot do without and `tolerance(case)`
how far two correct implementations may lie apart.

Row lengths are drawn by quantile and shuffled by the seed, so that a case has the same number of entries with every
seed; columns are uniform without repetition inside a row and ascending (where the operation does not sort them
itself), the 27-point stencil apart.

Run with the repository's root as the working folder.
"""
from __future__ import annotations

import ctypes
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

DTYPE = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "i32": torch.int32, "i8": torch.int8}
BYTES = {"f32": 4, "f16": 2, "bf16": 2, "i32": 4, "i8": 1}


def package():
    name = "ops_sparse_b200"
    if name not in sys.modules:
        folder = Path.cwd() / "ops-sparse_b200"
        spec = importlib.util.spec_from_file_location(name, folder / "__init__.py",
                                                      submodule_search_locations=[str(folder)])
        module = importlib.util.module_from_spec(spec)
        sys.modules[name] = module
        spec.loader.exec_module(module)
    return sys.modules[name]


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # The smallest solver call: a 4096-row system with 16 entries a row, inside an iteration.  Latency.
        {"name": "spmv_f32_4096", "op": "spmv", "pattern": "fixed", "rows": 4096, "cols": 4096, "mean": 16,
         "value": "f32", "out": "f32", "alpha": 1.0, "beta": 0.0, "plan": True, "device_scalars": False},
        # Web / social graph products (PageRank and the like): power-law rows, a million of them, accumulated into y.
        {"name": "spmv_f32_powerlaw_1m", "op": "spmv", "pattern": "zipf", "rows": 1 << 20, "cols": 1 << 20,
         "mean": 32, "slope": 1.8, "cap": 16384, "value": "f32", "out": "f32", "alpha": 1.5, "beta": 0.5,
         "plan": True, "device_scalars": False},
        # A discretised PDE in mixed precision: 27-point stencil on a 128^3 grid, fp16 matrix and x, fp32 y.
        {"name": "spmv_f16_stencil_2m", "op": "spmv", "pattern": "stencil", "grid": 128, "value": "f16", "out": "f32",
         "alpha": 1.0, "beta": 0.0, "plan": True, "device_scalars": False},
        # The plainest call sequence: a product without any analysed buffer, once per matrix; ragged rows, odd sizes.
        {"name": "spmv_bf16_unplanned", "op": "spmv", "pattern": "ragged", "rows": 300007, "cols": 250001, "mean": 24,
         "value": "bf16", "out": "bf16", "alpha": 1.0, "beta": 0.5, "plan": False, "device_scalars": False},
        # The adjoint product of least-squares and BiCG solvers, rectangular, skewed rows.
        {"name": "spmv_f32_transposed", "op": "spmv_t", "pattern": "zipf", "rows": 500009, "cols": 400003, "mean": 24,
         "slope": 1.8, "cap": 16384, "value": "f32", "out": "f32", "alpha": 1.0, "beta": 0.0},
        # Block solvers and spectral methods: 64 right-hand sides at once.
        {"name": "spmm_f32_n64", "op": "spmm", "pattern": "fixed", "rows": 1 << 18, "cols": 1 << 18, "mean": 64,
         "n": 64, "value": "f32", "out": "f32", "alpha": 1.0, "beta": 0.5, "order": "row", "kahan": False},
        # Graph neural network, forward: aggregate 256 bf16 features over a power-law adjacency.  The largest.
        {"name": "spmm_bf16_graph_n256", "op": "spmm", "pattern": "zipf", "rows": 1 << 21, "cols": 1 << 21, "mean": 16,
         "slope": 2.0, "cap": 65536, "n": 256, "value": "bf16", "out": "f32", "alpha": 1.0, "beta": 0.0,
         "order": "row", "kahan": False},
        # Column-major B and C, the order numerical codes hold their vectors in; ragged rows, odd sizes.
        {"name": "spmm_f16_columns_n40", "op": "spmm", "pattern": "ragged", "rows": 65537, "cols": 50001, "mean": 24,
         "n": 40, "value": "f16", "out": "f16", "alpha": 1.0, "beta": 0.0, "order": "col", "kahan": False},
        # A pruned, quantised layer: 4096 x 4096 int8 weights at one tenth density against 512 int8 activations.
        {"name": "spmm_i8_pruned_n512", "op": "spmm", "pattern": "ragged", "rows": 4096, "cols": 4096, "mean": 410,
         "n": 512, "value": "i8", "out": "i32", "alpha": 1.0, "beta": 0.0, "order": "row", "kahan": False},
        # Graph neural network, backward: the gradient of the edge weights, sampled on the adjacency.
        {"name": "sddmm_f16_graph_k256", "op": "sddmm", "pattern": "zipf", "rows": 1 << 20, "cols": 1 << 20, "mean": 16,
         "slope": 2.0, "cap": 65536, "k": 256, "value": "f16", "alpha": 1.0, "beta": 0.0},
        # Assembly: COO to CSR offsets, the columns of every row sorted, the transpose's structure, each with the map
        # to the original entries through which values are refreshed at every reassembly.
        {"name": "assemble_powerlaw_1m", "op": "assemble", "pattern": "zipf", "rows": 1 << 20, "cols": 1 << 20,
         "mean": 32, "slope": 1.8, "cap": 16384},
        # Residuals of an iterative refinement: compensated row sums through the plan API.
        {"name": "spmvop_f32_powerlaw_1m", "op": "spmvop", "pattern": "zipf", "rows": 1 << 20, "cols": 1 << 20,
         "mean": 32, "slope": 1.8, "cap": 16384, "alpha": -1.0, "beta": 1.0, "alg": 2, "offsets": "i32"},
    ]


def spread(rng, low, high):
    """A whole number spread over the logarithm of [low, high]."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    op = rng.choice(["spmv", "spmv", "spmv", "spmv_t", "spmm", "spmm", "spmm", "sddmm", "assemble", "spmvop"])
    case = {"op": op}
    kinds = {"spmv": ["fixed", "zipf", "ragged", "stencil"], "spmv_t": ["zipf", "ragged", "stencil"]}
    case["pattern"] = rng.choice(kinds.get(op, ["fixed", "zipf", "ragged"]))
    if case["pattern"] == "stencil":
        case["grid"] = spread(rng, 16, 128)
    else:
        if op == "spmvop" and rng.random() < 0.3:
            case["pattern"] = "ragged"
        case["rows"] = spread(rng, 1000, 1 << 20)
        case["cols"] = case["rows"] if rng.random() < 0.5 else spread(rng, 1000, 1 << 20)
        case["mean"] = spread(rng, 2, 64)
        if case["pattern"] == "zipf":
            case["slope"] = rng.choice([1.8, 2.0])
            case["cap"] = min(16384, case["cols"] // 4)
        case["mean"] = min(case["mean"], max(2, (32 << 20) // case["rows"]))
    if op in ("spmv", "spmv_t"):
        case["value"], case["out"] = rng.choice([("f32", "f32"), ("f32", "f32"), ("f16", "f32"), ("bf16", "f32"),
                                                 ("f16", "f16"), ("bf16", "bf16"), ("i32", "i32")])
        whole = case["value"] == "i32"
        case["alpha"] = 1.0 if whole else rng.choice([1.0, 1.5])
        case["beta"] = 0.0 if whole else rng.choice([0.0, 0.5])
        if op == "spmv":
            case["plan"] = rng.random() < 0.7
            case["device_scalars"] = not whole and rng.random() < 0.25
    elif op == "spmm":
        case["value"], case["out"] = rng.choice([("f32", "f32"), ("f32", "f32"), ("f16", "f16"), ("bf16", "f32"),
                                                 ("bf16", "bf16"), ("i8", "i32")])
        n = spread(rng, 4, 512)
        case["n"] = n if rng.random() < 0.3 else max(8, n // 8 * 8)
        case["order"] = "row" if rng.random() < 0.7 else "col"
        case["kahan"] = case["value"] == "f32" and rng.random() < 0.15
        case["alpha"] = 1.0
        case["beta"] = 0.0 if case["value"] == "i8" else rng.choice([0.0, 0.5])
        if case["value"] == "i8":  # pruned weights: denser rows than a graph's or a discretisation's
            case["mean"] = spread(rng, 16, min(410, case["cols"] // 4))
        plain = case["order"] == "row" and case["n"] % 8 == 0 and case["value"] != "i8"
        case["rows"] = max(500, min(case["rows"], (1 << 30 if plain else 1 << 28) // (case["mean"] * case["n"])))
    elif op == "sddmm":
        case["value"] = rng.choice(["f32", "f16", "f16"])
        k = spread(rng, 16, 512)
        case["k"] = k if rng.random() < 0.3 else k // 8 * 8
        case["alpha"], case["beta"] = 1.0, rng.choice([0.0, 0.5])
        case["rows"] = max(500, min(case["rows"], (1 << 30) // (case["mean"] * case["k"])))
    elif op == "spmvop":
        case["alpha"], case["beta"] = -1.0, 1.0
        case["alg"] = 2 if case["pattern"] == "zipf" else rng.choice([1, 2])
        case["offsets"] = rng.choice(["i32", "i64"])
    return case


# ---------------------------------------------------------------- matrices

def row_lengths(case):
    """Entries of every row, by quantile: the same multiset with every seed."""
    rows, mean = case["rows"], case["mean"]
    at = (np.arange(rows, dtype=np.float64) + 0.5) / rows
    if case["pattern"] == "fixed":
        return np.full(rows, min(mean, case["cols"]), dtype=np.int64)
    if case["pattern"] == "ragged":  # uniform on 0 .. 2 * mean: empty rows among them
        return np.minimum(np.floor(at * (2 * mean + 1)), case["cols"] // 4).astype(np.int64)
    k = np.arange(1, case["cap"] + 1, dtype=np.float64)  # zipf: P(k) ~ k^-slope, scaled to the mean, cut at the cap
    weight = k ** -case["slope"]
    mass = weight.sum()
    scale = mean * mass / (k * weight).sum()
    drawn = np.searchsorted(np.cumsum(weight) / mass, at, side="left") + 1
    return np.clip(np.floor(scale * drawn), 1, case["cap"]).astype(np.int64)


def extent(case):
    """(rows, cols, entries)"""
    if case["pattern"] == "stencil":
        g = case["grid"]
        return g ** 3, g ** 3, (3 * g - 2) ** 3
    return case["rows"], case["cols"], int(row_lengths(case).sum())


def stencil_structure(grid, device):
    node = torch.arange(grid, device=device)
    step = torch.tensor([-1, 0, 1], device=device)
    near = node[:, None] + step                                        # [grid, 3]
    inside = (near >= 0) & (near < grid)
    cols = (near[:, None, None, :, None, None] * grid + near[None, :, None, None, :, None]) * grid \
        + near[None, None, :, None, None, :]                           # [z, y, x, dz, dy, dx]
    valid = (inside[:, None, None, :, None, None] & inside[None, :, None, None, :, None]
             & inside[None, None, :, None, None, :])
    cols, valid = cols.reshape(-1, 27), valid.reshape(-1, 27)
    lengths = valid.sum(dim=1)
    centre = (cols == torch.arange(grid ** 3, device=device)[:, None])[valid]
    return lengths, cols[valid].to(torch.int32), centre


def columns_of(lengths, cols, gen):
    """Distinct columns for every row, uniform, ascending."""
    device = lengths.device
    start = torch.repeat_interleave(torch.arange(lengths.numel(), device=device), lengths) * cols
    key = start + torch.randint(cols, start.shape, generator=gen, device=device)
    while True:
        key = torch.sort(key).values
        again = torch.nonzero(key[1:] == key[:-1]).flatten() + 1
        if again.numel() == 0:
            return (key - start).to(torch.int32)
        key[again] = start[again] + torch.randint(cols, again.shape, generator=gen, device=device)


class Pattern:
    def __init__(self, case, gen):
        device = gen.device
        self.rows, self.cols, self.nnz = extent(case)
        self.centre = None
        if case["pattern"] == "stencil":
            self.lengths, self.col_ind, self.centre = stencil_structure(case["grid"], device)
        else:
            lengths = torch.from_numpy(row_lengths(case)).to(device)
            self.lengths = lengths[torch.randperm(self.rows, generator=gen, device=device)]
            self.col_ind = columns_of(self.lengths, self.cols, gen)
        self.row_ptr = torch.zeros(self.rows + 1, dtype=torch.int64, device=device)
        torch.cumsum(self.lengths, 0, out=self.row_ptr[1:])
        assert self.col_ind.numel() == self.nnz

    def row_of(self):
        return torch.repeat_interleave(torch.arange(self.rows, device=self.lengths.device), self.lengths)


def dense(shape, kind, gen):
    if kind == "i32":
        return torch.randint(-100, 101, shape, generator=gen, device=gen.device, dtype=torch.int32)
    if kind == "i8":
        return torch.randint(-127, 128, shape, generator=gen, device=gen.device, dtype=torch.int8)
    return torch.randn(shape, generator=gen, device=gen.device, dtype=torch.float32).to(DTYPE[kind])


def matrix_values(case, pattern, gen):
    if pattern.centre is not None and case["value"] != "i32":  # Laplacian: 26 against -1, jittered
        jitter = (torch.rand(pattern.nnz, generator=gen, device=gen.device) - 0.5) * 0.02
        return (torch.where(pattern.centre, 26.0, -1.0) + jitter).to(DTYPE[case["value"]])
    if case["op"] == "spmm" and case["value"] == "bf16" and pattern.rows == pattern.cols:  # normalised adjacency
        root = pattern.lengths.to(torch.float32).clamp_min(1).rsqrt()
        return (root[pattern.row_of()] * root[pattern.col_ind]).to(torch.bfloat16)
    return dense((pattern.nnz,), case["value"], gen)


# ---------------------------------------------------------------- states

def pointer(t):
    return ctypes.c_void_p(t.data_ptr())


def prepare_product(case, gen, pkg):
    from ops_sparse_b200 import api
    p = Pattern(case, gen)
    s = {"handle": api.Handle()}
    s["A"] = api.CsrMatrix(p.row_ptr.to(torch.int32), p.col_ind, matrix_values(case, p, gen), p.rows, p.cols)
    s["alpha"], s["beta"] = case["alpha"], case["beta"]
    if case["value"] in ("i32", "i8"):
        s["alpha"], s["beta"] = int(s["alpha"]), int(s["beta"])
    if case["op"] == "spmm":
        k, m, n = p.cols, p.rows, case["n"]
        row = case["order"] == "row"
        B = dense((k, n) if row else (n, k), case["value"], gen)
        C = dense((m, n) if row else (n, m), case["out"], gen)
        s["B"] = api.DnMat(B, k, n, n if row else k, case["order"])
        s["out"] = api.DnMat(C, m, n, n if row else m, case["order"])
        s["alg"] = pkg.ACL_SPARSE_SPMM_CSR_FP32_HIGH_PRECISION_ALG if case["kahan"] else pkg.ACL_SPARSE_SPMM_ALG_DEFAULT
        s["buffer"] = api.spmm_preprocess(s["handle"], s["A"], s["B"], s["out"], alg=s["alg"])
        return s
    turned = case["op"] == "spmv_t"
    s["op"] = pkg.ACL_SPARSE_OP_TRANSPOSE if turned else pkg.ACL_SPARSE_OP_NON_TRANSPOSE
    s["x"] = api.DnVec(dense((p.rows if turned else p.cols,), case["value"], gen))
    s["out"] = api.DnVec(dense((p.cols if turned else p.rows,), case["out"], gen))
    s["buffer"] = None
    if turned or case["plan"]:
        s["buffer"] = api.spmv_preprocess(s["handle"], s["A"], s["x"], s["out"], s["op"])
    if case.get("device_scalars"):
        s["handle"].set_pointer_mode_device(True)
        s["alpha"] = torch.tensor(s["alpha"], dtype=torch.float32, device=gen.device)
        s["beta"] = torch.tensor(s["beta"], dtype=torch.float32, device=gen.device)
    return s


def prepare_sddmm(case, gen, pkg):
    from ops_sparse_b200 import api
    p = Pattern(case, gen)
    k, kind, half = case["k"], case["value"], case["value"] == "f16"
    s = {"handle": api.Handle()}
    s["X"] = api.DnMat.row_major(dense((p.rows, k), kind, gen))
    s["Y"] = api.DnMat.row_major(dense((p.cols, k), kind, gen))  # one row per node: op(Y) is its transpose
    s["C"] = api.CsrMatrix(p.row_ptr.to(torch.int32), p.col_ind, dense((p.nnz,), kind, gen), p.rows, p.cols)
    word = (lambda v: ctypes.c_uint16(int(np.float16(v).view(np.uint16)))) if half else ctypes.c_float
    s["keep"] = word(case["alpha"]), word(case["beta"])
    a, b = (ctypes.c_void_p(ctypes.addressof(w)) for w in s["keep"])
    s["args"] = (s["handle"].raw, pkg.ACL_SPARSE_OP_NON_TRANSPOSE, pkg.ACL_SPARSE_OP_TRANSPOSE, a, s["X"].raw,
                 s["Y"].raw, b, s["C"].raw, pkg.ACL_FLOAT16 if half else pkg.ACL_FLOAT, 0)
    size = ctypes.c_size_t()
    pkg.check(pkg.lib().aclsparseSDDMMBufferSize(*s["args"], ctypes.byref(size)), "aclsparseSDDMMBufferSize")
    s["buffer"] = torch.empty(size.value, dtype=torch.uint8, device=gen.device)
    s["args"] += (pointer(s["buffer"]),)
    pkg.check(pkg.lib().aclsparseSDDMMPreprocess(*s["args"]), "aclsparseSDDMMPreprocess")
    return s


def prepare_assemble(case, gen, pkg):
    from ops_sparse_b200 import api
    L = pkg.lib()
    p = Pattern(case, gen)
    device, m, n, nnz = gen.device, p.rows, p.cols, p.nnz
    row_of = p.row_of()
    shuffled = torch.sort(row_of * (1 << 24) + torch.randint(1 << 24, (nnz,), generator=gen, device=device)).indices
    whole = dict(dtype=torch.int32, device=device)
    s = {"handle": api.Handle(), "m": m, "n": n, "nnz": nnz, "coo_row": row_of.to(torch.int32),
         "coo_col": p.col_ind[shuffled].contiguous(), "first": torch.arange(nnz, **whole),
         "row_ptr": torch.empty(m + 1, **whole), "col_ind": torch.empty(nnz, **whole), "map": torch.empty(nnz, **whole),
         "csc_ptr": torch.empty(n + 1, **whole), "csc_row": torch.empty(nnz, **whole),
         "csc_map": torch.empty(nnz, **whole)}
    s["descr"] = ctypes.c_void_p()
    pkg.check(L.aclsparseCreateMatDescr(ctypes.byref(s["descr"])), "aclsparseCreateMatDescr")
    size = ctypes.c_size_t()
    h = s["handle"].raw
    pkg.check(L.aclsparseXcsrsort_bufferSizeExt(h, m, n, nnz, pointer(s["row_ptr"]), pointer(s["col_ind"]),
                                                ctypes.byref(size)), "aclsparseXcsrsort_bufferSizeExt")
    s["sort_buffer"] = torch.empty(size.value, dtype=torch.uint8, device=device)
    # the map travels as the 4-byte values of the conversion
    s["convert_args"] = (h, m, n, nnz, pointer(s["map"]), pointer(s["row_ptr"]), pointer(s["col_ind"]),
                         pointer(s["csc_map"]), pointer(s["csc_ptr"]), pointer(s["csc_row"]), pkg.ACL_FLOAT, 1, 0, 0)
    pkg.check(L.aclsparseCsr2cscEx2_bufferSize(*s["convert_args"], ctypes.byref(size)), "aclsparseCsr2cscEx2_bufferSize")
    s["convert_buffer"] = torch.empty(size.value, dtype=torch.uint8, device=device)
    return s


def prepare_spmvop(case, gen, pkg):
    from ops_sparse_b200 import api
    p = Pattern(case, gen)
    offsets = p.row_ptr if case["offsets"] == "i64" else p.row_ptr.to(torch.int32)
    s = {"handle": api.Handle(), "alpha": case["alpha"], "beta": case["beta"]}
    s["A"] = api.CsrMatrix(offsets, p.col_ind, dense((p.nnz,), "f32", gen), p.rows, p.cols)
    s["x"], s["y"], s["out"] = (api.DnVec(dense((size,), "f32", gen)) for size in (p.cols, p.rows, p.rows))
    s["plan"] = api.SpMVOpPlan(s["handle"], s["A"], s["x"], s["y"], s["out"], alg=case["alg"])
    return s


def prepare(case, seed):
    pkg = package()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    make = {"sddmm": prepare_sddmm, "assemble": prepare_assemble, "spmvop": prepare_spmvop}
    state = make.get(case["op"], prepare_product)(case, gen, pkg)
    state["kind"] = case["op"]
    return state


# ---------------------------------------------------------------- one pass

def run(s):
    pkg = package()
    from ops_sparse_b200 import api
    kind = s["kind"]
    if kind in ("spmv", "spmv_t"):
        api.spmv(s["handle"], s["A"], s["x"], s["out"], s["alpha"], s["beta"], op=s["op"], buffer=s["buffer"])
        return s["out"].values
    if kind == "spmm":
        api.spmm(s["handle"], s["A"], s["B"], s["out"], s["alpha"], s["beta"], alg=s["alg"], buffer=s["buffer"])
        return s["out"].values
    if kind == "spmvop":
        s["plan"].run(s["x"], s["y"], s["out"], s["alpha"], s["beta"])
        return s["out"].values
    L = pkg.lib()
    if kind == "sddmm":
        pkg.check(L.aclsparseSDDMM(*s["args"]), "aclsparseSDDMM")
        return s["C"].values
    h = s["handle"].raw
    pkg.check(L.aclsparseXcoo2csr(h, pointer(s["coo_row"]), s["nnz"], s["m"], pointer(s["row_ptr"]), 0),
              "aclsparseXcoo2csr")
    s["col_ind"].copy_(s["coo_col"])  # the sort works in place, on the columns and on the map
    s["map"].copy_(s["first"])
    pkg.check(L.aclsparseXcsrsort(h, s["m"], s["n"], s["nnz"], s["descr"], pointer(s["row_ptr"]), pointer(s["col_ind"]),
                                  pointer(s["map"]), pointer(s["sort_buffer"])), "aclsparseXcsrsort")
    pkg.check(L.aclsparseCsr2cscEx2(*s["convert_args"], pointer(s["convert_buffer"])), "aclsparseCsr2cscEx2")
    return [s[key] for key in ("row_ptr", "col_ind", "map", "csc_ptr", "csc_row", "csc_map")]


# ---------------------------------------------------------------- what a pass needs, and how exact it is

def work(case):
    rows, cols, nnz = extent(case)
    op = case["op"]
    if op == "assemble":  # COO rows and columns and the first map in; offsets, columns, map, and the same of the CSC out
        return {"bytes": 12 * nnz + 4 * (rows + 1) + 8 * nnz + 4 * (cols + 1) + 8 * nnz, "flops": 0}
    if op == "spmvop":
        offset = 8 if case["offsets"] == "i64" else 4
        return {"bytes": offset * (rows + 1) + 8 * nnz + 4 * cols + 8 * rows, "flops": 2 * nnz}
    reads_out = 2 if case["beta"] != 0 else 1
    value = BYTES[case["value"]]
    if op == "sddmm":
        return {"bytes": value * case["k"] * (rows + cols) + 4 * (rows + 1) + 4 * nnz + value * nnz * reads_out,
                "flops": 2 * nnz * case["k"]}
    wide = case["n"] if op == "spmm" else 1
    dense_in, dense_out = (rows, cols) if op == "spmv_t" else (cols, rows)
    return {"bytes": 4 * (rows + 1) + (4 + value) * nnz + value * dense_in * wide
            + BYTES[case["out"]] * dense_out * wide * reads_out, "flops": 2 * nnz * wide}


def tolerance(case):
    if case["op"] == "assemble" or case.get("value") in ("i32", "i8"):
        return "exact"
    if case["op"] == "spmvop":  # compensated sums, one rounding of the result
        return {"rel": 1e-6}
    out = case["value"] if case["op"] == "sddmm" else case["out"]
    # 16-bit results: sums in fp32, one rounding to 11 or 8 bits that may fall the other way
    return {"rel": {"f32": 1e-5, "f16": 1e-3, "bf16": 8e-3}[out]}
