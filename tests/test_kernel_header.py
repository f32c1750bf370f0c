"""CPU: programs built against include/b200sp_kernels.h keep working when the library is replaced: the arguments of its functions
and the members of its structs only grow by new functions and new structs."""
from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

SOURCE = r"""
#include <stddef.h>
#include "b200sp_kernels.h"
_Static_assert(sizeof(b200spSpmmShape) == 88, "size");
_Static_assert(offsetof(b200spSpmmShape, order_b) == 48 && offsetof(b200spSpmmShape, kahan) == 60, "layout");
_Static_assert(offsetof(b200spSpmmShape, block_units) == 64 && offsetof(b200spSpmmShape, long_rows) == 68, "layout");
_Static_assert(offsetof(b200spSpmmShape, repack_bytes) == 72 && offsetof(b200spSpmmShape, mid_units) == 80, "layout");
size_t (*plan_bytes)(int64_t, int64_t, int64_t) = b200sp_spmm_plan_bytes;
size_t (*repack_bytes)(const b200spSpmmShape *, int) = b200sp_spmm_repack_bytes;
int (*copies)(const b200spSpmmShape *, int, int32_t, const void *) = b200sp_spmm_copies;
int (*units)(const int32_t *, int64_t, int64_t, int64_t, void *, size_t, int32_t *, int32_t *, void *) = b200sp_spmm_analyze_units;
int (*analyze)(const int32_t *, int64_t, int64_t, int64_t, void *, size_t, int32_t *, void *) = b200sp_spmm_analyze;
int (*blocks)(const int32_t *, const int32_t *, int64_t, int64_t, int64_t, int64_t, int64_t, void *, size_t, int32_t *, int32_t *,
              void *) = b200sp_spmm_analyze_blocks;
int (*launch)(const int32_t *, const int32_t *, const void *, const void *, void *, const b200spSpmmShape *, const b200spScalars *, int, int,
              void *, int32_t, void *) = b200sp_spmm_launch;
"""


def test_spmm_declarations(tmp_path):
    source = tmp_path / "caller.c"
    source.write_text(SOURCE)
    built = subprocess.run(["gcc", "-std=c11", "-Wall", "-Werror", "-I", str(ROOT / "include"), "-c", str(source), "-o", str(tmp_path / "caller.o")],
                           capture_output=True, text=True)
    assert built.returncode == 0, built.stderr
