"""Which loads the chained kernels may take from the read-only path.

A chained kernel (launch.cuh) is resident while the kernel before it on the
stream still writes: x, converted x, chunk sums, carries and partial sums change
in its lifetime.  `__ldg`, `ld.global.nc` and `const __restrict__` promise data
that nobody writes while the kernel runs, and let the compiler move a load
across the wait, so in these files they are for arrays of the plan alone."""
from __future__ import annotations

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "vnec_gb300", "csrc")

# Arrays that are in place before a plan is handed out.
PLAN_ARRAYS = {"tasks", "val", "col", "rowid", "col16", "first", "pat16", "row_scale", "chunk_scale", "hot", "hot_cols",
               "long_row", "long_first", "long_heavy", "chunk_long", "row_end", "tile_row", "tile_nz"}
# Helpers that load from the read-only path, and what they are called on.
NC_HELPERS = {"ld_once", "ld_na", "load_items"}
NC_ARGUMENTS = {"cp", "vp", "p"}


def _source(name: str) -> str:
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


FILES = ["sliced_kernels.cu", "sliced_mixed.cu", "batch_kernels.cu", "mp_kernels.cu", "vector_ops.cu", "long_rows.cuh"]


@pytest.mark.parametrize("name", FILES)
def test_files_launch_chained_kernels(name):
    text = _source(name)
    assert name.endswith(".cuh") or "launch_chained(" in text


@pytest.mark.parametrize("name", FILES)
def test_ldg_reads_plan_arrays_only(name):
    for arg in re.findall(r"__ldg\(([^;]*)", _source(name)):
        base = re.match(r"(?:reinterpret_cast<[^>]*>\()?\(?(?:a\.)?(\w+)", arg).group(1)
        assert base in PLAN_ARRAYS, f"{name}: __ldg({arg}"


@pytest.mark.parametrize("name", FILES)
def test_restrict_is_for_plan_arrays_only(name):
    for arg in re.findall(r"__restrict__\s+(\w+)", _source(name)):
        assert arg in PLAN_ARRAYS, f"{name}: __restrict__ {arg}"


@pytest.mark.parametrize("name", FILES)
def test_nc_loads_stay_in_the_helpers_for_plan_arrays(name):
    text = _source(name)
    for m in re.finditer(r"ld\.global\.nc", text):
        head = re.findall(r"__device__ __forceinline__ [^\n{;]*?(\w+)\([^\n]*\{", text[:m.start()])[-1]
        assert head in NC_HELPERS, f"{name}: ld.global.nc in {head}"
    for helper, arg in re.findall(r"\b(ld_once|ld_na|load_items(?:<\w+>)?)\((\w+)[,)]", text):
        assert arg in NC_ARGUMENTS, f"{name}: {helper}({arg}"
