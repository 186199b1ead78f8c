"""Host-vector calls where page-locked memory is not to be had.

A short y is written by the kernels to a page-locked buffer of the plan.  Where
that buffer cannot be allocated or mapped, the call goes by device memory and a
copy instead, as it did before there was such a buffer: it is not refused, no
kernel gets a null y, and nothing is left allocated.  Run on the library's own
host code with the runtime calls faked (tests/fake_cudart.c)."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

import pytest

from conftest import ROOT

PROGRAM = """
import numpy as np, sys
sys.path.insert(0, {root!r})
from vnec_gb300 import api
class M: pass
m = M(); m.n_rows = m.n_cols = 40
m.row_ptr = np.arange(41, dtype=np.int64); m.col = np.arange(40, dtype=np.int32); m.val = np.ones(40); m.nnz = 40
p = api.Plan(m, kernel=api.KERNEL_S, items_per_thread=8)
for _ in range(3):
    y = np.full(40, 7.0)
    p.mxv_host(np.ones(40), y)
    print("y", y.min(), y.max(), flush=True)  # the launches do nothing: zeros from a zeroed buffer
p.free()
print("done", flush=True)
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory, built):
    so = tmp_path_factory.mktemp("fake") / "fake_cudart.so"
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-I", os.path.join(home, "include"),
                    os.path.join(ROOT, "tests", "fake_cudart.c"), "-o", str(so)], check=True)
    return so


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
@pytest.mark.parametrize("fail,y,copies", [("", "mapped", 0), ("hostalloc", "device", 3), ("hostmap", "device", 3)])
def test_short_y_without_page_locked_memory(fake, fail, y, copies):
    env = dict(os.environ, LD_PRELOAD=str(fake), FAKE_FAIL=fail, CUDA_VISIBLE_DEVICES="")
    r = subprocess.run([sys.executable, "-c", PROGRAM.format(root=ROOT)], capture_output=True, text=True, env=env,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    lines = r.stdout.split("\n")
    assert "done" in lines
    assert [ln for ln in lines if ln.startswith("y ") and ln[2].isalpha()] == [f"y {y}"] * 3
    assert [ln for ln in lines if ln.startswith("y 0")] == ["y 0.0 0.0"] * 3
    assert lines.count("copy out 320") == copies
    freed = [ln for ln in lines if ln.startswith("live")]
    assert not freed or freed[-1] == "live 0"
    assert fail == "hostalloc" or freed
