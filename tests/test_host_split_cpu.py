"""Host-vector calls of plans built with host_parts run the SpMV in that many
parts, others in one, or four where y is page-locked and long: counted by the launches of the library's own host code
with the runtime calls faked (tests/fake_cudart.c)."""
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
from vnec_gb300 import api, generators as G
m = G.uniform_k(50_000, 3, seed=1)
for parts in (0, 1, 3, 8):
    p = api.Plan(m, kernel=api.KERNEL_S, items_per_thread=8, window_rows=1000, host_parts=parts)
    print("parts", parts, flush=True)
    p.mxv_host(np.ones(m.n_cols))
    p.free()
"""


LONG = """
import numpy as np, sys
sys.path.insert(0, {root!r})
from vnec_gb300 import api, generators as G
for dtype, mb in ((np.float64, 9), (np.float64, 11), (np.float32, 6), (np.float32, 8)):
    m = G.uniform_k((mb << 20) // np.dtype(dtype).itemsize, 1, seed=1)
    p = api.Plan(m, kernel=api.KERNEL_S, dtype=dtype, items_per_thread=8, hot_columns=-1)
    print("parts", np.dtype(dtype).name, mb, flush=True)
    p.mxv_host(np.ones(m.n_cols, dtype))
    p.free()
"""


def _launches(program, tmp_path, **env):
    so = tmp_path / "fake_cudart.so"
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-I", os.path.join(home, "include"),
                    os.path.join(ROOT, "tests", "fake_cudart.c"), "-o", str(so)], check=True)
    r = subprocess.run([sys.executable, "-c", program.format(root=ROOT)], capture_output=True, text=True,
                       env=dict(os.environ, LD_PRELOAD=str(so), CUDA_VISIBLE_DEVICES="", **env), timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    launches = {}
    for ln in r.stdout.splitlines():
        if ln.startswith("parts"):
            parts = " ".join(ln.split()[1:])
            launches[parts] = 0
        elif ln.startswith("y "):
            launches[parts] += 1
    return launches


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
def test_parts_of_a_host_call(built, tmp_path):
    assert _launches(PROGRAM, tmp_path) == {"0": 1, "1": 1, "3": 3, "8": 8}


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
def test_parts_by_the_length_of_y(built, tmp_path):
    assert _launches(LONG, tmp_path) == {"float64 9": 1, "float64 11": 1, "float32 6": 1, "float32 8": 1}
    assert _launches(LONG, tmp_path, FAKE_LOCKED="1") == {"float64 9": 1, "float64 11": 4, "float32 6": 1,
                                                          "float32 8": 4}
