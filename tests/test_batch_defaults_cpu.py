"""Chunk length that a batch plan takes by default, over the size of the batch.

Short chunks pay in small batches, where a long one runs alone at the end, and
cost partial sums in large ones.  The plans are built by the library's own host
code with the runtime calls faked (tests/fake_cudart.c)."""
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
def matrix(nnz, width=64):
    m = M(); m.n_rows, m.n_cols, m.nnz = nnz // width, width, nnz // width * width
    m.row_ptr = np.arange(m.n_rows + 1, dtype=np.int64) * width
    m.col = np.tile(np.arange(width, dtype=np.int32), m.n_rows); m.val = np.ones(m.nnz)
    return m
cases = [(1 << 20, "FP64", 4), (1 << 20, "DF32", 16), (1 << 20, "FP32", 16), (1 << 22, "FP64", 4), (1 << 22, "DF32", 16),
         (1 << 25, "FP64", 16), (1 << 25, "DF32", 16)]
for nnz, form, k in cases:
    p = api.BatchPlan([matrix(nnz)], k, precision=getattr(api, "PREC_" + form), max_steps=32)
    print("plan", nnz, form, k, p.info().long_row_len, flush=True)
    p.free()
"""


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
def test_default_chunk_length(built, tmp_path):
    so = tmp_path / "fake_cudart.so"
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-I", os.path.join(home, "include"),
                    os.path.join(ROOT, "tests", "fake_cudart.c"), "-o", str(so)], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), CUDA_VISIBLE_DEVICES="")
    r = subprocess.run([sys.executable, "-c", PROGRAM.format(root=ROOT)], capture_output=True, text=True, env=env,
                       timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    got = {(int(n), f, int(k)): int(v) for _, n, f, k, v in (ln.split() for ln in r.stdout.splitlines()
                                                            if ln.startswith("plan"))}
    assert got == {(1 << 20, "FP64", 4): 256, (1 << 20, "DF32", 16): 256, (1 << 20, "FP32", 16): 1024,
                   (1 << 22, "FP64", 4): 512, (1 << 22, "DF32", 16): 256,
                   (1 << 25, "FP64", 16): 512, (1 << 25, "DF32", 16): 1024}
