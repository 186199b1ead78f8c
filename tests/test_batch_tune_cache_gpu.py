"""Choices of the batch autotuner in the cache file: those timed on other kernels
are not taken."""
from __future__ import annotations

import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = """
import sys, json
sys.path.insert(0, {root!r})
from vnec_gb300 import api, generators as G
mats = [G.uniform_k(900 + i, 9, seed=i) for i in range(3)]
p = api.BatchPlan(mats, 8, precision=api.PREC_FP32, autotune=True)
i = p.info()
print(json.dumps([len(p.tuning()[0]), i.lanes, i.long_row_len, i.threads_per_block // 32]))
"""


def _run(cache):
    env = dict(os.environ, VNEC_TUNE_CACHE=str(cache))
    r = subprocess.run([sys.executable, "-c", PROGRAM.format(root=ROOT)], capture_output=True, text=True, env=env,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_cache_entries_of_other_kernels(built, tmp_path):
    cache = tmp_path / "tune.jsonl"
    assert _run(cache)[0] > 0
    entry = json.loads(cache.read_text().splitlines()[-1])

    def write(path, key):
        e = {**entry, "key": key, "lanes": 4, "long_row_len": 4096, "warps_per_block": 8, "deep_unroll": 0,
             "dispatch": 2}
        if "tasks_log2" in e:
            e["tasks_log2"] = 0
        path.write_text("{" + ", ".join(f'"{k}": {json.dumps(v)}' for k, v in e.items()) + "}\n")

    # An entry of the present version is taken, without timing.
    mine = tmp_path / "mine.jsonl"
    write(mine, entry["key"])
    assert _run(mine) == [0, 4, 4096, 8]
    # One without a version, or of another, is not.
    key = entry["key"].split("|", 1)
    assert key[0].startswith("v")
    for other in (key[1], "v0|" + key[1]):
        old = tmp_path / "old.jsonl"
        write(old, other)
        assert _run(old)[0] > 0
