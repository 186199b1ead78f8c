"""The batch autotuner: what a plan takes untuned is among its candidates."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,k,long_len", [("FP64", 8, 512), ("DF32", 16, 256), ("FP32", 8, 1024)])
def test_untuned_layout_is_a_candidate(built, precision, k, long_len):
    """On a batch between 2^22 and 2^25 nonzeros."""
    from vnec_gb300 import api
    from vnec_gb300 import generators as G

    mats = [G.uniform_k(120_000 + i, 20, seed=60 + i) for i in range(2)]
    prec = getattr(api, f"PREC_{precision}")
    plain = api.BatchPlan(mats, k, precision=prec)
    tuned = api.BatchPlan(mats, k, precision=prec, autotune=True)
    inf = plain.info()
    assert inf.long_row_len == long_len
    cand, ms, best = tuned.tuning()
    assert (inf.lanes, long_len, inf.threads_per_block // 32, 0) in cand
    assert tuned.info().lanes == cand[best][0] and tuned.info().long_row_len == cand[best][1]
    x = np.random.default_rng(5).uniform(-1, 1, k * sum(m.n_cols for m in mats))
    a, b = plain.mxv_host(x), tuned.mxv_host(x)
    tol = 2e-6 if precision == "FP32" else 1e-12
    assert np.abs(a - b).max() <= tol * np.abs(a).max()
    plain.free()
    tuned.free()
