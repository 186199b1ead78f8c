"""FP32 batches: the default layouts' kernels take several tasks per warp.

Every slot's sums are those of the same layout with one task per warp, which is
what a plan with its lanes given runs: the two agree bit for bit, through
unaligned x and y where the default layout takes them, and with the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from test_batch_gpu import TOL, check, oracle_batch, small_batch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def batch():
    return small_batch(seed=11, n=13)


@pytest.mark.parametrize("k", [2, 4, 8, 16, 32])
@pytest.mark.parametrize("dispatch", [1, 2])
@pytest.mark.parametrize("long_row_len", [0, 64])
def test_several_tasks_per_warp_same_bits(built, batch, k, dispatch, long_row_len):
    from vnec_gb300 import api

    kw = dict(precision=api.PREC_FP32, dispatch=dispatch, long_row_len=long_row_len)
    shared = api.BatchPlan(batch, k, **kw)
    lanes = shared.info().lanes
    single = api.BatchPlan(batch, k, lanes=lanes, **kw)
    ro, co = shared.offsets()
    X = np.random.default_rng(3).uniform(-1, 1, int(co[-1]) * k)
    Y = shared.mxv_host(X)
    assert Y.tobytes() == single.mxv_host(X).tobytes()
    Yref, cond = oracle_batch(batch, X, k, co, ro)
    check(Y, Yref, cond, TOL[1])
    if k <= 4:
        import torch

        x = torch.zeros(X.size + 1, dtype=torch.float64, device="cuda")
        y = torch.zeros(Y.size + 1, dtype=torch.float64, device="cuda")
        x[1:] = torch.from_numpy(X).cuda()
        torch.cuda.synchronize()
        shared.mxv_device(x.data_ptr() + 8, y.data_ptr() + 8, 0)
        torch.cuda.synchronize()
        assert y[1:].cpu().numpy().tobytes() == Y.tobytes()
    shared.free()
    single.free()
