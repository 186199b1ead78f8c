"""Warps in flight of the batch kernels, layout by layout.

The kernels are bound by the latency of the X gathers, so a build whose
registers leave 8 or 16 of an SM's 64 warps runs up to 2.8 times slower than one
with fewer loads in flight per lane and more warps.  The bound per layout is
what its steps in flight leave it (at most 80 registers with up to four
right-hand sides per lane, at most 128 with eight)."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["FP32", "DF32"])
@pytest.mark.parametrize("rhs_per_lane", [1, 2, 4, 8])
@pytest.mark.parametrize("unroll", [1, 2])
def test_warps_per_sm(built, precision, rhs_per_lane, unroll):
    import torch

    from vnec_gb300 import api
    from vnec_gb300 import generators as G

    mats = [G.uniform_k(200, 5, seed=s) for s in (1, 2)]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for warps in (4, 8):
        p = api.BatchPlan(mats, 8, precision=getattr(api, f"PREC_{precision}"), lanes=8 // rhs_per_lane,
                          unroll=unroll, warps_per_block=warps)
        assert p.info().blocks * warps // sms >= (16 if rhs_per_lane == 8 else 24), (warps, p.info().blocks)
        p.free()
