"""The device reduction at the edges of its rounds (pairs, four pairs a thread, one
block's 2,048 values, all 1,024 blocks), on vectors that are 16-byte aligned or
only 8-byte aligned, in both modes."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [0, 1, 2, 255, 2047, 2048, 2049, 524287, 2097152, 2097155, 4200001])
def test_dot_edges(built, n, mode):
    import torch

    from vnec_gb300 import api

    rng = np.random.default_rng(n)
    a, b = rng.uniform(-1, 1, n + 1), rng.uniform(-1, 1, n + 1)
    ad, bd = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    part = torch.empty(api.DOT_BLOCKS, dtype=torch.float64, device="cuda")
    out = torch.full((1,), float("nan"), dtype=torch.float64, device="cuda")
    for sa, sb in ((0, 0), (1, 1), (1, 0)):
        u, v = a[sa:sa + n], b[sb:sb + n]
        terms = u * v if mode == 0 else np.abs(u - v)
        bits = set()
        for _ in range(2):
            api.dot(n, ad.data_ptr() + 8 * sa, bd.data_ptr() + 8 * sb, mode, part.data_ptr(), out.data_ptr())
            torch.cuda.synchronize()
            bits.add(out.item())
        assert len(bits) == 1
        # Fewer than 60 additions to any term: 60 eps of the sum of sizes.
        assert abs(out.item() - math.fsum(terms)) <= 60 * 2.3e-16 * np.abs(terms).sum()
