"""Shared-pattern tasks in every kernel that reads them: rows of 1 to 32 entries
with the same gaps (rounds of 4, 8, 12 and 16 steps and their remainders), all
value types and forms, the fused epilogue, and y bit for bit as without them."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import Csr

pytestmark = pytest.mark.gpu


def _pattern(width, dtype, n=700):
    """Interior rows share `width` gaps; the first and last rows are cut off."""
    rng = np.random.default_rng(width)
    gaps = np.sort(rng.choice(np.arange(-60, 60), size=width, replace=False))
    rows = [np.unique(c[(c >= 0) & (c < n)]) for c in (r + gaps for r in range(n))]
    rp = np.concatenate([[0], np.cumsum([c.size for c in rows])])
    return Csr(n, n, rp, np.concatenate(rows), rng.uniform(-1, 1, int(rp[-1])).astype(dtype)), \
        rng.uniform(-1, 1, n).astype(dtype)


@pytest.mark.parametrize("form", ["fp64", "fp32 type", "fp32", "bf16", "df32"])
@pytest.mark.parametrize("width", [1, 3, 4, 5, 8, 9, 12, 15, 16, 17, 31, 32])
def test_shared_steps(built, width, form):
    import torch

    from oracle import oracle as O
    from vnec_gb300 import api

    dtype = np.float32 if form == "fp32 type" else np.float64
    prec = {"fp32": api.PREC_FP32, "bf16": api.PREC_BF16, "df32": api.PREC_DF32}.get(form, api.PREC_FP64)
    tol = {"fp64": 1e-12, "fp32 type": 1e-4, "fp32": 1e-6, "bf16": 1e-2, "df32": 1e-12}[form]  # the forms' parity bounds
    m, x = _pattern(width, dtype)
    y_ref, cond = O.spmv_neumaier(Csr(m.n_rows, m.n_cols, m.row_ptr, m.col, m.val.astype(np.float64)),
                                  x.astype(np.float64))
    xd = torch.from_numpy(x).cuda()
    for unroll in (4, 8, 12, 16):
        for lanes in (0, -1, 1):
            got = []
            for shared in (1, -1):
                p = api.Plan(m, dtype=dtype, kernel=api.KERNEL_S, precision=prec, items_per_thread=unroll, max_steps=32,
                             shared_patterns=shared, lane_vectors=lanes)
                z = torch.from_numpy(x[::-1].copy()).cuda()
                p.mxv_axpby(xd.data_ptr(), z.data_ptr(), alpha=0.5, beta=-2.0, d_z=z.data_ptr(), gamma=0.25)
                torch.cuda.synchronize()
                got.append((p.mxv_host(x), z.cpu().numpy(), p.info().algorithmic_bytes))
                p.free()
            assert got[0][0].tobytes() == got[1][0].tobytes() and got[0][1].tobytes() == got[1][1].tobytes()
            assert got[0][2] < got[1][2]
            assert np.all(np.abs(got[0][0].astype(np.float64) - y_ref) <= tol * cond)


@pytest.mark.parametrize("form,least", [("fp64", 14), ("fp32 type", 4), ("fp32", 2)])
def test_default_rule(built, form, least):
    """By default plain plans share patterns from 14 (FP64) or 4 (FP32 type) steps
    on, the precision forms at every length; the bits are those of all and of none."""
    from vnec_gb300 import api

    dtype = np.float32 if form == "fp32 type" else np.float64
    for width in (2, 3, 4, 5, 13, 14, 15):
        m, x = _pattern(width, dtype)
        got = {}
        for shared in (-1, 0, 1):
            p = api.Plan(m, dtype=dtype, kernel=api.KERNEL_S, precision=api.PREC_FP32 if form == "fp32" else api.PREC_FP64,
                         max_steps=32, shared_patterns=shared, column_deltas=0)
            got[shared] = (p.mxv_host(x).tobytes(), p.info().algorithmic_bytes)
            p.free()
        assert got[-1][0] == got[0][0] == got[1][0]
        assert got[0][1] == got[1 if width >= least else -1][1] and got[1][1] < got[-1][1]
