"""Precision forms of small plans gather FP64 x and convert it on the way; larger
plans, and calls in place (x and y the same buffer), convert x first.  Both must
give the same bits on each side of the size rule (2^19 nonzeros), also for x
beyond FP32's range, and a DF32 call whose x leaves the split range must not
affect the next one."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import Csr

pytestmark = pytest.mark.gpu


def _square(nnz, kind, seed):
    """`nnz` entries, 16 a row or (last row) fewer: random columns, or a band."""
    rng = np.random.default_rng(seed)
    n = max(-(-nnz // 16), 40)
    lens = np.minimum(16, np.maximum(nnz - 16 * np.arange(n), 0))
    rp = np.concatenate([[0], np.cumsum(lens)])
    row = np.repeat(np.arange(n), lens)
    k = np.arange(nnz) - rp[row]
    if kind == "random":  # distinct ascending columns
        col = k * (n // 16) + rng.integers(0, n // 16, nnz)
    else:
        col = np.minimum(row, n - 32) + 2 * k
    return Csr(n, n, rp, col, rng.uniform(-1, 1, nnz)), rng


@pytest.mark.parametrize("form", ["fp32", "bf16", "df32"])
@pytest.mark.parametrize("kind", ["random", "band"])
@pytest.mark.parametrize("nnz", [17, 5000, (1 << 19) - 3, 1 << 19, (1 << 19) + 1])
def test_same_bits_as_converted_first(built, nnz, kind, form):
    import torch

    from vnec_gb300 import api

    prec = {"fp32": api.PREC_FP32, "bf16": api.PREC_BF16, "df32": api.PREC_DF32}[form]
    m, rng = _square(nnz, kind, nnz)
    n = m.n_cols
    plain = rng.uniform(-1, 1, n)
    plain[::7] = 0.0
    plain[3::11] = -0.0
    wide = plain.copy()
    wide[::5] = np.resize([1e-40, -3e-45, 5e-324, 3.5e38, -1e300, np.inf, 1 + 2.0**-24, 1 + 3 * 2.0**-24], wide[::5].size)
    nan = wide.copy()
    nan[1::13] = np.nan
    for lanes in (0, -1):
        p = api.Plan(m, kernel=api.KERNEL_S, precision=prec, lane_vectors=lanes, hot_columns=-1)
        # In place, a DF32 call whose x leaves the split range recomputes from an x it overwrites.
        vectors = (plain, plain * 2.0**30) if form == "df32" else (plain, wide, nan)
        for v in vectors:
            x = torch.from_numpy(v).cuda()
            y = torch.zeros(n, dtype=torch.float64, device="cuda")
            z = x.clone()
            p.mxv_device(x.data_ptr(), y.data_ptr())
            p.mxv_device(z.data_ptr(), z.data_ptr())
            torch.cuda.synchronize()
            assert y.cpu().numpy().tobytes() == z.cpu().numpy().tobytes()
        p.free()


@pytest.mark.parametrize("nnz", [5000, 1 << 19, (1 << 19) + 1])
@pytest.mark.parametrize("hot", [-1, 64])
def test_df32_flag_clears(built, nnz, hot):
    import torch

    from vnec_gb300 import api

    m, rng = _square(nnz, "random", nnz + 1)
    v = rng.uniform(0.5, 1, m.n_cols)
    bad = v.copy()
    bad[m.col[nnz // 2]] = 1e300
    p = api.Plan(m, kernel=api.KERNEL_S, precision=api.PREC_DF32, hot_columns=hot)
    f64 = api.Plan(m, kernel=api.KERNEL_S, hot_columns=hot)
    out = {}
    for name, w in (("good", v), ("bad", bad), ("good", v), ("bad", bad), ("bad", bad), ("good", v)):
        x = torch.from_numpy(w).cuda()
        y = torch.full((m.n_rows,), 7.0, dtype=torch.float64, device="cuda")
        r = torch.empty_like(y)
        p.mxv_device(x.data_ptr(), y.data_ptr())
        f64.mxv_device(x.data_ptr(), r.data_ptr())
        torch.cuda.synchronize()
        got = y.cpu().numpy()
        assert out.setdefault(name, got).tobytes() == got.tobytes()
        if name == "bad":
            # The recompute is FP64: 16 products a row, any order, 16 x 2^-53 of the sum of moduli each way.
            scale = np.add.reduceat(np.abs(m.val * bad[m.col]), m.row_ptr[:-1][np.diff(m.row_ptr) > 0])
            rows = np.flatnonzero(np.diff(m.row_ptr) > 0)
            assert np.all(np.abs(got[rows] - r.cpu().numpy()[rows]) <= 4e-15 * scale)
    p.free()
    f64.free()
