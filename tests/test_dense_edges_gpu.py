"""The dense-block kernel where its rounds end: rows of 1 to 14 blocks (rounds of 4
and 6), blocks against the last columns, and rows long enough for several lanes
and for chunks."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import Csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("blocks", [1, 3, 4, 5, 6, 7, 12, 13, 14, 150, 1100])
def test_dense_rounds(built, blocks, dtype):
    from oracle import oracle as O
    from vnec_gb300 import api

    rng = np.random.default_rng(blocks)
    n_rows, n_cols = 70, 4 * blocks + 5
    cols = [np.unique(np.concatenate([(4 * np.arange(blocks))[:, None] + rng.integers(0, 4, (blocks, 2)) + r % 2,
                                      [[n_cols - 1, n_cols - 2 - r % 3]]]).ravel()) for r in range(n_rows)]
    rp = np.concatenate([[0], np.cumsum([c.size for c in cols])])
    m = Csr(n_rows, n_cols, rp, np.concatenate(cols), rng.uniform(-1, 1, int(rp[-1])).astype(dtype))
    x = rng.uniform(-1, 1, n_cols).astype(dtype)
    p = api.Plan(m, dtype=dtype, kernel=api.KERNEL_D)
    y = p.mxv_host(x)
    p.free()
    m64 = Csr(n_rows, n_cols, rp, m.col, m.val.astype(np.float64))
    y_ref, cond = O.spmv_neumaier(m64, x.astype(np.float64))
    # The parity bounds; a row has at most 4,500 products over 32 lanes and chunks.
    assert np.all(np.abs(y.astype(np.float64) - y_ref) <= (1e-12 if dtype == np.float64 else 1e-4) * cond)


@pytest.mark.parametrize("dtype", [np.float64, np.float32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("blocks", [1, 2, 3, 9, 10, 11, 12])
def test_short_and_long_tasks(built, blocks, dtype):
    """One lane per row and tasks of up to `blocks` steps, on both sides of the
    limit (10) between the two numbers of blocks in flight, rows of different length
    in a task; the same bits as rows of the same matrix whose plan also has a longer
    task."""
    from oracle import oracle as O
    from vnec_gb300 import api

    rng = np.random.default_rng(blocks)
    n_cols, n_rows = 200, 100
    cols = [np.arange(4 * max(blocks - r % 3, 1)) + r % 7 for r in range(n_rows)] + [np.arange(160)]
    rp = np.concatenate([[0], np.cumsum([c.size for c in cols])])
    val = rng.uniform(-1, 1, int(rp[-1])).astype(dtype)
    x = rng.uniform(-1, 1, n_cols).astype(dtype)
    ys = []
    for n in (n_rows, n_rows + 1):
        m = Csr(n, n_cols, rp[:n + 1], np.concatenate(cols[:n]), val[:rp[n]])
        p = api.Plan(m, dtype=dtype, kernel=api.KERNEL_D, max_steps=64)
        ys.append(p.mxv_host(x))
        p.free()
        m64 = Csr(n, n_cols, rp[:n + 1], m.col, m.val.astype(np.float64))
        y_ref, cond = O.spmv_neumaier(m64, x.astype(np.float64))
        # The parity bounds; a row has at most 160 products.
        assert np.all(np.abs(ys[-1].astype(np.float64) - y_ref) <= (1e-12 if dtype == np.float64 else 1e-4) * cond)
    assert ys[0].tobytes() == ys[1][:n_rows].tobytes()
