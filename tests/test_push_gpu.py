"""SpMSpV at the edges of its chunks: 255 to 513 entries of x, hub columns that
many blocks share among columns of one entry, repeated and out-of-range
indices, zeros in x, and the dense-x call."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import Csr

pytestmark = pytest.mark.gpu


def _matrix(dtype):
    """A with columns of 0 to 3 entries and hubs of 6,000 at columns 0, 1 and 900."""
    rng = np.random.default_rng(7)
    n_rows, n_cols = 7000, 1500
    lens = rng.integers(0, 4, n_cols)
    lens[[0, 1, 900]] = 6000
    col = np.repeat(np.arange(n_cols), lens)
    row = np.concatenate([rng.choice(n_rows, size=k, replace=False) for k in lens])
    order = np.lexsort((col, row))
    rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n_rows))])
    return Csr(n_rows, n_cols, rp, col[order], rng.uniform(-1, 1, order.size).astype(dtype))


@pytest.mark.parametrize("dtype", [np.float64, np.float32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("nx", [1, 31, 255, 256, 257, 513, 1500])
def test_spmspv_chunks(built, nx, dtype):
    from oracle import oracle as O
    from vnec_gb300 import api

    m = _matrix(dtype)
    rng = np.random.default_rng(nx)
    idx = rng.integers(0, m.n_cols, nx).astype(np.int32)  # repeats add up
    idx[: min(nx, 3)] = [900, 0, 1][: min(nx, 3)]
    xv = rng.uniform(-1, 1, nx).astype(dtype)
    xv[nx // 2:nx // 2 + nx // 7] = 0
    dense = np.zeros(m.n_cols)
    np.add.at(dense, idx, xv.astype(np.float64))
    size = np.zeros(m.n_cols)
    np.add.at(size, idx, np.abs(xv.astype(np.float64)))
    m64 = Csr(m.n_rows, m.n_cols, m.row_ptr, m.col, m.val.astype(np.float64))
    y_ref = O.spmv_neumaier(m64, dense)[0]
    # Condition with repeats counted one by one; a row has fewer than 1,600
    # additions, 1.8e-13 of it in FP64 and 1e-4 in FP32.
    cond = O.spmv_neumaier(Csr(m.n_rows, m.n_cols, m.row_ptr, m.col, np.abs(m64.val)), size)[0]
    tol = 1e-12 if dtype == np.float64 else 1e-4
    p = api.Plan(m, dtype=dtype, kernel=api.KERNEL_PUSH)
    y = p.spmspv_host(idx, xv)
    assert np.all(np.abs(y.astype(np.float64) - y_ref) <= tol * cond)
    # An index out of range is skipped and reported; the other entries count.
    if nx > 3:
        bad = idx.copy()
        bad[3] = m.n_cols
        with pytest.raises(api.VnecError, match="outside"):
            p.spmspv_host(bad, xv)
    x = np.zeros(m.n_cols, dtype=dtype)
    x[idx] = xv
    y_ref, cond = O.spmv_neumaier(m64, x.astype(np.float64))
    assert np.all(np.abs(p.mxv_host(x).astype(np.float64) - y_ref) <= tol * cond)
    p.free()
