"""SpMSpV on both sides of the lines between its two kernels: a warp per column
(plans whose longest column has at most 512 entries) and shared chunks."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import Csr

pytestmark = pytest.mark.gpu


def _matrix(n_rows, lens, seed, dtype):
    rng = np.random.default_rng(seed)
    col = np.repeat(np.arange(lens.size), lens)
    row = rng.integers(0, n_rows, col.size)
    key = np.unique(row.astype(np.int64) * lens.size + col)
    row, col = key // lens.size, key % lens.size
    rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n_rows))])
    return Csr(n_rows, lens.size, rp, col, rng.uniform(-1, 1, col.size).astype(dtype))


CASES = [("nine", nx) for nx in (1, 255, 256, 16384, 16385, 131072, 131073, 140000)] + \
        [("one", nx) for nx in (255, 16384, 16385, 20000)] + \
        [("512", nx) for nx in (255, 256, 600)] + [("513", nx) for nx in (255, 256, 600)]


@pytest.mark.parametrize("dtype", [np.float64, np.float32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("kind,nx", CASES)
def test_spmspv_of_short_columns(built, kind, nx, dtype):
    from oracle import oracle as O
    from vnec_gb300 import api

    rng = np.random.default_rng(nx)
    if kind == "nine":
        lens = rng.integers(8, 11, 140000)
    elif kind == "one":
        lens = rng.integers(0, 3, 20000)
    else:
        lens = np.full(600, int(kind))
    if kind in ("512", "513"):  # each row at most once a column, so that the columns keep their length
        n_rows = 4000
        row = np.concatenate([rng.choice(n_rows, k, replace=False) for k in lens])
        col = np.repeat(np.arange(lens.size), lens)
        order = np.lexsort((col, row))
        rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n_rows))])
        m = Csr(n_rows, lens.size, rp, col[order], rng.uniform(-1, 1, order.size).astype(dtype))
    else:
        m = _matrix(3000, lens, 5, dtype)
    idx = rng.choice(m.n_cols, nx, replace=False).astype(np.int32)
    xv = rng.uniform(-1, 1, nx).astype(dtype)
    xv[:: 7] = 0
    dense = np.zeros(m.n_cols)
    dense[idx] = xv
    m64 = Csr(m.n_rows, m.n_cols, m.row_ptr, m.col, m.val.astype(np.float64))
    y_ref, cond = O.spmv_neumaier(m64, dense)
    # A row has fewer than 700 additions: 7.8e-14 of its condition in FP64, 4.2e-5 in FP32.
    assert np.diff(m.row_ptr).max() < 700
    tol = 1e-13 if dtype == np.float64 else 5e-5
    p = api.Plan(m, dtype=dtype, kernel=api.KERNEL_PUSH)
    y = p.spmspv_host(idx, xv)
    assert np.all(np.abs(y.astype(np.float64) - y_ref) <= tol * cond)
    if nx > 1:
        bad = idx.copy()
        bad[nx // 2] = m.n_cols if nx % 2 else -1
        with pytest.raises(api.VnecError, match="outside"):
            p.spmspv_host(bad, xv)
        skipped = np.zeros(m.n_cols)
        skipped[np.delete(idx, nx // 2)] = np.delete(xv, nx // 2)
        y_ref, cond = O.spmv_neumaier(m64, skipped)
        import torch

        d = torch.from_numpy(bad).cuda(), torch.from_numpy(xv).cuda()
        out = torch.full((m.n_rows,), 9.0, dtype=d[1].dtype, device="cuda")
        p.spmspv_device(nx, d[0].data_ptr(), d[1].data_ptr(), out.data_ptr(), 0)
        torch.cuda.synchronize()
        assert np.all(np.abs(out.cpu().numpy().astype(np.float64) - y_ref) <= tol * cond)
        with pytest.raises(api.VnecError, match="outside"):
            p.device_status()
    p.free()
