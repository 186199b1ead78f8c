"""The merge-path tile kernel at the edges of its threads and tiles: rows that
end on, before and after a thread's 8 nonzeros and a tile of 896, 1,016 or 2,040 items, rows of
many threads and of many tiles, runs of empty rows, and caller arrays without
the 32-byte alignment that its vector loads use."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import Csr

pytestmark = pytest.mark.gpu

LENGTHS = {
    "one": [1] * 3000,
    "thread": [7, 8, 9, 15, 16, 17, 1] * 300,
    "walk": [31, 32, 33, 40, 41, 200, 3] * 60,  # rows of up to, and past, four threads
    "tile": [894, 895, 896, 897, 1, 888, 0, 7, 1014, 1015, 1016, 1017, 2039, 2040, 2041] * 5,
    "hub": [0, 5, 20000, 0, 0, 3, 4481, 2] + [4] * 500 + [9000],
    "empty_runs": ([0] * 2000 + [3, 0, 12]) * 3 + [0] * 1500,
}


def _matrix(lens, dtype, seed=3):
    rng = np.random.default_rng(seed)
    n_cols = 30011
    rp = np.concatenate([[0], np.cumsum(lens)])
    col = np.concatenate([np.sort(rng.choice(n_cols, size=k, replace=False)) for k in lens])
    return Csr(len(lens), n_cols, rp, col, rng.uniform(-1, 1, int(rp[-1])).astype(dtype)), \
        rng.uniform(-1, 1, n_cols).astype(dtype)


def _check(y, m, x, tol):
    from oracle import oracle as O

    m64 = Csr(m.n_rows, m.n_cols, m.row_ptr, m.col, m.val.astype(np.float64))
    y_ref, cond = O.spmv_neumaier(m64, x.astype(np.float64))
    assert np.all(np.abs(y.astype(np.float64) - y_ref) <= tol * cond)


@pytest.mark.parametrize("dtype", [np.float64, np.float32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("name", sorted(LENGTHS))
def test_tile_edges(built, name, dtype):
    from vnec_gb300 import api

    m, x = _matrix(LENGTHS[name], dtype)
    # The parity bounds of the other merge-path tests; a product here goes through
    # fewer than 200 additions, 2.2e-14 of the row's condition in FP64.
    tol = 1e-12 if dtype == np.float64 else 1e-4
    for kw in (dict(), dict(pipeline_stages=1, threads_per_block=256, items_per_thread=10)):
        p = api.Plan(m, dtype=dtype, kernel=api.KERNEL_L, **kw)
        assert p.info().pipeline_stages == 0
        y = p.mxv_host(x)
        _check(y, m, x, tol)
        assert p.mxv_host(x).tobytes() == y.tobytes()
        p.free()


@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("name", ["thread", "hub"])
def test_unaligned_caller_arrays(built, name, shift):
    """SpB_mxv_csr_noalloc_ext on columns and values that start `shift` items
    into their allocations: same y as on aligned arrays, and nothing past the
    last nonzero is read as part of a row (the items there are NaN)."""
    import torch

    from vnec_gb300 import api

    f = api.lib().SpB_mxv_csr_noalloc_ext
    f.argtypes, f.restype = [C.c_int64] * 3 + [C.c_void_p] * 6, C.c_int
    m, x = _matrix(LENGTHS[name], np.float64)
    nnz = m.nnz
    col = torch.zeros(nnz + 8, dtype=torch.int32, device="cuda")
    val = torch.full((nnz + 8,), float("nan"), dtype=torch.float64, device="cuda")
    col[shift:shift + nnz] = torch.from_numpy(m.col).cuda()
    val[shift:shift + nnz] = torch.from_numpy(m.val).cuda()
    rp, xd = torch.from_numpy(m.row_ptr.astype(np.int32)).cuda(), torch.from_numpy(x).cuda()
    y = torch.full((m.n_rows,), float("nan"), dtype=torch.float64, device="cuda")
    rc = f(m.n_rows, m.n_cols, nnz, rp.data_ptr(), col.data_ptr() + 4 * shift, val.data_ptr() + 8 * shift,
           xd.data_ptr(), y.data_ptr(), None)
    assert rc == api.SpB_SUCCESS, api.last_error()
    torch.cuda.synchronize()
    _check(y.cpu().numpy(), m, x, 1e-12)


@pytest.mark.parametrize("shape", [(128, 4), (0, 0), (256, 4), (128, 10), (256, 7), (256, 10)])
@pytest.mark.parametrize("width", [8, 16, 23, 24, 25, 31, 32, 33, 255, 257])
def test_carries_between_threads(built, width, shape):
    """Rows on both sides of the longest one that threads carry by walking back
    (24 nonzeros, and by alignment up to 32), in tiles of 3, 4, 5, 6, 8 and 11
    warps; a NaN and an infinity stay in their rows."""
    from vnec_gb300 import api

    m, x = _matrix([width] * 700 + [1, width + 1, 0] * 50, np.float64, seed=width)
    for row, v in ((3, np.nan), (350, np.inf)):
        m.val[m.row_ptr[row] + width // 2] = v
    p = api.Plan(m, kernel=api.KERNEL_L, pipeline_stages=1, threads_per_block=shape[0], items_per_thread=shape[1])
    y = p.mxv_host(x)
    p.free()
    assert np.isnan(y[3]) and np.isinf(y[350])
    rows = np.setdiff1d(np.arange(m.n_rows), [3, 350])
    assert np.all(np.isfinite(y[rows]))
    m.val[~np.isfinite(m.val)] = 0.0
    y[[3, 350]] = [m.val[m.row_ptr[r]:m.row_ptr[r + 1]] @ x[m.col[m.row_ptr[r]:m.row_ptr[r + 1]]] for r in (3, 350)]
    # At most 257 products, 257 x 2^-53 of the row's condition (2.9e-14).
    _check(y, m, x, 1e-13)
