"""The routes of a blocking host-vector call give the bits of the device call: y of
up to 128 KB written straight to page-locked memory, longer y copied back, and y
from 12 MB on split into parts where the caller's array is page-locked."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _device(p, x, n):
    import torch

    xd = torch.from_numpy(x).cuda()
    y = torch.empty(n, dtype=xd.dtype, device="cuda")
    p.mxv_device(xd.data_ptr(), y.data_ptr(), 0)
    torch.cuda.synchronize()
    return y.cpu().numpy()


@pytest.mark.parametrize("dtype", [np.float64, np.float32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("kernel", ["S", "L", "D", "HYBRID", "PUSH"])
def test_short_y(built, kernel, dtype):
    from vnec_gb300 import api
    from vnec_gb300 import generators as G

    edge = (128 << 10) // np.dtype(dtype).itemsize
    for n in (1, 33, edge, edge + 1):
        m = G.banded(n, 5, seed=3)
        x = G.vector(n, seed=4).astype(dtype)
        p = api.Plan(m, dtype=dtype, kernel=getattr(api, "KERNEL_" + kernel))
        want = _device(p, x, n)
        y = np.full(n, np.nan, dtype=dtype)
        for _ in range(2):  # the second call writes over the first one's y
            p.mxv_host(x, y)
            if kernel == "PUSH":  # atomics: the order of a row's additions varies
                assert np.allclose(y, want, rtol=0, atol=1e-12 if dtype == np.float64 else 1e-5)
            else:
                assert y.tobytes() == want.tobytes()
            x = -x
            want = -want
        p.free()


def test_long_y_split_when_page_locked(built):
    import torch

    from vnec_gb300 import api
    from vnec_gb300 import generators as G

    n = (12 << 20) // 8 + 77
    m = G.banded(n, 3, seed=5)
    x = G.vector(n, seed=6)
    p = api.Plan(m, kernel=api.KERNEL_S)
    want = _device(p, x, n).tobytes()
    locked = torch.empty(n, dtype=torch.float64).pin_memory()
    for y in (np.empty(n), locked.numpy()):
        y[:] = np.nan
        p.mxv_host(x, y)
        assert y.tobytes() == want
    p.free()
