"""Host-vector calls split into parts (host_parts): each part's tasks, long rows
(light and heavy ones), hot-column window and prefetch offsets are its own, and
the result has the bits of the one-launch device call.  Without host_parts calls
of this size run whole (tests/test_host_split_cpu.py counts the launches)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(name):
    from vnec_gb300 import generators as G

    return {"rmat": lambda: G.rmat(17, 16 << 17, seed=5),
            "lognormal": lambda: G.lognormal(150_000, sigma=2.0, cap=3000, seed=6),
            "stencil": lambda: G.stencil27(40, seed=7),
            "band": lambda: G.banded(100_000, 24, seed=8)}[name]()


@pytest.mark.parametrize("host_parts", [0, 3, 8])
@pytest.mark.parametrize("dtype", [np.float64, np.float32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("name,kw", [
    ("rmat", dict(window_rows=1000, hot_columns=4096)),               # hot window, long rows
    ("rmat", dict(window_rows=1000, long_row_len=64, hot_columns=-1)),  # many long rows, heavy ones
    ("rmat", dict()),
    ("lognormal", dict(window_rows=1000, long_row_len=64)),
    ("lognormal", dict(window_rows=4096, hot_columns=4096, long_row_len=16)),
    ("stencil", dict(window_rows=2000)),                              # shared patterns
    ("stencil", dict(window_rows=2000, l2_prefetch=4096)),
    ("band", dict(window_rows=1000)),
    ("band", dict(window_rows=1000, shared_patterns=-1))])            # 16-bit deltas
def test_split_call_has_the_bits_of_the_whole(built, name, kw, dtype, host_parts):
    import torch

    from vnec_gb300 import api
    from vnec_gb300 import generators as G

    m = _matrix(name)
    xv = G.vector(m.n_cols, seed=3).astype(dtype)
    p = api.Plan(m, kernel=api.KERNEL_S, dtype=dtype, host_parts=host_parts, **kw)
    x = torch.from_numpy(xv).cuda()
    y = torch.full((m.n_rows,), float("nan"), dtype=x.dtype, device="cuda")
    p.mxv_device(x.data_ptr(), y.data_ptr(), 0)
    torch.cuda.synchronize()
    want = y.cpu().numpy().tobytes()
    for buf in (np.empty(m.n_rows, dtype), torch.empty(m.n_rows, dtype=x.dtype).pin_memory().numpy()):
        for _ in range(2):
            buf[:] = np.nan
            p.mxv_host(xv, buf)
            assert buf.tobytes() == want
    p.free()
