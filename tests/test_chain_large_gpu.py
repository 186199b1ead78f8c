"""Unsynchronised chains of calls with many waves of blocks: each call's x is the
y the call before it wrote, in place through the epilogue's z, so a block that
starts before its predecessor has finished and read early or stale data would
change the result.  The chain must give the bits of the same chain with a device
synchronisation after every call."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1 << 20  # 4,096 blocks or more a kernel; x of 8 MB


def _matrix(kind):
    from vnec_gb300 import generators as G

    return {"rmat": lambda: G.rmat(20, 8 << 20, seed=21),      # hot columns, long rows
            "band": lambda: G.banded(N, 16, seed=22),          # 16-bit deltas, shared patterns
            "uniform": lambda: G.uniform_k(N, 6, seed=23)}[kind]()


CASES = [("S", "rmat"), ("S", "band"), ("S", "uniform"), ("L", "rmat"), ("L", "uniform"), ("D", "band"),
         ("fp32", "rmat"), ("fp32", "band"), ("bf16", "band"), ("df32", "rmat"), ("df32", "band"),
         ("S type 32", "rmat"), ("S type 32", "band"), ("L type 32", "rmat")]


@pytest.mark.parametrize("name,kind", CASES)
def test_chain_of_large_grids(built, name, kind):
    import torch

    from vnec_gb300 import api

    single = name.endswith("type 32")
    kw = {"S": dict(kernel=api.KERNEL_S), "L": dict(kernel=api.KERNEL_L), "D": dict(kernel=api.KERNEL_D),
          "fp32": dict(kernel=api.KERNEL_S, precision=api.PREC_FP32),
          "bf16": dict(kernel=api.KERNEL_S, precision=api.PREC_BF16),
          "df32": dict(kernel=api.KERNEL_S, precision=api.PREC_DF32)}[name.split()[0]]
    m = _matrix(kind)
    scale = 0.5 / float(np.abs(np.add.reduceat(np.abs(m.val), np.minimum(m.row_ptr[:-1], m.nnz - 1))).max())
    if single:
        kw["dtype"] = np.float32
    p = api.Plan(m, **kw)
    x0 = torch.from_numpy(np.random.default_rng(3).uniform(-1, 1, N)).cuda()
    if single:
        x0 = x0.float()

    def chain(sync):
        a, b = x0.clone(), x0.flip(0).contiguous()
        torch.cuda.synchronize()
        s = torch.cuda.Stream()
        for _ in range(24):
            p.mxv_axpbyg(a.data_ptr(), b.data_ptr(), alpha=scale, beta=0.5, d_z=b.data_ptr(), stream=s.cuda_stream)
            if sync:
                torch.cuda.synchronize()
            a, b = b, a
        torch.cuda.synchronize()
        return a.cpu().numpy(), b.cpu().numpy()

    want = chain(True)
    assert all(np.isfinite(w).all() and np.abs(w).max() > 0 for w in want)
    for _ in range(3):
        got = chain(False)
        assert all(g.tobytes() == w.tobytes() for g, w in zip(got, want))
    p.free()


@pytest.mark.parametrize("k,precision", [(4, "FP32"), (8, "FP32"), (8, "FP64"), (16, "DF32")])
@pytest.mark.parametrize("graph", [True, False])
def test_batch_chain_of_large_grids(built, k, precision, graph):
    """Batches: y of one call is X of the next, scaled by another library's kernel in between."""
    import torch

    from vnec_gb300 import api
    from vnec_gb300 import generators as G

    mats = [G.uniform_k(20_000 + 501 * i, 7, seed=40 + i) for i in range(8)]
    p = api.BatchPlan(mats, k, precision=getattr(api, f"PREC_{precision}"), graph=graph)
    n = sum(m.n_rows for m in mats)
    x0 = torch.from_numpy(np.random.default_rng(4).uniform(-1, 1, n * k)).cuda()

    def chain(sync):
        a, b = x0.clone(), torch.zeros_like(x0)
        torch.cuda.synchronize()
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for i in range(24):
                p.mxv_device(a.data_ptr(), b.data_ptr(), s.cuda_stream)
                if sync:
                    torch.cuda.synchronize()
                if i % 3 == 0:
                    b.mul_(0.25)
                a, b = b, a
        torch.cuda.synchronize()
        return a.cpu().numpy(), b.cpu().numpy()

    want = chain(True)
    assert all(np.isfinite(w).all() and np.abs(w).max() > 0 for w in want)
    for _ in range(3):
        got = chain(False)
        assert all(g.tobytes() == w.tobytes() for g, w in zip(got, want))
    p.free()
