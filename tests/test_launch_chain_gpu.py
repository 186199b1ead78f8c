"""Chained launches keep stream order: a call may start while the kernel before
it drains, so a chain of calls whose inputs are the outputs of the calls (and of
other kernels, copies and streams) before them is run without any wait and must
give the bits of the same chain with a device synchronisation after every step."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plans(name):
    from vnec_gb300 import api
    from vnec_gb300 import generators as G

    r = G.rmat(13, 12 << 13, seed=3)      # hot columns, long rows
    u = G.uniform_k(1 << 13, 9, seed=4)   # one launch per call
    b = G.banded(1 << 13, 17, seed=5)     # 16-bit deltas
    kw = {"S": dict(kernel=api.KERNEL_S, hot_columns=256, long_row_len=64),
          "L": dict(kernel=api.KERNEL_L),
          "D": dict(kernel=api.KERNEL_D),
          "fp32": dict(kernel=api.KERNEL_S, precision=api.PREC_FP32, long_row_len=64),
          "bf16": dict(kernel=api.KERNEL_S, precision=api.PREC_BF16),
          "df32": dict(kernel=api.KERNEL_S, precision=api.PREC_DF32, hot_columns=256)}[name]
    return [api.Plan(m, **kw) for m in (r, u, b)]


@pytest.mark.parametrize("name", ["S", "L", "D", "fp32", "bf16", "df32"])
def test_chain_matches_synchronised_chain(built, name):
    import torch

    from vnec_gb300 import api

    plans = _plans(name)
    n = 1 << 13
    x0 = torch.from_numpy(np.random.default_rng(1).uniform(-1, 1, n)).cuda()
    part = torch.empty(api.DOT_BLOCKS, dtype=torch.float64, device="cuda")

    def chain(sync):
        wait = torch.cuda.synchronize if sync else (lambda: None)
        main, side = torch.cuda.Stream(), torch.cuda.Stream()
        main.wait_stream(torch.cuda.current_stream())
        a, b = x0.clone(), torch.empty_like(x0)
        scal = torch.zeros(1, dtype=torch.float64, device="cuda")
        torch.cuda.current_stream().synchronize()
        with torch.cuda.stream(main):
            for i in range(60):
                p = plans[i % 3]
                p.mxv_device(a.data_ptr(), b.data_ptr(), main.cuda_stream)
                wait()
                api.dot(n, b.data_ptr(), b.data_ptr(), 0, part.data_ptr(), scal.data_ptr(), main.cuda_stream)
                wait()
                if i % 4 == 0:    # a kernel of another library writes x just before the next call
                    torch.div(b, scal.sqrt(), out=a)
                elif i % 4 == 1:  # a device-to-device copy does
                    a.copy_(b)
                    a.mul_(0.125)
                    p.mxv_axpbyg(b.data_ptr(), a.data_ptr(), alpha=0.01, beta=1.0, d_z=a.data_ptr(),
                                 d_g=scal.data_ptr(), g_scale=1e-3, stream=main.cuda_stream)
                else:             # a kernel on another stream does, ordered by events
                    side.wait_stream(main)
                    with torch.cuda.stream(side):
                        torch.div(b, scal.sqrt(), out=a)
                    main.wait_stream(side)
                wait()
        torch.cuda.synchronize()
        return a.cpu().numpy(), scal.cpu().numpy()

    want = chain(True)
    assert np.isfinite(want[0]).all() and np.abs(want[0]).max() > 0
    for _ in range(3):
        got = chain(False)
        assert got[0].tobytes() == want[0].tobytes() and got[1].tobytes() == want[1].tobytes()
    for p in plans:
        p.free()


@pytest.mark.parametrize("name", ["S", "L", "fp32", "df32"])
def test_captured_chain(built, name):
    """The same calls captured in a CUDA graph, with another library's kernels around them."""
    import torch

    plans = _plans(name)
    n = 1 << 13
    x = torch.from_numpy(np.random.default_rng(2).uniform(-1, 1, n)).cuda()
    a, b, c = (torch.empty_like(x) for _ in range(3))

    def calls(stream):
        torch.mul(x, 0.5, out=a)
        plans[0].mxv_device(a.data_ptr(), b.data_ptr(), stream)
        plans[1].mxv_device(b.data_ptr(), a.data_ptr(), stream)
        a.mul_(0.25)
        plans[2].mxv_device(a.data_ptr(), c.data_ptr(), stream)

    calls(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    want = c.cpu().numpy().tobytes()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        calls(torch.cuda.current_stream().cuda_stream)
    for _ in range(3):
        c.zero_()
        g.replay()
        g.replay()
        torch.cuda.synchronize()
        assert c.cpu().numpy().tobytes() == want
    for p in plans:
        p.free()
