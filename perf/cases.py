"""The SpMV work that the performance of this library is followed on.

Each case is one pass through the public Python interface (``vnec_gb300.api``,
``vnec_gb300.pagerank``) as a user's program makes it: a plan built once from a
host CSR matrix, then calls on vectors that live where that user keeps them
(device tensors, or host arrays for the reference's own calls).  Matrices are
the generator mix of this repository's benchmark and tuner: uniform rows,
R-MAT graphs, 27-point stencils, lognormal row lengths, bands and dense
diagonal blocks.  They are drawn here with torch on the GPU, from the seed
alone.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare``/``run`` make and run one, ``work`` counts the bytes and operations
it cannot do without and ``exact`` is the result in plain 64-bit torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from vnec_gb300 import api, pagerank

KERNEL = {"auto": api.KERNEL_AUTO, "L": api.KERNEL_L, "D": api.KERNEL_D, "S": api.KERNEL_S}
PRECISION = {"fp64": api.PREC_FP64, "fp32": api.PREC_FP32, "bf16": api.PREC_BF16, "df32": api.PREC_DF32}
VALUE_BYTES = {"fp64": 8, "fp32": 4, "bf16": 2, "df32": 8}
DEVICE = torch.device("cuda", 0)
LOGNORMAL_MU, LOGNORMAL_CAP = math.log(8.0), 4096
PAGERANK_STEPS, DAMPING = 4, 0.85


def listed():
    return [
        # The smallest call: the reference's own flow (Build_VNEC_S + SpMV_VNEC_S_FP64 on host
        # vectors) on a matrix of the size of its test fixtures.  Latency and launches count.
        {"name": "host_small", "kind": "host", "family": "lognormal", "rows": 3001, "sigma": 1.0, "kernel": "S"},
        # The benchmark's CPU-sized configuration, through the automatic selection: a solver's small
        # operator that stays in L2.
        {"name": "uniform64k", "kind": "mxv", "family": "uniform", "rows": 65536, "width": 16, "kernel": "auto",
         "form": "fp64", "dtype": "f64"},
        # The power-law benchmark shape (average degree 16) that goes beyond L2.
        {"name": "rmat22", "kind": "mxv", "family": "rmat", "scale": 22, "degree": 16.0, "kernel": "auto",
         "form": "fp64", "dtype": "f64"},
        # What the reference harness runs from 3 million rows on: the merge-path variant, on the same
        # kind of graph.
        {"name": "rmat22_merge", "kind": "mxv", "family": "rmat", "scale": 22, "degree": 12.0, "kernel": "L",
         "form": "fp64", "dtype": "f64"},
        # A PDE operator (27-point stencil), the benchmark's second matrix, in plain FP64 ...
        {"name": "stencil144", "kind": "mxv", "family": "stencil", "grid": 144, "kernel": "auto", "form": "fp64",
         "dtype": "f64"},
        # ... and in the FP32 precision form that the selection builds for it.
        {"name": "stencil160_fp32", "kind": "mxv", "family": "stencil", "grid": 160, "kernel": "auto", "form": "fp32",
         "dtype": "f64"},
        # The BF16 form on the power-law shape (the benchmark's other precision form and matrix).
        {"name": "rmat21_bf16", "kind": "mxv", "family": "rmat", "scale": 21, "degree": 16.0, "kernel": "auto",
         "form": "bf16", "dtype": "f64"},
        # The dense-block variant on an FP32-typed matrix of dense diagonal blocks (multi-component
        # unknowns), last block ragged.
        {"name": "blockdiag_dense", "kind": "mxv", "family": "blockdiag", "rows": 500003, "width": 24, "kernel": "D",
         "form": "fp64", "dtype": "f32"},
        # Many uneven matrices with a block of right-hand sides, in one call: the FP32 form, few
        # right-hand sides ...
        {"name": "batch_k8_fp32", "kind": "batch", "matrices": 48, "rows": 100000, "k": 8, "form": "fp32"},
        # ... and plain FP64 with the most it takes.
        {"name": "batch_k32_fp64", "kind": "batch", "matrices": 32, "rows": 100000, "k": 32, "form": "fp64"},
        # Sparse x (the push side): a graph traversal's frontier, reached along random edges.
        {"name": "frontier", "kind": "spmspv", "scale": 20, "degree": 16.0, "nnz_x": 50000},
        # A power iteration on the device: four PageRank steps and their convergence test.
        {"name": "pagerank", "kind": "pagerank", "scale": 20, "degree": 16.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_matrix(rng, nnz):
    """A family with about `nnz` nonzeros."""
    family = rng.choice(["uniform", "rmat", "stencil", "lognormal", "banded", "blockdiag"])
    if family == "uniform":
        width = rng.randint(3, 40)
        return {"family": family, "rows": max(1000, nnz // width), "width": width}
    if family == "rmat":
        degree = round(rng.uniform(6.0, 24.0), 2)
        return {"family": family, "scale": min(22, max(10, round(math.log2(nnz / degree)))), "degree": degree}
    if family == "stencil":
        return {"family": family, "grid": max(10, round((nnz / 26.0) ** (1.0 / 3.0)))}
    if family == "lognormal":
        sigma = round(rng.uniform(0.5, 2.0), 2)
        return {"family": family, "rows": max(1000, int(nnz / _lognormal_mean(sigma))), "sigma": sigma}
    if family == "banded":
        width = 2 * rng.randint(1, 64) + 1
        return {"family": family, "rows": max(1000, nnz // width), "width": width}
    width = rng.randint(8, 64)
    return {"family": family, "rows": max(1000, nnz // width), "width": width}


def draw(rng):
    kind = rng.choice(["host", "mxv", "mxv", "mxv", "mxv", "mxv", "batch", "batch", "spmspv", "pagerank"])
    if kind == "host":
        m = _draw_matrix(rng, _log_int(rng, 2e4, 3e6))
        return {"kind": kind, **m, "kernel": rng.choice(["L", "S", "D"])}
    if kind == "mxv":
        m = _draw_matrix(rng, _log_int(rng, 1e5, 5e7))
        kernel = rng.choice(["auto", "auto", "auto", "S", "L", "D"])
        if kernel == "D" and m["family"] not in ("stencil", "banded", "blockdiag"):
            kernel = "L"
        form = rng.choice(["fp64", "fp64", "fp32", "bf16", "df32"]) if kernel in ("auto", "S") else "fp64"
        dtype = rng.choice(["f64", "f64", "f32"]) if form == "fp64" else "f64"
        return {"kind": kind, **m, "kernel": kernel, "form": form, "dtype": dtype}
    if kind == "batch":
        return {"kind": kind, "matrices": rng.randint(8, 32), "rows": _log_int(rng, 5e3, 1e5),
                "k": rng.choice([1, 2, 4, 8, 16, 32]), "form": rng.choice(["fp64", "fp32", "df32"])}
    scale, degree = rng.randint(14, 20), round(rng.uniform(8.0, 20.0), 2)
    if kind == "spmspv":
        return {"kind": kind, "scale": scale, "degree": degree, "nnz_x": _log_int(rng, 64, (1 << scale) / 8)}
    return {"kind": kind, "scale": scale, "degree": degree}


# --- matrices -------------------------------------------------------------------------------------

class Csr:
    """Host CSR arrays as ``api.Plan`` takes them."""

    def __init__(self, n_rows, n_cols, row_ptr, col, val):
        self.n_rows, self.n_cols, self.row_ptr, self.col, self.val = n_rows, n_cols, row_ptr, col, val


def _lognormal_mean(sigma):
    return math.exp(LOGNORMAL_MU + 0.5 * sigma * sigma)


def _from_keys(n, keys):
    """(row counts, columns) of sorted distinct keys row * n + column."""
    return torch.bincount(keys // n, minlength=n), (keys % n).to(torch.int32)


def _pattern(c, g):
    """(rows, row counts, columns) on the GPU; every family is square, with increasing columns in a row."""
    family = c["family"]
    if family == "rmat":
        n, edges = 1 << c["scale"], int(c["degree"] * (1 << c["scale"]))
        key = torch.zeros(edges, dtype=torch.int64, device=DEVICE)
        for level in range(c["scale"]):  # a, b, c, d = 0.57, 0.19, 0.19, 0.05
            u = torch.rand(edges, generator=g, device=DEVICE)
            row, col = u >= 0.76, ((u >= 0.57) & (u < 0.76)) | (u >= 0.95)
            key += (row.to(torch.int64) << (2 * c["scale"] - 1 - level)) + (col.to(torch.int64) << (c["scale"] - 1 - level))
        return n, *_from_keys(n, torch.unique(key))
    if family == "lognormal":
        n = c["rows"]
        length = torch.exp(LOGNORMAL_MU + c["sigma"] * torch.randn(n, generator=g, device=DEVICE))
        length = length.round().clamp(0, min(LOGNORMAL_CAP, n)).to(torch.int64)
        row = torch.repeat_interleave(torch.arange(n, device=DEVICE), length)
        return n, *_from_keys(n, torch.unique(row * n + torch.randint(n, row.shape, generator=g, device=DEVICE)))
    if family == "uniform":
        n, k = c["rows"], c["width"]
        row = torch.arange(n, device=DEVICE).repeat_interleave(k) * n
        keys = torch.unique(row + torch.randint(n, (n * k,), generator=g, device=DEVICE))
        while keys.numel() < n * k:  # exactly k distinct columns a row: draw again what fell together
            short = k - torch.bincount(keys // n, minlength=n)
            row = torch.arange(n, device=DEVICE).repeat_interleave(short) * n
            keys = torch.unique(torch.cat([keys, row + torch.randint(n, row.shape, generator=g, device=DEVICE)]))
        return n, *_from_keys(n, keys)
    if family == "stencil":
        s = c["grid"]
        n = s ** 3
        i = torch.arange(n, device=DEVICE)
        z, y, x = i // (s * s), (i // s) % s, i % s
        cols, keep = [], []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    keep.append((z + dz >= 0) & (z + dz < s) & (y + dy >= 0) & (y + dy < s) & (x + dx >= 0) & (x + dx < s))
                    cols.append((i + (dz * s + dy) * s + dx).to(torch.int32))
        keep = torch.stack(keep, 1)
        return n, keep.sum(1), torch.stack(cols, 1)[keep]
    n, w = c["rows"], c["width"]
    i = torch.arange(n, device=DEVICE)
    first = i - w // 2 if family == "banded" else i // w * w
    cols = first[:, None] + torch.arange(w, device=DEVICE)
    keep = (cols >= 0) & (cols < n)
    return n, keep.sum(1), cols.to(torch.int32)[keep]


def _matrix(c, g):
    """(rows, row counts, columns, FP64 values) on the GPU."""
    n, counts, col = _pattern(c, g)
    val = torch.rand(col.shape, generator=g, device=DEVICE, dtype=torch.float64)
    if c["family"] == "stencil":  # off-diagonals U(-1, 0], diagonal 1 + the sum of their sizes
        row = torch.repeat_interleave(torch.arange(n, device=DEVICE), counts)
        off = col != row
        size = torch.segment_reduce(torch.where(off, val, 0.0), "sum", lengths=counts)  # in one order on every run
        val = torch.where(off, -val, 1.0 + size[row])
    elif c["family"] != "rmat":  # U(-1, 1); a graph's weights are U(0, 1)
        val = 2.0 * val - 1.0
    return n, counts, col, val


def _host(n, counts, col, val):
    row_ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEVICE)
    row_ptr[1:] = torch.cumsum(counts, 0)
    return Csr(n, n, row_ptr.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy())


def _vector(n, g, dtype=torch.float64):
    return (2.0 * torch.rand(n, generator=g, device=DEVICE, dtype=torch.float64) - 1.0).to(dtype)


def _batch_cases(c):
    """The matrices of a batch: row counts spread evenly over log [1000, rows], small and large ones in turn."""
    count = c["matrices"]
    step = math.log(c["rows"] / 1000.0) / max(1, count - 1)
    sizes = [int(1000.0 * math.exp(step * i)) for i in range(count)]
    return [{"family": "lognormal", "rows": sizes[-1 - i // 2] if i & 1 else sizes[i // 2], "sigma": 1.5}
            for i in range(count)]


def _inputs(case, seed):
    """The matrices and vectors of a case, on the GPU: what prepare() plans and exact() computes with."""
    g = torch.Generator(DEVICE).manual_seed(seed)
    kind = case["kind"]
    if kind == "batch":
        mats = [_matrix(m, g) for m in _batch_cases(case)]
        return mats, [_vector(m[0] * case["k"], g).reshape(m[0], case["k"]) for m in mats]
    if kind in ("spmspv", "pagerank"):
        mat = _matrix({"family": "rmat", **case}, g)
        if kind == "pagerank":
            rank = torch.rand(mat[0], generator=g, device=DEVICE, dtype=torch.float64)
            return mat, rank / rank.sum()
        # The endpoints of random edges: hubs are on a frontier more often than leaves.
        ends = mat[2][torch.randint(mat[2].numel(), (4 * case["nnz_x"],), generator=g, device=DEVICE)]
        idx = torch.unique(ends)
        idx = idx[torch.randperm(idx.numel(), generator=g, device=DEVICE)[: case["nnz_x"]]]
        return mat, (idx.to(torch.int32), _vector(idx.numel(), g))
    mat = _matrix(case, g)
    if case.get("dtype") == "f32":
        return (*mat[:3], mat[3].to(torch.float32)), _vector(mat[0], g, torch.float32)
    return mat, _vector(mat[0], g)


# --- one pass -------------------------------------------------------------------------------------

def _stream():
    return torch.cuda.current_stream(DEVICE).cuda_stream


def prepare(case, seed):
    mat, x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "host":
        csr = _host(*mat)
        A = api.Matrix.from_csr(csr)
        build = {"L": api.Build_VNEC_L, "S": api.Build_VNEC_S_FP64, "D": api.Build_VNEC_D_FP64}[case["kernel"]]
        free = {"L": api.VNEC_L_free, "S": api.VNEC_S_free_fp64, "D": api.VNEC_D_free_fp64}[case["kernel"]]
        call = {"L": api.SpMV_VNEC_L_FP64, "S": api.SpMV_VNEC_S_FP64, "D": api.SpMV_VNEC_D_FP64}[case["kernel"]]
        return Host(A, api.Vector(x.cpu().numpy()), api.Vector(n=csr.n_rows), build(A), call, free)
    if kind == "mxv":
        csr = _host(*mat)
        plan = api.Plan(csr, dtype=csr.val.dtype, kernel=KERNEL[case["kernel"]], precision=PRECISION[case["form"]])
        return {"kind": kind, "plan": plan, "x": x, "y": torch.empty_like(x)}
    if kind == "batch":
        plan = api.BatchPlan([_host(*m) for m in mat], case["k"], precision=PRECISION[case["form"]])
        X = torch.cat(x)
        return {"kind": kind, "plan": plan, "x": X, "y": torch.empty_like(X)}
    if kind == "spmspv":
        idx, val = x
        return {"kind": kind, "plan": api.Plan(_host(*mat), kernel=api.KERNEL_PUSH), "idx": idx, "val": val,
                "y": torch.empty(mat[0], dtype=torch.float64, device=DEVICE)}
    transition, dangling = pagerank.transition(_host(*mat))
    return {"kind": kind, "n": mat[0], "plan": api.Plan(transition, kernel=api.KERNEL_S, transpose=True),
            "rank": x, "next": [torch.empty_like(x), torch.empty_like(x)],
            "mask": torch.from_numpy(dangling.astype(np.float64)).to(DEVICE),
            "scalars": torch.zeros(2, dtype=torch.float64, device=DEVICE),
            "partial": torch.empty(api.DOT_BLOCKS, dtype=torch.float64, device=DEVICE)}


class Host:
    """The reference's objects of a host-vector call; the handle is freed with them."""

    def __init__(self, A, x, y, handle, call, free):
        self.A, self.x, self.y, self.handle, self.call, self.free = A, x, y, handle, call, free

    def __del__(self):
        self.free(self.handle)


def run(state):
    if isinstance(state, Host):
        state.call(state.y, state.A, state.x, state.handle)
        return state.y.values
    s, plan = _stream(), state["plan"]
    if state["kind"] == "spmspv":
        plan.spmspv_device(state["idx"].numel(), state["idx"].data_ptr(), state["val"].data_ptr(),
                           state["y"].data_ptr(), s)
        return state["y"]
    if state["kind"] == "pagerank":
        n, r, scalars, partial = state["n"], state["rank"], state["scalars"], state["partial"].data_ptr()
        for step in range(PAGERANK_STEPS):
            out = state["next"][step & 1]
            api.dot(n, r.data_ptr(), state["mask"].data_ptr(), 0, partial, scalars.data_ptr(), s)
            plan.mxv_axpbyg(r.data_ptr(), out.data_ptr(), alpha=DAMPING, gamma=(1.0 - DAMPING) / n,
                            d_g=scalars.data_ptr(), g_scale=DAMPING / n, stream=s)
            last, r = r, out
        api.dot(n, r.data_ptr(), last.data_ptr(), 1, partial, scalars.data_ptr() + 8, s)
        return [r, scalars]
    plan.mxv_device(state["x"].data_ptr(), state["y"].data_ptr(), s)
    return state["y"]


# --- what a pass cannot do without -----------------------------------------------------------------

def _sizes(c):
    """(rows, nonzeros) of a matrix: exact, or the expectation where they are random."""
    family = c["family"]
    if family == "rmat":
        n = 1 << c["scale"]
        return n, c["degree"] * n
    if family == "lognormal":
        return c["rows"], c["rows"] * _lognormal_mean(c["sigma"])
    if family == "stencil":
        return c["grid"] ** 3, (3 * c["grid"] - 2) ** 3
    n, w = c["rows"], c["width"]
    if family == "uniform":
        return n, n * w
    if family == "banded":
        h = w // 2
        return n, n * w - h * (h + 1)
    return n, n // w * w * w + (n % w) ** 2


def _frontier_entries(c):
    """(vertices, entries of their columns) expected of a frontier: an edge ends at a vertex of h one bits with
    probability 0.24^h 0.76^(scale - h); of the distinct ends of 4 nnz_x edges, nnz_x are kept."""
    s, draws = c["scale"], 4 * c["nnz_x"]
    p = [0.24 ** h * 0.76 ** (s - h) for h in range(s + 1)]
    found = [math.comb(s, h) * -math.expm1(-draws * p[h]) for h in range(s + 1)]
    kept = min(1.0, c["nnz_x"] / sum(found))
    return kept * sum(found), kept * sum(f * q for f, q in zip(found, p)) * c["degree"] * (1 << s)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = [_sizes(m) for m in _batch_cases(case)]
        n, nnz = sum(s[0] for s in sizes), sum(s[1] for s in sizes)
        return {"bytes": nnz * (VALUE_BYTES[case["form"]] + 4) + (n + len(sizes)) * 4 + 2 * n * case["k"] * 8,
                "flops": 2 * nnz * case["k"]}
    n, nnz = _sizes({"family": "rmat", **case})
    if kind == "spmspv":
        vertices, entries = _frontier_entries(case)
        return {"bytes": entries * 12 + vertices * 28 + n * 8, "flops": 2 * entries}
    if kind == "pagerank":
        step = nnz * 12 + n * 4 + 3 * n * 8
        return {"bytes": PAGERANK_STEPS * step + 2 * n * 8, "flops": PAGERANK_STEPS * (2 * nnz + 4 * n) + 3 * n}
    io = 4 if case.get("dtype") == "f32" else 8
    value = io if case.get("form", "fp64") == "fp64" else VALUE_BYTES[case["form"]]
    return {"bytes": nnz * (value + 4) + (n + 1) * 4 + 2 * n * io, "flops": 2 * nnz}


# --- the result in 64 bits --------------------------------------------------------------------------

def _product(mat, x):
    """A x with plain torch in FP64; x is a vector or a row-major block of right-hand sides."""
    n, counts, col, val = mat
    y = torch.zeros((n, *x.shape[1:]), dtype=torch.float64, device=DEVICE)
    row = torch.repeat_interleave(torch.arange(n, device=DEVICE), counts)
    for b in range(0, col.numel(), 1 << 22):
        part = x.double()[col[b:b + (1 << 22)].long()]
        scale = val[b:b + (1 << 22)].double()
        y.index_add_(0, row[b:b + (1 << 22)], part * (scale[:, None] if x.dim() == 2 else scale))
    return y


def exact(case, seed):
    mat, x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        return torch.cat([_product(m, v) for m, v in zip(mat, x)]).reshape(-1)
    if kind == "spmspv":
        full = torch.zeros(mat[0], dtype=torch.float64, device=DEVICE)
        full[x[0].long()] = x[1]
        return _product(mat, full)
    if kind == "pagerank":
        n, counts, col, _ = mat
        row = torch.repeat_interleave(torch.arange(n, device=DEVICE), counts)
        share = 1.0 / counts.clamp(min=1).double()
        r, last, mass = x, x, 0.0
        for _ in range(PAGERANK_STEPS):
            mass = r[counts == 0].sum()
            y = torch.zeros(n, dtype=torch.float64, device=DEVICE).index_add_(0, col.long(), (share * r)[row])
            r, last = DAMPING * y + ((1.0 - DAMPING) + DAMPING * mass) / n, r
        return [r, torch.stack([mass, (r - last).abs().sum()])]
    y = _product(mat, x)
    return y.cpu().numpy() if kind == "host" else y
