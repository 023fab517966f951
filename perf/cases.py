"""Timed work of this framework: sparse products through its public calls.

A case is one call (or one short sequence of calls) that a program makes
again and again: a single-vector product in one of the storage formats, a
product with several right-hand sides, a conversion of a matrix that is
already on the device, a batch of uneven matrices, or steps of A^k x on a
partitioned matrix. Fields of a case:

  kind    "spmv", "spmm", "convert", "batch" or "iterate"
  fmt     storage format ("batch" and "iterate" choose their own)
  shape   structure of the matrix: "laplacian" (5-point, square grid),
          "stencil27" (27-point, cube), "banded" (consecutive diagonals),
          "blocks" (dense 4x4 blocks), "random" (uneven random rows) or
          "powerlaw" (Zipf row lengths)
  rows    rows (the grids take the largest grid that fits)
  per_row mean entries per row where the structure leaves it open
  values  "f32", or "bf16" / "f16" for 16-bit stored values
  op      "ax" (y = A x) or "residual" (r = b - A x)
  k       right-hand sides
  jobs    matrices of a batch
  steps   steps of A^k x

Matrices and vectors are made on the GPU from the seed alone: N(0, 1) values
(the Laplacian's are 4 and -1), x uniform in [-1, 1]. The row lengths belong
to the case, so that a converted matrix has one size whatever the seed; the
columns, values and vectors follow the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from clspmv_mic_b200 import cocktail, formats
from clspmv_mic_b200.batch import Batch, Job

DEVICE = "cuda"
ZIPF_S, ZIPF_MAX = 2.0, 10_000
BLOCK_FORMATS = ("b4csr", "b4ell", "sbell")


def listed():
    return [
        # a solver's inner product on a small grid: the call itself and its launches are the cost
        dict(name="csr_spmv_laplacian64", kind="spmv", fmt="csr", shape="laplacian", rows=64 * 64, per_row=5,
             values="f32", op="ax"),
        # power iteration / polynomial smoothing on a grid that stays in the L2 cache
        dict(name="iterate_laplacian256", kind="iterate", shape="laplacian", rows=256 * 256, per_row=5, steps=40),
        # structured-grid solver: the 27-point stencil by diagonals
        dict(name="dia_spmv_stencil128", kind="spmv", fmt="dia", shape="stencil27", rows=128 ** 3, per_row=27,
             values="f32", op="ax"),
        # graph with a few very long rows: the residual of a linear solve
        dict(name="csr_spmv_powerlaw", kind="spmv", fmt="csr", shape="powerlaw", rows=1 << 20, per_row=16,
             values="f32", op="residual"),
        # the same graph in slices, through its length plan
        dict(name="sell_spmv_powerlaw", kind="spmv", fmt="sell", shape="powerlaw", rows=1 << 20, per_row=16,
             values="f32", op="ax"),
        # finite elements with 4 unknowns per node
        dict(name="bcsr_spmv_blocks", kind="spmv", fmt="b4csr", shape="blocks", rows=2_000_000, per_row=32,
             values="f32", op="ax"),
        # graph features: many columns at once over uneven rows
        dict(name="csr_spmm_powerlaw_k16", kind="spmm", fmt="csr", shape="powerlaw", rows=1 << 20, per_row=16,
             values="f32", k=16),
        # block Krylov on a structured grid of odd side, values stored in 16 bits
        dict(name="dia_spmm_stencil101_k8_bf16", kind="spmm", fmt="dia", shape="stencil27", rows=101 ** 3,
             per_row=27, values="bf16", k=8),
        # block Krylov on finite elements, the widest X of the range
        dict(name="sbell_spmm_blocks_k32", kind="spmm", fmt="sbell", shape="blocks", rows=2_000_000, per_row=32,
             values="f32", k=32),
        # assembly ends with a COO on the device: into block slices, the largest conversion
        dict(name="convert_sbell_blocks", kind="convert", fmt="sbell", shape="blocks", rows=2_000_000, per_row=32),
        # an uneven graph of ragged size from COO into slices
        dict(name="convert_sell_powerlaw", kind="convert", fmt="sell", shape="powerlaw", rows=700_001, per_row=16),
        # a server's mix: 48 matrices of 1k to 500k rows in several formats, one launch
        dict(name="batch_uneven_k4", kind="batch", rows=500_000, per_row=32, jobs=48, values="f32", k=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes from 1k rows up to the listed ones, spread over their logarithm."""
    kind = rng.choice(["spmv", "spmv", "spmv", "spmm", "spmm", "convert", "convert", "batch", "iterate"])
    if kind == "iterate":
        return dict(kind=kind, shape="laplacian", rows=_log_int(rng, 1_000, 160_000), per_row=5,
                    steps=rng.randint(1, 64))
    if kind == "batch":
        return dict(kind=kind, rows=_log_int(rng, 5_000, 500_000), per_row=rng.randint(5, 32),
                    jobs=rng.randint(2, 48), values=rng.choice(["f32", "f32", "bf16", "f16"]), k=rng.choice([1, 4, 8]))
    shape = rng.choice(["laplacian", "stencil27", "banded", "blocks", "random", "powerlaw"])
    per_row = {"laplacian": 5, "stencil27": 27, "banded": rng.randint(3, 31), "blocks": 4 * rng.randint(2, 8),
               "random": rng.randint(4, 40), "powerlaw": rng.randint(8, 16)}[shape]
    fmt = rng.choice({"laplacian": ["csr", "coo", "dia", "bdia", "ell", "sell"],
                      "stencil27": ["csr", "dia", "bdia", "ell", "sell"],
                      "banded": ["csr", "coo", "dia", "bdia", "ell", "sell"],
                      "blocks": ["b4csr", "b4ell", "sbell", "csr"],
                      "random": ["csr", "coo", "ell", "sell"],
                      "powerlaw": ["csr", "coo", "sell"]}[shape])
    case = dict(kind=kind, fmt=fmt, shape=shape, rows=_log_int(rng, 1_000, 1_000_000), per_row=per_row)
    if kind == "convert":
        if fmt == "coo":
            case["fmt"] = "csr"
        return case
    case["values"] = rng.choice(["f32", "f32", "bf16", "f16"])
    if kind == "spmv":
        case["op"] = rng.choice(["ax", "residual"])
    else:
        case["k"] = rng.choice([4, 8, 12, 16, 24, 32, rng.randint(1, 31)])
    return case


# ---------------------------------------------------------------------------
# Matrices, on the GPU, as (rows, columns, row id, column id, value) sorted by row and column
# ---------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _side(rows, dims):
    n = int(round(rows ** (1.0 / dims)))
    while n ** dims > rows:
        n -= 1
    return max(2, n)


def _zipf(per_row):
    """Lengths 1..ZIPF_MAX of Zipf(2) rows scaled to a mean of per_row, with their probabilities."""
    k = np.arange(1, ZIPF_MAX + 1, dtype=np.float64)
    p = k ** -ZIPF_S
    p /= p.sum()
    lens = np.clip(np.rint(k * (per_row / float((p * k).sum()))), 1, ZIPF_MAX)
    return lens, p


def _grid(n, dims, points, g):
    m = n ** dims
    r = torch.arange(m, device=DEVICE)
    ok, cols = [], []
    for d in points:
        inside = torch.ones(m, dtype=torch.bool, device=DEVICE)
        off, stride = 0, 1
        for axis in range(dims):
            at = (r // stride) % n + d[axis]
            inside &= (at >= 0) & (at < n)
            off += d[axis] * stride
            stride *= n
        ok.append(inside)
        cols.append((off, r + off))
    order = sorted(range(len(points)), key=lambda i: cols[i][0])
    ok = torch.stack([ok[i] for i in order], dim=1)
    col = torch.stack([cols[i][1] for i in order], dim=1)[ok]
    row = r[:, None].expand(m, len(points))[ok]
    if dims == 2:
        val = torch.where(row == col, 4.0, -1.0).float()
    else:
        val = torch.randn(row.numel(), generator=g, device=DEVICE)
    return m, row, col, val


def _rows_of(lens, n, g):
    """Rows of the given lengths: entry j of a row of L lies anywhere in the j-th of L equal bands of the columns,
    so that columns are distinct and sorted."""
    m = lens.numel()
    start = torch.cumsum(lens, 0) - lens
    row = torch.repeat_interleave(torch.arange(m, device=DEVICE), lens)
    j, L = torch.arange(row.numel(), device=DEVICE) - start[row], lens[row]
    lo = j * n // L
    wide = (j + 1) * n // L - lo
    return row, lo + (torch.rand(row.numel(), generator=g, device=DEVICE, dtype=torch.float64) * wide).long()


def _entries(case, g):
    shape, rows, per_row = case["shape"], int(case["rows"]), int(case["per_row"])
    if shape == "laplacian":
        rows, row, col, val = _grid(_side(rows, 2), 2, [(0, 0), (-1, 0), (1, 0), (0, -1), (0, 1)], g)
        return rows, row.int(), col.int(), val
    if shape == "stencil27":
        pts = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)]
        rows, row, col, val = _grid(_side(rows, 3), 3, pts, g)
        return rows, row.int(), col.int(), val
    if shape == "banded":
        r = torch.arange(rows, device=DEVICE)[:, None]
        col = r + torch.arange(per_row, device=DEVICE) - per_row // 2
        ok = (col >= 0) & (col < rows)
        row, col = r.expand_as(col)[ok], col[ok]
    elif shape == "blocks":
        per = per_row // 4
        brows = (rows + 3) // 4
        band = (rows // 4) // per
        bc = torch.randint(0, band, (brows, per), generator=g, device=DEVICE) + torch.arange(per, device=DEVICE) * band
        col = (bc[:, None, :, None] * 4 + torch.arange(4, device=DEVICE)).expand(brows, 4, per, 4).reshape(-1)
        row = torch.arange(brows * 4, device=DEVICE).repeat_interleave(per * 4)
        if rows % 4:
            ok = row < rows
            row, col = row[ok], col[ok]
    elif shape == "random":
        lens = torch.randint(max(1, per_row // 2), per_row + per_row // 2 + 1, (rows,), generator=_generator(rows),
                             device=DEVICE)
        row, col = _rows_of(lens, rows, g)
    else:
        lens, p = _zipf(per_row)
        cdf = torch.from_numpy(np.cumsum(p)).to(DEVICE)
        u = torch.rand(rows, generator=_generator(rows), device=DEVICE, dtype=torch.float64)
        at = torch.searchsorted(cdf, u).clamp_(max=ZIPF_MAX - 1)
        lens = torch.from_numpy(lens).to(DEVICE)[at].long().clamp_(max=rows)
        row, col = _rows_of(lens, rows, g)
    val = torch.randn(row.numel(), generator=g, device=DEVICE)
    return rows, row.int(), col.int(), val


def _device_coo(rows, row, col, val):
    return formats.DeviceMatrix.from_device_arrays("coo", dict(width=rows, height=rows, nnz=row.numel()),
                                                   dict(coo_row_id=row, coo_col_id=col, coo_data=val))


def _in_format(coo, fmt):
    if fmt == "coo":
        return coo
    return formats.device_convert(coo, fmt, *((4, 4) if fmt in BLOCK_FORMATS else ()))


def _batch_shapes(case):
    """(structure, format, rows) of a batch's matrices: rows spread over their logarithm from 1k to case["rows"]."""
    kinds = [("random", "csr"), ("banded", "ell"), ("blocks", "sbell"), ("random", "csr"), ("banded", "dia"),
             ("blocks", "b4csr")]
    jobs, hi = int(case["jobs"]), math.log(int(case["rows"]) / 1000.0)
    out = []
    for i in range(jobs):
        f = (i * 0.6180339887498949) % 1.0
        out.append(kinds[i % len(kinds)] + (int(1000 * math.exp(f * hi)) | 1,))
    return out


def _batch_case(case, i, shape, rows):
    per = max(4, int(case["per_row"]) - (i * 7) % max(1, int(case["per_row"]) // 2))
    return dict(shape=shape, rows=rows, per_row=max(4, per // 4 * 4) if shape == "blocks" else per)


def _uniform(shape, g):
    return torch.rand(shape, generator=g, device=DEVICE) * 2 - 1


# ---------------------------------------------------------------------------
# What a program has before the call, and the call
# ---------------------------------------------------------------------------
def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "batch":
        specs = _batch_shapes(case)
        k = int(case["k"])
        Y = torch.zeros((sum(rows for _, _, rows in specs), k), device=DEVICE)
        jobs, at = [], 0
        for i, (shape, fmt, rows) in enumerate(specs):
            m = _in_format(_device_coo(*_entries(_batch_case(case, i, shape, rows), g)), fmt)
            packed = None if case["values"] == "f32" else m.pack(case["values"])
            jobs.append(Job(m, _uniform((rows, k), g), Y[at: at + rows], 1.0, 0.0, packed=packed))
            at += rows
        b = Batch(len(jobs))
        b.set(jobs)
        return dict(kind=kind, batch=b, Y=Y)
    rows, row, col, val = _entries(case, g)
    if kind == "iterate":
        host = formats.coo_matrix(rows, rows, row.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy())
        dev = cocktail.analyze(host).to_device()
        x0 = _uniform((rows,), g)
        return dict(kind=kind, matrix=dev, x0=x0, x=x0.clone(), y=torch.zeros_like(x0), steps=int(case["steps"]))
    coo = _device_coo(rows, row, col, val)
    if kind == "convert":
        return dict(kind=kind, coo=coo, fmt=case["fmt"])
    m = _in_format(coo, case["fmt"])
    packed = None if case["values"] == "f32" else m.pack(case["values"])
    if kind == "spmm":
        k = int(case["k"])
        return dict(kind=kind, matrix=m, packed=packed, X=_uniform((rows, k), g), Y=torch.zeros((rows, k), device=DEVICE))
    kw = {}
    if case["fmt"] == "csr":
        m.chunk_plan()
    if case["fmt"] == "sell":
        m.sell_plan()
        kw["variant"] = "planned"
    return dict(kind=kind, matrix=m, packed=packed, kw=kw, op=case["op"], x=_uniform((rows,), g),
                b=_uniform((rows,), g), y=torch.zeros(rows, device=DEVICE))


def run(state):
    kind = state["kind"]
    if kind == "spmv":
        y = state["y"]
        if state["op"] == "residual":
            y.copy_(state["b"])
            state["matrix"].spmv(state["x"], y, -1.0, 1.0, packed=state["packed"], **state["kw"])
        else:
            state["matrix"].spmv(state["x"], y, 1.0, 0.0, packed=state["packed"], **state["kw"])
        return y
    if kind == "spmm":
        state["matrix"].spmm(state["X"], state["Y"], 1.0, 0.0, packed=state["packed"])
        return state["Y"]
    if kind == "convert":
        return dict(_in_format(state["coo"], state["fmt"]).tensors)
    if kind == "batch":
        state["batch"].run()
        return state["Y"]
    state["x"].copy_(state["x0"])
    state["matrix"].iterate(state["x"], state["y"], state["steps"], 0.125, 0.0)
    return state["y"]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _counts(case):
    """(rows, entries, diagonals) to be expected of a case's matrix."""
    shape, rows, per = case["shape"], int(case["rows"]), int(case["per_row"])
    if shape == "laplacian":
        n = _side(rows, 2)
        return n * n, 5 * n * n - 4 * n, 5
    if shape == "stencil27":
        n = _side(rows, 3)
        return n ** 3, (3 * n - 2) ** 3, 27
    if shape == "banded":
        return rows, rows * per, per
    if shape == "powerlaw":
        lens, p = _zipf(per)
        return rows, int(rows * float((np.minimum(lens, rows) * p).sum())), 0
    return rows, rows * per, 0


def _slice_slots(case, height=32):
    """Slots of SELL slices to be expected: the longest of `height` rows, over all slices."""
    rows, nnz, _ = _counts(case)
    if case["shape"] == "powerlaw":
        lens, p = _zipf(int(case["per_row"]))
        lens = np.minimum(lens, rows)
        longest = float(np.sum((np.cumsum(p) ** height - np.concatenate([[0.0], np.cumsum(p)[:-1]]) ** height) * lens))
        return rows * longest
    if case["shape"] == "random":
        per = int(case["per_row"])
        return rows * float(per + per // 2)
    return float(nnz)


def _matrix_bytes(case, fmt, value_bytes=4):
    """The matrix in its format: values, indices and pointers, without padding that a kernel may skip."""
    rows, nnz, diagonals = _counts(case)
    if fmt in ("dia", "bdia"):
        return value_bytes * nnz + 4 * diagonals
    if fmt in BLOCK_FORMATS:
        return value_bytes * nnz + 4 * nnz / 16 + 4 * rows / 4
    if fmt == "coo":
        return (8 + value_bytes) * nnz
    if fmt in ("csr", "sell"):
        return (4 + value_bytes) * nnz + 4 * rows
    return (4 + value_bytes) * nnz


def work(case):
    kind = case["kind"]
    if kind == "batch":
        vb = 4 if case["values"] == "f32" else 2
        k, by, fl = int(case["k"]), 0.0, 0.0
        for i, (shape, fmt, rows) in enumerate(_batch_shapes(case)):
            c = _batch_case(case, i, shape, rows)
            by += _matrix_bytes(c, fmt, vb) + 8.0 * rows * k + (4.0 * rows if vb == 2 else 0)
            fl += 2.0 * _counts(c)[1] * k
        return {"bytes": by, "flops": fl}
    rows, nnz, diagonals = _counts(case)
    if kind == "iterate":   # matrix and vectors once: the steps between run on chip
        return {"bytes": 4.0 * nnz + 8.0 * rows, "flops": 2.0 * nnz * int(case["steps"])}
    if kind == "convert":
        fmt = case["fmt"]
        if fmt == "sell":
            out = 8.0 * _slice_slots(case)
        elif fmt == "ell":
            most = {"random": int(case["per_row"]) + int(case["per_row"]) // 2}.get(case["shape"], int(case["per_row"]))
            out = 8.0 * rows * most
        elif fmt in ("dia", "bdia"):
            out = 4.0 * rows * diagonals
        else:
            out = _matrix_bytes(case, fmt)
        return {"bytes": 12.0 * nnz + out, "flops": 0.0}
    vb = 4 if case["values"] == "f32" else 2
    by = _matrix_bytes(case, case["fmt"], vb) + (4.0 * rows if vb == 2 else 0)
    if kind == "spmm":
        return {"bytes": by + 8.0 * rows * int(case["k"]), "flops": 2.0 * nnz * int(case["k"])}
    return {"bytes": by + (12.0 if case["op"] == "residual" else 8.0) * rows, "flops": 2.0 * nnz}


# ---------------------------------------------------------------------------
# The same results in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _product64(rows, row, col, val, x):
    """A x for a vector x, in 64 bits."""
    y = torch.zeros(rows, dtype=torch.float64, device=DEVICE)
    return y.index_add_(0, row, val.double() * x[col])


def _columns64(rows, row, col, val, X):
    X = X.double()
    row, col = row.long(), col.long()
    return torch.stack([_product64(rows, row, col, val, X[:, j].contiguous()) for j in range(X.shape[1])], dim=1)


def exact(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "convert":
        return None   # entries moved, none computed
    if kind == "batch":
        out = []
        for i, (shape, _, rows) in enumerate(_batch_shapes(case)):
            entries = _entries(_batch_case(case, i, shape, rows), g)
            out.append(_columns64(*entries, _uniform((rows, int(case["k"])), g)))
        return torch.cat(out)
    rows, row, col, val = _entries(case, g)
    if kind == "spmm":
        return _columns64(rows, row, col, val, _uniform((rows, int(case["k"])), g))
    row, col = row.long(), col.long()
    x = _uniform((rows,), g).double()
    if kind == "iterate":
        for _ in range(int(case["steps"])):
            x = 0.125 * _product64(rows, row, col, val, x)
        return x
    y = _product64(rows, row, col, val, x)
    return _uniform((rows,), g).double() - y if case["op"] == "residual" else y
