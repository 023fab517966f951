"""clspmv_cocktail_iterate_f32 with beta = 0, whose steps go back and forth
between x and y where both serve as a vector (square matrix, both 16-byte
aligned) and copy otherwise: step counts on both sides of a graph's 16, odd
and even, one part and several, both schedules, a y off the boundary, a wide
matrix, and buffers that hold no number before the call. Against the loop of
single steps: the same bits for one part without atomics, 1e-4 of the largest
entry otherwise (the bound of test_cocktail_gpu)."""
import numpy as np
import pytest

from clspmv_mic_b200 import synth
from tests.test_cocktail_gpu import _cuda, _iterate_by_steps, setup  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg,mname", [("plain", "laplace128"), ("block_partial", "mixed"), ("sell_ell_fast", "powerlaw"),
                                       ("plain", "wide")])
@pytest.mark.parametrize("k", [0, 1, 2, 15, 16, 17, 32, 49])
@pytest.mark.parametrize("off", [False, True])
def test_against_single_steps(setup, cfg, mname, k, off):  # noqa: F811
    import torch
    coo, ck = setup[(cfg, mname)]
    dev = ck.to_device()
    h, w = coo.shape
    a = coo.arrays()
    rowsum = np.zeros(h)
    np.add.at(rowsum, a["coo_row_id"], np.abs(a["coo_data"]))
    alpha = float(1.0 / max(rowsum.max(), 1.0))
    x0 = torch.from_numpy(synth.x_vector(w)).cuda()
    y0 = torch.full((h + 1,), float("nan"), device="cuda")
    for schedule in ("auto", "fused") if len(dev.parts) > 1 else ("auto",):
        dev.set_schedule(schedule)
        x1, y1 = x0.clone(), y0.clone()[1:] if off else y0.clone()[:h]
        for _ in range(2):   # the second call replays the cached graph
            x1.copy_(x0)
            y1.fill_(float("nan"))
            dev.iterate(x1, y1, k, alpha, 0.0)
        x2, y2 = x0.clone(), y0.clone()[1:] if off else y0.clone()[:h]
        _iterate_by_steps(dev, x2, y2, k, alpha, 0.0)
        torch.cuda.synchronize()
        if k == 0:
            assert torch.equal(x1, x0) and bool(torch.isnan(y1).all())
            continue
        assert torch.equal(x1[:h], y1)
        assert torch.equal(x1[h:], x0[h:])
        if len(dev.parts) == 1 and dev.parts[0] in ("dia", "bdia", "ell", "bell", "sbell", "bcsr"):
            assert torch.equal(y1, y2), dev.parts
        else:
            assert float((y1 - y2).abs().max()) <= 1e-4 * (float(y2.abs().max()) + 1e-30), dev.parts


def _grid(n):
    return synth.laplacian_2d(n)


def _uneven(rows, cols, longest, seed):
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, longest + 1, rows)
    r = np.repeat(np.arange(rows), lens)
    c = np.concatenate([np.sort(rng.choice(cols, n, replace=False)) for n in lens])
    return rows, cols, r, c, rng.standard_normal(r.size).astype(np.float32) / max(1, longest)


@pytest.mark.parametrize("fmt", ["dia", "bdia", "coo", "csr"])
@pytest.mark.parametrize("name", ["grid5", "grid33", "grid70", "grid150", "uneven", "wide", "long"])
def test_one_part_resident_in_a_cluster(fmt, name):
    """Matrices of one part from one CTA's rows to all of a cluster's (and
    wider than tall, with rows too long for it): every step count and beta
    against the loop of single steps in 64 bits. Per entry the error is at
    most steps * 1e-5 of the largest entry of |A|^k-scaled terms, taken as
    the largest result (the rows are scaled to sums of at most 1)."""
    import torch
    from clspmv_mic_b200 import _abi
    from clspmv_mic_b200 import cocktail as CK
    from clspmv_mic_b200 import formats as F
    if name.startswith("grid"):
        h, w, r, c, v = _grid(int(name[4:]))
        v = v / 8
    elif fmt in ("dia", "bdia"):
        h, w, r, c, v = synth.banded(3001, 9)
        v = v / 9
    else:
        h, w, r, c, v = _uneven(*{"uneven": (9000, 9000, 12, 1), "wide": (2500, 2600, 20, 2), "long": (700, 700, 90, 3)}[name])
    coo = F.coo_matrix(h, w, r, c, v)
    part = coo if fmt == "coo" else getattr(F, f"coo2{fmt}")(coo)
    st = _abi.Cocktail()
    st.mat_height, st.mat_width, st.mat_nnz = h, w, coo.nnz
    setattr(st, f"ifuse{fmt}", True)
    setattr(st, fmt, type(getattr(st, fmt)).from_buffer_copy(part.struct))
    host = CK.CocktailMatrix(st, owner=None)
    dev = host.to_device()
    a = torch.sparse_coo_tensor(torch.stack([torch.as_tensor(np.asarray(r)), torch.as_tensor(np.asarray(c))]),
                                torch.as_tensor(np.asarray(v, np.float64)), (h, w)).cuda()
    x0 = torch.from_numpy(synth.x_vector(w)).cuda()
    y0 = torch.from_numpy(np.random.default_rng(4).uniform(-1, 1, h).astype(np.float32)).cuda()
    for k in (1, 3, 4, 5, 18):
        for alpha, beta in ((1.0, 0.0), (0.5, 0.25)):
            x, y = x0.clone(), (torch.full_like(y0, float("nan")) if beta == 0 else y0.clone())
            dev.iterate(x, y, k, alpha, beta)
            xd, yd = x0.double(), y0.double()
            for _ in range(k):
                yd = alpha * (a @ xd) + (beta * yd if beta else 0)
                xd[:h] = yd
            torch.cuda.synchronize()
            assert torch.equal(x[:h], y) and torch.equal(x[h:], x0[h:])
            assert float((y.double() - yd).abs().max()) <= k * 1e-5 * max(1.0, float(yd.abs().max())), (k, alpha, beta)
