"""Steps of A^k x in one launch: which matrices take it, by launch counts, and
every entry of the result. Matrices and vectors are positive, so that each step
is a sum of positive terms: with rows of at most L entries an FP32 step has a
relative error of at most (L + 3) 2^-24 per entry, k steps of k times that to
first order (2 % added for the rest), whatever the size of the result."""
import numpy as np
import pytest

from clspmv_mic_b200 import _abi
from clspmv_mic_b200 import cocktail as CK
from clspmv_mic_b200 import formats as F

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def _banded(h, w, offsets, seed, keep=1.0):
    r = np.repeat(np.arange(h), len(offsets))
    c = r + np.tile(np.sort(offsets), h)
    ok = (c >= 0) & (c < w) & (np.random.default_rng(seed).random(r.size) < keep)
    return h, w, r[ok], c[ok]


def _uneven(h, w, longest, seed):
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, longest + 1, h)
    r = np.repeat(np.arange(h), lens)
    return h, w, r, np.concatenate([np.sort(rng.choice(w, n, replace=False)) for n in lens])


def _grid(n):
    h, w, r, c = _banded(n * n, n * n, [-n, -1, 0, 1, n], 1)
    ok = ~((np.abs(c - r) == 1) & (c // n != r // n))
    return h, w, r[ok], c[ok]


# name -> (structure, resident as DIA / BDIA, resident as COO / CSR)
CASES = {"one": (lambda: _banded(1, 1, [0], 1), True, True), "grid6": (lambda: _grid(6), True, True),
         "grid32": (lambda: _grid(32), True, True), "grid33": (lambda: _grid(33), True, True),
         "grid100": (lambda: _grid(100), True, True), "grid256": (lambda: _grid(256), True, True),
         "grid300": (lambda: _grid(300), False, False), "wide": (lambda: _banded(2500, 2600, [-70, -3, 0, 1, 2, 90, 99], 2, 0.8), True, True),
         "holes": (lambda: _banded(17000, 17000, [-5000, -2, 0, 3, 9000], 3, 0.7), True, True),
         "uneven": (lambda: _uneven(9000, 9000, 12, 4), None, False), "few": (lambda: _uneven(700, 760, 12, 5), None, True),
         "long80": (lambda: _uneven(700, 700, 80, 6), None, False),
         "near": (lambda: _banded(9000, 9000, np.arange(-7, 8), 8, 0.5), True, True),
         "band40": (lambda: _banded(4000, 4000, np.arange(-20, 20), 9), None, False),
         "band150": (lambda: _banded(900, 900, np.arange(-75, 75), 9), False, False)}


@pytest.mark.parametrize("fmt", ["dia", "bdia", "coo", "csr"])
@pytest.mark.parametrize("name", list(CASES))
def test_every_entry_and_the_launches(fmt, name):
    make, as_dia, as_rows = CASES[name]
    resident = as_dia if fmt in ("dia", "bdia") else as_rows
    if resident is None:
        pytest.skip("too many diagonals")
    h, w, r, c = make()
    rng = np.random.default_rng(7)
    v = rng.uniform(0.5, 1.5, r.size).astype(np.float32)
    rowsum, longest = np.bincount(r, v, h), int(np.bincount(r, minlength=h).max())
    v = (v / np.float32(rowsum.max())).astype(np.float32)
    coo = F.coo_matrix(h, w, r, c, v)
    part = coo if fmt == "coo" else getattr(F, f"coo2{fmt}")(coo)
    st = _abi.Cocktail()
    st.mat_height, st.mat_width, st.mat_nnz = h, w, coo.nnz
    setattr(st, f"ifuse{fmt}", True)
    setattr(st, fmt, type(getattr(st, fmt)).from_buffer_copy(part.struct))
    dev = CK.CocktailMatrix(st, owner=None).to_device()
    a = torch.sparse_coo_tensor(torch.from_numpy(np.stack([r, c])), torch.from_numpy(v.astype(np.float64)), (h, w)).cuda()
    x0 = torch.from_numpy(rng.uniform(0.5, 1, w).astype(np.float32)).cuda()
    y0 = torch.from_numpy(rng.uniform(0.5, 1, h).astype(np.float32)).cuda()
    for k in (1, 3, 4, 5, 19):
        for alpha, beta in ((1.0, 0.0), (0.75, 0.25), (1.0, 1.0)):
            x, y = x0.clone(), (torch.full_like(y0, float("nan")) if beta == 0 else y0.clone())
            n = F.launch_count()
            dev.iterate(x, y, k, alpha, beta)
            n = F.launch_count() - n
            assert k == 1 or (n == 1) == (resident and k >= 4), (n, k)
            xd, yd = x0.double(), y0.double()
            for _ in range(k):
                yd = alpha * (a @ xd) + (beta * yd if beta else 0)
                xd[:h] = yd
            torch.cuda.synchronize()
            assert torch.equal(x[:h], y) and torch.equal(x[h:], x0[h:])
            lim = 1.02 * k * (longest + 3) * 2.0 ** -24 * yd
            assert bool(((y.double() - yd).abs() <= lim).all()), (k, alpha, beta, float(((y.double() - yd).abs() / yd).max()))


@pytest.mark.parametrize("fmt,name", [("coo", "uneven"), ("csr", "uneven"), ("coo", "band40"), ("csr", "band40"), ("bdia", "band150"),
                                      ("bdia", "band40"), ("dia", "grid100"), ("csr", "grid256")])
def test_no_slower_than_single_steps(fmt, name):
    """A cluster that holds the matrix reads other CTAs' entries one after another: uneven rows took 3, bands 2 to 4 times
    as long as the single steps."""
    h, w, r, c = CASES[name][0]()
    coo = F.coo_matrix(h, w, r, c, np.full(r.size, 1e-3, np.float32))
    part = coo if fmt == "coo" else getattr(F, f"coo2{fmt}")(coo)
    st = _abi.Cocktail()
    st.mat_height, st.mat_width, st.mat_nnz = h, w, coo.nnz
    setattr(st, f"ifuse{fmt}", True)
    setattr(st, fmt, type(getattr(st, fmt)).from_buffer_copy(part.struct))
    dev = CK.CocktailMatrix(st, owner=None).to_device()
    x, y = torch.rand(w, device="cuda"), torch.rand(h, device="cuda")

    def us(f):
        times = []
        for _ in range(9):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            f()
            e[1].record()
            torch.cuda.synchronize()
            times.append(e[0].elapsed_time(e[1]) * 1000)
        return float(np.median(times[2:]))

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for _ in range(48):
            dev.spmv(x, y, 1.0, 0.5)
            x[:h].copy_(y)
    assert us(lambda: dev.iterate(x, y, 48, 1.0, 0.5)) <= 1.25 * us(g.replay)
