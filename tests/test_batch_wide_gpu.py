"""Batches on either side of the choice between 4 and 6 CTAs per SM: one
column, k = 4, several lanes per row with a small and a large X, 8 and more
lanes, and mixtures. Per entry |Y - Y64| <= 1e-5 (|alpha| sum |a x| +
|beta y|) for FP32 values, 2^-8 / 2^-10 for BF16 / FP16 (the bounds of
gpu_util)."""
import numpy as np
import pytest

from clspmv_mic_b200 import formats as F
from clspmv_mic_b200.batch import Batch, Job
from tests.gpu_util import VALUE_RTOL, columns_reference

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def _band(h, w, seed):
    """Rows of 0 to 9 nonzeros on 9 diagonals (few enough for DIA and BDIA)."""
    rng = np.random.default_rng(seed)
    r, d = np.meshgrid(np.arange(h), [-40, -2, -1, 0, 1, 2, 3, 50, 51], indexing="ij")
    keep = (r + d >= 0) & (r + d < w) & (rng.random(r.shape) < 0.8)
    rows, cols = r[keep], (r + d)[keep]
    return F.coo_matrix(h, w, rows, cols, rng.uniform(-1, 1, rows.size).astype(np.float32))


def _scattered(h, w, seed):
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, 40, h)
    key = np.unique(np.repeat(np.arange(h, dtype=np.int64), lens) * w + rng.integers(0, w, lens.sum()))
    return F.coo_matrix(h, w, key // w, key % w, rng.uniform(-1, 1, key.size).astype(np.float32))


def _stored(coo, fmt):
    if fmt == "csr":
        return F.coo2csr(coo)
    if fmt == "dia":
        return F.coo2dia(coo)
    if fmt == "bdia":
        return F.coo2bdia(coo)
    if fmt == "ell":
        return F.coo2ell(coo, 32, 9)
    return F.coo2sell(coo, 32)


def _run(parts, value_type):
    """parts: (coo, format, k, beta)."""
    rng = np.random.default_rng(7)
    jobs, checks = [], []
    for coo, fmt, k, beta in parts:
        h, w = coo.shape
        m = F.DeviceMatrix(_stored(coo, fmt))
        X = rng.uniform(-1, 1, (w, k)).astype(np.float32)
        Y0 = rng.uniform(-1, 1, (h, k)).astype(np.float32)
        Y = torch.from_numpy(Y0).cuda()
        jobs.append(Job(m, torch.from_numpy(X).cuda(), Y, alpha=-1.5, beta=beta,
                        packed=None if value_type == "f32" else m.pack(value_type)))
        checks.append((coo, X, Y0, Y, beta))
    b = Batch(len(jobs))
    b.set(jobs)
    b.run()
    torch.cuda.synchronize()
    for i, (coo, X, Y0, Y, beta) in enumerate(checks):
        _, y64, scale = columns_reference(coo, X, -1.5)
        want = y64 + beta * Y0.astype(np.float64)
        lim = VALUE_RTOL[value_type] * scale + 1e-5 * abs(beta) * np.abs(Y0) + 1e-30
        err = np.abs(Y.cpu().numpy().astype(np.float64) - want)
        assert (err <= lim).all(), (parts[i][1:], value_type, np.argwhere(~(err <= lim))[:4].tolist())
    b.close()


@pytest.mark.parametrize("value_type", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("k", [1, 3, 4, 8, 28, 32, 36, 128])
def test_one_width(k, value_type):
    _run([(_band(h, h + 11, h), fmt, k, beta) for h, fmt, beta in
          [(1, "csr", 0.0), (33, "ell", 0.5), (257, "dia", 0.0), (600, "bdia", 1.0), (1000, "sell", 0.0), (2049, "csr", 0.5)]], value_type)


@pytest.mark.parametrize("value_type", ["f32", "bf16"])
def test_large_x(value_type):
    _run([(_scattered(700, 4_200_000, 1), "csr", 8, 0.5), (_band(100, 100, 2), "ell", 8, 0.0)], value_type)


@pytest.mark.parametrize("ks", [(1, 32, 4), (4, 4, 1), (64, 3, 8), (32, 4, 4)])
def test_mixtures(ks):
    _run([(_scattered(900 + 31 * i, 1000, i), "csr", k, 0.25 * i) for i, k in enumerate(ks)], "f32")
