"""CSR and COO products with several right-hand sides where the warp-run
kernel changes path: nonzero counts around a run, rows cut by slot, run and
warp edges, long runs of empty rows, arrays off a 16-byte boundary, beta 0,
1 and between, every slot width. Per entry |Y - Y64| <= 1e-5 (|alpha| sum
|a x| + |beta y|) for FP32 values, 2^-8 / 2^-10 for BF16 / FP16 (the bounds
of gpu_util)."""
import numpy as np
import pytest

from clspmv_mic_b200 import formats as F
from tests.gpu_util import VALUE_RTOL, columns_reference

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def _matrix(lens, w, seed):
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(len(lens)), lens)
    cols = np.concatenate([np.sort(rng.choice(w, n, replace=False)) for n in lens if n] or [np.zeros(0, int)])
    return F.coo_matrix(len(lens), w, rows, cols, rng.standard_normal(rows.size).astype(np.float32))


def _case(name):
    rng = np.random.default_rng(3)
    if name.startswith("nnz"):     # one nonzero count around a run of 128, rows of 1 .. 5
        n, lens = int(name[3:]), []
        while n:
            lens.append(min(n, 1 + len(lens) % 5))
            n -= lens[-1]
        return _matrix(lens, 97, 1)
    if name == "empty_runs":       # empty rows: singly, 9, 300 and 5000 in a row, first and last
        lens = [0] * 7 + [3, 0, 2] + [0] * 9 + [140, 1] + [0] * 300 + [5] * 20 + [0] * 5000 + [129, 0, 0, 1] + [0] * 40
        return _matrix(lens, 501, 2)
    if name == "long_rows":
        lens = [1, 700, 2, 3, 1500, 0, 64, 64, 128, 256, 5, 40] + list(rng.integers(0, 20, 60))
        return _matrix(lens, 1601, 4)
    if name == "mixed":
        return _matrix(list(rng.integers(0, 33, 1500)), 1203, 5)
    if name == "full":             # over 1.2M nonzeros: 8 per lane, several runs per warp
        lens = np.minimum(4000, rng.zipf(1.7, 120_000)).astype(int)
        lens[::17] = 0
        lens = np.concatenate([lens, np.full(40_000, 25)])
        rows = np.repeat(np.arange(lens.size), lens)
        key = np.unique(rows * 50_000 + rng.integers(0, 50_000, rows.size))
        rows, cols = key // 50_000, key % 50_000
        return F.coo_matrix(lens.size, 50_000, rows, cols, rng.standard_normal(rows.size).astype(np.float32))
    raise KeyError(name)


def _check(coo, fmt, k, beta, value_type="f32", off=False):
    rng = np.random.default_rng(k)
    h, w = coo.shape
    dev = F.DeviceMatrix(F.coo2csr(coo) if fmt == "csr" else coo)
    if off:
        t = {n: (torch.cat([v[:1], v])[1:] if not n.endswith("row_ptr") else v) for n, v in dev.tensors.items()}
        dev = F.DeviceMatrix.from_device_arrays(fmt, dict(width=w, height=h, nnz=coo.nnz), t)
    X = rng.uniform(-1, 1, (w, k)).astype(np.float32)
    Y0 = rng.uniform(-1, 1, (h, k)).astype(np.float32)
    Y = torch.full((h, k), float("nan"), device="cuda") if beta == 0 else torch.from_numpy(Y0).cuda()
    packed = None if value_type == "f32" else dev.pack(value_type)
    alpha = 1.0 if beta == 0 else -1.5
    F.device_spmm(dev, torch.from_numpy(X).cuda(), Y, alpha, beta, packed)
    _, y64, scale = columns_reference(coo, X, alpha)
    want = y64 + (beta * Y0.astype(np.float64) if beta else 0)
    lim = VALUE_RTOL[value_type] * scale + (1e-5 * abs(beta) * np.abs(Y0) if beta else 0) + 1e-30
    err = np.abs(Y.cpu().numpy().astype(np.float64) - want)
    assert (err <= lim).all(), (fmt, k, beta, value_type, np.argwhere(~(err <= lim))[:4].tolist())


NAMES = ["nnz1", "nnz127", "nnz128", "nnz129", "nnz255", "nnz257", "empty_runs", "long_rows", "mixed"]


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("fmt", ["csr", "coo"])
@pytest.mark.parametrize("k", [1, 3, 4, 8, 12, 16, 31, 64, 128])
def test_widths(name, fmt, k):
    for beta in (0.0, 1.0, 0.5):
        _check(_case(name), fmt, k, beta)


@pytest.mark.parametrize("fmt", ["csr", "coo"])
@pytest.mark.parametrize("k,beta", [(4, 0.0), (7, 0.5), (16, 0.0), (32, 1.0)])
def test_several_runs_per_warp(fmt, k, beta):
    _check(_case("full"), fmt, k, beta)


@pytest.mark.parametrize("fmt", ["csr", "coo"])
@pytest.mark.parametrize("value_type", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("off", [False, True])
def test_value_types_and_alignment(fmt, value_type, off):
    for k in (2, 8, 20):
        _check(_case("long_rows"), fmt, k, 0.0, value_type, off)
        _check(_case("mixed"), fmt, k, 0.5, value_type, off)
