"""CSR and COO products small enough for one launch (a cluster that applies
beta to y, then adds): nonzero counts around a chunk of 256 and the most the
launch takes, rows around its row limit, rows of one chunk and of many, runs
of empty rows, beta 0 over NaN and between, 16-bit values, under capture.
Per row the bounds of gpu_util."""
import numpy as np
import pytest

from clspmv_mic_b200 import formats as F
from tests.gpu_util import VALUE_RTOL, reference_y

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def _matrix(lens, w, seed=1):
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(len(lens)), lens)
    cols = np.concatenate([np.sort(rng.choice(w, n, replace=False)) for n in lens if n] or [np.zeros(0, int)])
    return F.coo_matrix(len(lens), w, rows, cols, rng.standard_normal(rows.size).astype(np.float32))


def _lens(name):
    rng = np.random.default_rng(5)
    if name.startswith("nnz"):
        n, lens = int(name[3:]), []
        while n:
            lens.append(min(n, 1 + len(lens) % 9))
            n -= lens[-1]
        return lens
    return {"long": [3] * 20 + [1900] + [1] * 300 + [700, 0, 0, 5], "empty": [0] * 400 + [2, 0, 0, 300] + [0] * 3000 + [1] * 40 + [0] * 99,
            "rows32768": [1] * 32768, "rows32769": [1] * 32769, "mixed": list(rng.integers(0, 30, 2000))}[name]


@pytest.mark.parametrize("name", ["nnz0", "nnz1", "nnz255", "nnz256", "nnz257", "nnz4096", "nnz4097", "nnz32768", "nnz32769", "long",
                                  "empty", "rows32768", "rows32769", "mixed"])
@pytest.mark.parametrize("fmt", ["csr", "coo"])
@pytest.mark.parametrize("value_type", ["f32", "bf16", "f16"])
def test_against_oracle(name, fmt, value_type):
    lens = _lens(name)
    coo = _matrix(lens, max(2000, 50)) if lens else F.coo_matrix(40, 50, np.zeros(0, int), np.zeros(0, int), np.zeros(0, np.float32))
    h, w = coo.shape
    rng = np.random.default_rng(2)
    x, y0 = (rng.uniform(-1, 1, n).astype(np.float32) for n in (w, h))
    dev = F.DeviceMatrix(F.coo2csr(coo) if fmt == "csr" else coo)
    packed = None if value_type == "f32" else dev.pack(value_type)
    xd = torch.from_numpy(x).cuda()
    for beta in (0.0, -0.5, 1.0):
        y = torch.full((h,), float("nan"), device="cuda") if beta == 0 else torch.from_numpy(y0).cuda()
        dev.spmv(xd, y, 2.0, beta, packed=packed)
        _, y64, bound = reference_y(coo, x, y0, 2.0, beta)
        err = np.abs(y.cpu().numpy().astype(np.float64) - y64)
        assert (err <= VALUE_RTOL[value_type] * bound + 1e-30).all(), (beta, np.argwhere(~(err <= VALUE_RTOL[value_type] * bound + 1e-30))[:4])


def test_under_capture():
    coo = _matrix(_lens("mixed"), 2000)
    dev = F.DeviceMatrix(F.coo2csr(coo))
    x = torch.rand(2000, device="cuda")
    y, z = torch.zeros(coo.shape[0], device="cuda"), torch.zeros(coo.shape[0], device="cuda")
    dev.spmv(x, z, 1.0, 0.0)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        dev.spmv(x, y, 1.0, 0.0)
    y.fill_(float("nan"))
    g.replay()
    assert torch.allclose(y, z, rtol=1e-5, atol=1e-5)
