"""Batches whose time is that of a few long rows, each walked by one lane group:
a column more or less must not change how many lookups a lane has in flight."""
import numpy as np
import pytest

from clspmv_mic_b200 import formats as F
from clspmv_mic_b200.batch import Batch, Job

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def _us(m, k):
    jobs = [Job(m, torch.rand((m.shape[1], k), device="cuda"), torch.zeros((m.shape[0], k), device="cuda"), 1.0, 0.0)]
    b = Batch(1)
    b.set(jobs)
    times = []
    for _ in range(9):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        b.run()
        e[1].record()
        torch.cuda.synchronize()
        times.append(e[0].elapsed_time(e[1]) * 1000)
    b.close()
    return float(np.median(times[2:]))


@pytest.mark.parametrize("fmt", ["csr", "sell"])
@pytest.mark.parametrize("k,beside", [(1, 2), (32, 16)])
def test_long_rows_keep_their_pace(fmt, k, beside):
    """40,000 rows of 3 and ten of 20,000: with 6 CTAs per SM a lane had one lookup in flight, 2.6 times as long."""
    n, rng = 40_000, np.random.default_rng(3)
    lens = np.full(n, 3)
    lens[rng.choice(n, 10, replace=False)] = 20_000
    rows = np.repeat(np.arange(n), lens)
    start = np.repeat(np.cumsum(lens) - lens, lens)
    cols = (np.arange(rows.size) - start) * n // lens[rows]
    coo = F.coo_matrix(n, n, rows, cols, np.ones(rows.size, np.float32))
    m = F.DeviceMatrix(F.coo2csr(coo) if fmt == "csr" else F.coo2sell(coo, 32))
    assert _us(m, k) <= 1.5 * _us(m, beside)
