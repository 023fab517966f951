"""SELL and ELL products with several right-hand sides around the slot counts
where the batched walk changes path (rows of fewer than a batch, whole
batches, half and single remainders), slices of every height class, uneven
and empty rows, beta 0 and between. Per entry the bounds of gpu_util."""
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


def _matrix(lens, w, seed=1):
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(len(lens)), lens)
    cols = np.concatenate([np.sort(rng.choice(w, n, replace=False)) for n in lens if n] or [np.zeros(0, int)])
    return F.coo_matrix(len(lens), w, rows, cols, rng.standard_normal(rows.size).astype(np.float32))


def _check(coo, host, k, beta, value_type):
    rng = np.random.default_rng(k)
    h, w = coo.shape
    dev = F.DeviceMatrix(host)
    X, Y0 = (rng.uniform(-1, 1, (n, k)).astype(np.float32) for n in (w, h))
    Y = torch.full((h, k), float("nan"), device="cuda") if beta == 0 else torch.from_numpy(Y0).cuda()
    packed = None if value_type == "f32" else dev.pack(value_type)
    F.device_spmm(dev, torch.from_numpy(X).cuda(), Y, -1.5, beta, packed)
    _, y64, scale = columns_reference(coo, X, -1.5)
    want = y64 + (beta * Y0.astype(np.float64) if beta else 0)
    lim = VALUE_RTOL[value_type] * scale + (1e-5 * abs(beta) * np.abs(Y0) if beta else 0) + 1e-30
    err = np.abs(Y.cpu().numpy().astype(np.float64) - want)
    assert (err <= lim).all(), np.argwhere(~(err <= lim))[:4].tolist()


@pytest.mark.parametrize("slots", [7, 8, 9, 12, 13, 16, 21])
@pytest.mark.parametrize("k", [2, 3, 4, 12, 32])
def test_slot_counts(slots, k):
    coo = _matrix([slots] * 75, 203)
    for value_type in ("f32", "bf16", "f16"):
        for host in (F.coo2sell(coo, 32), F.coo2ell(coo)):
            _check(coo, host, k, 0.5 if k == 4 else 0.0, value_type)


@pytest.mark.parametrize("sh", [1, 4, 7, 32, 128])
def test_uneven_slices(sh):
    lens = [0, 40, 3, 8, 16, 1] + list(np.random.default_rng(2).integers(0, 30, 131)) + [0] * 9
    coo = _matrix(lens, 301, 3)
    for k, beta, value_type in ((8, 0.0, "f32"), (5, 0.5, "f32"), (16, 0.0, "bf16")):
        _check(coo, F.coo2sell(coo, sh), k, beta, value_type)
