"""The planned SELL product of matrices with little padding (4 rows per thread
up to their real lengths) beside the split walk: widths on both sides of the
rule, ragged heights, slice heights a multiple of 4 and not, an infinity in
x that only padding would touch, beta 0 and between, 16-bit values."""
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


def _matrix(lens, w, seed):
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(len(lens)), lens)
    cols = np.concatenate([np.sort(rng.choice(w, n, replace=False)) for n in lens])
    return F.coo_matrix(len(lens), w, rows, cols, rng.standard_normal(rows.size).astype(np.float32))


def _check(coo, sh, value_type, beta):
    rng = np.random.default_rng(sh)
    h, w = coo.shape
    x, y0 = (rng.uniform(-1, 1, n).astype(np.float32) for n in (w, h))
    dev = F.DeviceMatrix(F.coo2sell(coo, sh))
    packed = None if value_type == "f32" else dev.pack(value_type)
    y = torch.full((h,), float("nan"), device="cuda") if beta == 0 else torch.from_numpy(y0).cuda()
    dev.spmv(torch.from_numpy(x).cuda(), y, 0.5, beta, variant="planned", packed=packed)
    _, y64, bound = reference_y(coo, x, y0, 0.5, beta)
    err = np.abs(y.cpu().numpy().astype(np.float64) - y64)
    assert (err <= VALUE_RTOL[value_type] * bound + 1e-30).all(), np.argwhere(~(err <= VALUE_RTOL[value_type] * bound + 1e-30))[:4]


@pytest.mark.parametrize("sh", [4, 8, 12, 32, 128, 7])
@pytest.mark.parametrize("width", [1, 12, 13, 33])
@pytest.mark.parametrize("rows", [1, 31, 130, 1027])
def test_widths(sh, width, rows):
    coo = _matrix([max(1, width - (r % 3)) for r in range(rows)], 200, width)
    for value_type in ("f32", "bf16", "f16"):
        _check(coo, sh, value_type, 0.0)
    _check(coo, sh, "f32", 0.75)


def test_wide_rows_of_a_large_matrix():
    """Rows of 27 past the row count from which FP32 takes the thread's walk."""
    n = 500_003
    r = np.repeat(np.arange(n), 27)
    c = (r + np.tile(np.arange(27) * 7, n)) % n
    order = np.lexsort((c, r))
    coo = F.coo_matrix(n, n, r[order], c[order], np.random.default_rng(1).standard_normal(r.size).astype(np.float32))
    _check(coo, 32, "f32", 0.0)


def test_padding_multiplies_nothing():
    """Row 0's last column holds an infinity of x; its neighbours' padding must not reach it."""
    lens = [2, 5, 5, 5] * 8
    coo = _matrix(lens, 64, 3)
    dev = F.DeviceMatrix(F.coo2sell(coo, 32))
    x = np.ones(64, np.float32)
    last = coo.array("coo_col_id")[1]
    x[last] = np.inf
    y = torch.zeros(32, device="cuda")
    dev.spmv(torch.from_numpy(x).cuda(), y, 1.0, 0.0, variant="planned")
    assert torch.isinf(y[0])   # its own entry, and no 0 * inf from its padding
