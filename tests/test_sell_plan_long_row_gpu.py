"""The planned SELL product of slices with little padding gives 4 rows to a
thread only where no row is long: slices of 4 and 8 rows hold a long row
without much padding. Launch counts tell the two ways apart (the split walk
applies beta in a launch of its own)."""
import numpy as np
import pytest

from clspmv_mic_b200 import formats as F
from tests.gpu_util import assert_close, reference_y

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("sh", [4, 8, 32])
@pytest.mark.parametrize("longest,launches", [(3, 1), (24, 1), (25, 2), (3000, 2)])
def test_long_rows_are_split(sh, longest, launches):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    rng = np.random.default_rng(longest)
    lens = np.full(30000, 3)
    lens[[4001, 29998]] = longest
    r = np.repeat(np.arange(lens.size), lens)
    c = np.concatenate([np.sort(rng.choice(4000, n, replace=False)) for n in lens])
    coo = F.coo_matrix(lens.size, 4000, r, c, rng.standard_normal(r.size).astype(np.float32))
    dev = F.DeviceMatrix(F.coo2sell(coo, sh))
    x = rng.uniform(-1, 1, 4000).astype(np.float32)
    for packed in (None, dev.pack("f16")):
        y = torch.full((lens.size,), float("nan"), device="cuda")
        dev.sell_plan()
        n = F.launch_count()
        dev.spmv(torch.from_numpy(x).cuda(), y, 1.0, 0.0, variant="planned", packed=packed)
        if longest < 3000 or sh < 32:   # a 32-row slice of 3,000 columns is mostly padding: the split walk before, too
            assert F.launch_count() - n == launches
        ref, y64, bound = reference_y(coo, x)
        if packed is None:
            assert_close(y.cpu().numpy(), ref, bound, f"sell{sh}")
        else:
            assert (np.abs(y.cpu().numpy() - y64) <= 2.0 ** -10 * bound + 1e-30).all()
