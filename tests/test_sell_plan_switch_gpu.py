"""CLSPMV_SELL_SPLIT=0 keeps the planned SELL product on its walk over every
column, also for slices of little padding: beta is applied by a launch of its
own there, which the 4 rows per thread that such slices take do not need."""
import numpy as np
import pytest

from clspmv_mic_b200 import formats as F
from clspmv_mic_b200 import synth
from tests.gpu_util import assert_close, reference_y

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("split,launches", [("1", 1), ("0", 2)])
def test_switch_reaches_even_slices(monkeypatch, split, launches):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    monkeypatch.setenv("CLSPMV_SELL_SPLIT", split)
    coo = F.coo_matrix(*synth.laplacian_2d(40))
    dev = F.DeviceMatrix(F.coo2sell(coo, 32))
    dev.sell_plan()
    x = synth.x_vector(coo.shape[1])
    y = torch.zeros(coo.shape[0], device="cuda")
    n = F.launch_count()
    dev.spmv(torch.from_numpy(x).cuda(), y, 1.0, 0.0, variant="planned")
    assert F.launch_count() - n == launches
    ref, _, bound = reference_y(coo, x)
    assert_close(y.cpu().numpy(), ref, bound, split)
