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
