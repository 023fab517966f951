"""Releasing a device matrix waits for the work that reads it, and leaves a
stream capture of another thread, or a relaxed one of this thread, intact."""
import threading

import numpy as np
import pytest

from clspmv_mic_b200 import formats as F
from clspmv_mic_b200 import synth
from tests.test_device_convert_gpu import device_coo

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def _converted():
    return F.device_convert(device_coo(F.coo_matrix(*synth.laplacian_2d(40))), "csr")


@pytest.mark.parametrize("mode,other_thread", [("thread_local", True), ("relaxed", True), ("relaxed", False)])
def test_capture_survives_a_release(mode, other_thread):
    keep, drop = _converted(), [_converted(), F.DeviceMatrix(F.coo2csr(F.coo_matrix(*synth.laplacian_2d(30))))]
    x, y, want = (torch.zeros(keep.shape[0], device="cuda") for _ in range(3))
    x.fill_(0.5)
    x[7] = 2.0
    keep.spmv(x, want, 1.0, 0.0)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode=mode):
        keep.spmv(x, y, 1.0, 0.0)
        if other_thread:
            t = threading.Thread(target=drop.clear)
            t.start()
            t.join()
        else:
            drop.clear()
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy(), want.cpu().numpy())


def test_release_waits_for_work_on_other_streams():
    m = _converted()
    s = torch.cuda.Stream()
    done = torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        torch.cuda._sleep(20_000_000)
        done.record()
    assert not done.query()
    del m
    assert done.query()
