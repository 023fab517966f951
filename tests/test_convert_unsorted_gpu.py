"""Device conversion of a COO that is not sorted: the host's status or, for
DIA / BDIA, its result, at row counts whose gaps between entries are long, and
in a time like that of the sorted COO."""
import time

import numpy as np
import pytest

from clspmv_mic_b200 import _abi
from clspmv_mic_b200 import formats as F
from tests.test_device_convert_gpu import check_pair

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


@pytest.mark.parametrize("h,step", [(40, 1), (5000, 33), (400_000, 4999)])
@pytest.mark.parametrize("order", ["shuffled", "reversed", "last_first"])
def test_statuses_and_diagonals_match_host(h, step, order):
    rng = np.random.default_rng(h)
    r = np.repeat(np.arange(0, h, step), 3)
    c = np.minimum(r + np.tile([0, 1, 5], r.size // 3), h - 1)
    v = np.arange(1, r.size + 1, dtype=np.float32)
    at = {"shuffled": rng.permutation(r.size), "reversed": np.arange(r.size)[::-1], "last_first": np.roll(np.arange(r.size), 1)}[order]
    coo = F.coo_matrix(h, h, r[at], c[at], v[at])
    for fmt, args in (("csr", ()), ("ell", ()), ("sell", ()), ("b4csr", (4, 4)), ("sbell", (4, 4)), ("dia", ()), ("bdia", ())):
        check_pair(fmt, coo, *args)


def test_takes_no_longer_than_sorted():
    """1M entries over 20M rows; filling the overlapping gaps took 200 times as long."""
    h, n = 20_000_000, 1_000_000
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    r = torch.randint(0, h, (n,), generator=g, device="cuda", dtype=torch.int32)

    def best(rows):
        dev = F.DeviceMatrix.from_device_arrays("coo", dict(width=h, height=h, nnz=n),
                                                dict(coo_row_id=rows, coo_col_id=rows, coo_data=torch.ones(n, device="cuda")))
        times, status = [], None
        for _ in range(5):
            torch.cuda.synchronize()
            t = time.perf_counter()
            status, out = F.device_convert_raw(dev, "csr")
            torch.cuda.synchronize()
            times.append(time.perf_counter() - t)
            if status == _abi.OK:
                F.lib().clspmv_device_free_csr_f32(__import__("ctypes").byref(out))
        return status, min(times)

    ok, sorted_s = best(r.sort().values)
    bad, unsorted_s = best(r)
    assert (ok, bad) == (_abi.OK, _abi.ERR_NOT_SORTED)
    assert unsorted_s <= 10 * sorted_s
