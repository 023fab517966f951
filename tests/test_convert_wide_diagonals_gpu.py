"""Device DIA / BDIA conversion of rows that are walked by windows of 32 entries:
row lengths around a window, repeated entries on both sides of its edge, rows
without entries, a few long rows among short ones. Byte for byte the host's,
in a time like that of narrow bands for the same bytes."""
import time

import numpy as np
import pytest

from clspmv_mic_b200 import formats as F
from tests.test_device_convert_gpu import check_pair

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def _band(n, nd, keep):
    r = np.repeat(np.arange(n), nd)
    c = r + np.tile(np.arange(nd) - nd // 2, n)
    ok = (c >= 0) & (c < n) & keep(r, c)
    return r[ok], c[ok]


@pytest.mark.parametrize("n,nd", [(45, 43), (64, 63), (65, 64), (200, 65), (1000, 97), (333, 400)])
@pytest.mark.parametrize("kind", ["full", "holes", "empty_rows", "repeats"])
def test_matches_host(n, nd, kind):
    rng = np.random.default_rng(n)
    keep = {"full": lambda r, c: np.full(r.size, True), "holes": lambda r, c: (r * 7 + c * 3) % 5 != 0,
            "empty_rows": lambda r, c: r % 3 != 1, "repeats": lambda r, c: np.full(r.size, True)}[kind]
    r, c = _band(n, nd, keep)
    if kind == "repeats":   # entries 30 .. 34 of a row twice or three times, so that a window ends inside a run of repeats
        at = np.arange(r.size) - np.searchsorted(r, r)
        times = np.where((at >= 30) & (at <= 34), 2 + (r + at) % 2, 1)
        r, c = np.repeat(r, times), np.repeat(c, times)
    coo = F.coo_matrix(n, n, r, c, rng.standard_normal(r.size).astype(np.float32))
    for fmt in ("dia", "bdia"):
        check_pair(fmt, coo, 32)
        check_pair(fmt, coo, 1)


@pytest.mark.parametrize("short", [1, 20])
def test_a_few_long_rows(short):
    n, nd = 1500, 300
    r, c = _band(n, nd, lambda r, c: (np.abs(r - 700) < 40) | (np.abs(c - r) <= short // 2))
    check_pair("dia", F.coo_matrix(n, n, r, c, np.arange(1, r.size + 1, dtype=np.float32)), 32)


def test_takes_as_long_as_narrow_bands():
    """30M entries on 3,001 diagonals took 10 times as long as on 30."""
    def us(n, nd):
        r = torch.arange(n, device="cuda").repeat_interleave(nd)
        c = r + (torch.arange(nd, device="cuda") - nd // 2).repeat(n)
        ok = (c >= 0) & (c < n)
        r, c = r[ok].int(), c[ok].int()
        dev = F.DeviceMatrix.from_device_arrays("coo", dict(width=n, height=n, nnz=r.numel()),
                                                dict(coo_row_id=r, coo_col_id=c, coo_data=torch.ones(r.numel(), device="cuda")))
        times = []
        for _ in range(7):
            torch.cuda.synchronize()
            t = time.perf_counter()
            F.device_convert(dev, "dia")
            torch.cuda.synchronize()
            times.append(time.perf_counter() - t)
        return min(times) * 1e6

    assert us(10_000, 3001) <= 5 * us(1_000_000, 30)
