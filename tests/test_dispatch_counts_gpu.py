"""What launch counts and addresses tell of the dispatch: small CSR / COO
products take one launch up to their limits and two past them, released arrays
come back and are given back; and the blocks of a block row that is cut into
several items, between repeats of one entry."""
import numpy as np
import pytest

from clspmv_mic_b200 import formats as F
from tests.gpu_util import assert_close, reference_y
from tests.test_device_convert_gpu import check_pair, device_coo

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


@pytest.mark.parametrize("rows,nnz,launches", [(100, 1, 1), (4000, 32768, 1), (4000, 32769, 2), (32768, 32768, 1), (32769, 32769, 2)])
@pytest.mark.parametrize("fmt", ["csr", "coo"])
def test_small_products(fmt, rows, nnz, launches):
    rng = np.random.default_rng(nnz)
    r = np.sort(rng.integers(0, rows, nnz))
    c = np.arange(nnz) - np.searchsorted(r, r)
    coo = F.coo_matrix(rows, 200, r, c, rng.standard_normal(nnz).astype(np.float32))
    dev = F.DeviceMatrix(F.coo2csr(coo) if fmt == "csr" else coo)
    if fmt == "csr":
        dev.chunk_plan()
    x, y0 = (rng.uniform(-1, 1, n).astype(np.float32) for n in (200, rows))
    for beta, want in ((0.0, launches), (-0.5, launches), (1.0, 1)):
        y = torch.from_numpy(y0).cuda()
        n = F.launch_count()
        dev.spmv(torch.from_numpy(x).cuda(), y, 2.0, beta)
        assert F.launch_count() - n == want, beta
        ref, _, bound = reference_y(coo, x, y0, 2.0, beta)
        assert_close(y.cpu().numpy(), ref, bound, f"{fmt} {beta}")


def test_released_arrays_come_back_and_are_given_back():
    n = 1 << 21
    r = torch.arange(n, device="cuda", dtype=torch.int32)
    coo = F.DeviceMatrix.from_device_arrays("coo", dict(width=n, height=n, nnz=n),
                                            dict(coo_row_id=r, coo_col_id=r, coo_data=torch.ones(n, device="cuda")))
    F.device_trim()
    first = F.device_convert(coo, "csr")
    ptrs = {t.data_ptr() for t in first.tensors.values()}
    del first
    again = F.device_convert(coo, "csr")
    assert {t.data_ptr() for t in again.tensors.values()} == ptrs
    del again
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    F.device_trim()
    assert torch.cuda.mem_get_info()[0] - before >= 20 << 20   # three arrays of 8 MB


def test_released_arrays_stay_within_their_share():
    n = 50_000_000   # 200 MB an array, 600 MB a matrix
    r = torch.arange(n, device="cuda", dtype=torch.int32)
    coo = F.DeviceMatrix.from_device_arrays("coo", dict(width=n, height=n, nnz=n),
                                            dict(coo_row_id=r, coo_col_id=r, coo_data=torch.ones(n, device="cuda")))
    F.device_trim()
    mats = [F.device_convert(coo, "csr") for _ in range(8)]
    torch.cuda.synchronize()
    held, total = torch.cuda.mem_get_info()
    del mats
    torch.cuda.synchronize()
    freed = torch.cuda.mem_get_info()[0] - held
    assert 8 * 3 * 4 * n - freed <= total // 64 + (64 << 20)   # what is kept, and slack for the driver's pages
    F.device_trim()


@pytest.mark.parametrize("fmt,args", [("b4csr", (4, 4)), ("b4csr", (8, 1)), ("b4ell", (4, 2)), ("sbell", (4, 4)), ("sbell", (8, 2))])
@pytest.mark.parametrize("width", [97, 2000])
def test_repeats_where_a_block_row_is_cut(fmt, args, width):
    """Rows of 700 to 1,900 entries, every entry up to 5 times, so that each cut lies beside or between repeats."""
    rng = np.random.default_rng(width)
    rows, cols = [], []
    for row, length in enumerate([1900, 700, 0, 1300, 1024, 513, 512, 1800, 3]):
        c = np.sort(rng.integers(0, width, length // 3))
        c = np.repeat(c, rng.integers(1, 6, c.size))
        rows.append(np.full(c.size, row))
        cols.append(c)
    r, c = np.concatenate(rows), np.concatenate(cols)
    check_pair(fmt, F.coo_matrix(9, width, r, c, np.arange(1, r.size + 1, dtype=np.float32)), *args)
