"""CSR products with several right-hand sides where the rows, not the nonzeros,
are the work: mostly empty rows, rows of 2, few nonzeros. Against 64 bits for
every beta with rows of Y wider than k (whose rest stays as it is), and times
beside the same product without that work."""
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


def _host(h, filled, per, seed=1):
    """Rows of `per` entries, a share `filled` of them, the others empty."""
    rng = np.random.default_rng(seed)
    rows = np.nonzero(rng.random(h) < filled)[0]
    cols = (np.arange(per) * (h // per) + rng.integers(0, h // per, (rows.size, per))).reshape(-1)
    return F.coo_matrix(h, h, np.repeat(rows, per), cols, rng.standard_normal(cols.size).astype(np.float32))


def _device(h, filled, per):
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    rows = torch.nonzero(torch.rand(h, generator=g, device="cuda") < filled).flatten()
    col = torch.arange(per, device="cuda") * (h // per) + torch.randint(0, h // per, (rows.numel(), per), generator=g, device="cuda")
    coo = dict(coo_row_id=rows.repeat_interleave(per).int(), coo_col_id=col.flatten().int(),
               coo_data=torch.ones(rows.numel() * per, device="cuda"))
    return F.device_convert(F.DeviceMatrix.from_device_arrays("coo", dict(width=h, height=h, nnz=col.numel()), coo), "csr")


def _median_us(f):
    for _ in range(50):   # clocks and caches as in a stream of calls
        f()
    times = []
    for _ in range(21):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        for _ in range(10):
            f()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) * 100)
    return float(np.median(times))


def _us(m, k, beta):
    X, Y = (torch.rand((m.shape[0], k), device="cuda") for _ in range(2))
    return _median_us(lambda: m.spmm(X, Y, 0.5, beta))


@pytest.mark.parametrize("h,filled,per", [(1, 1, 1), (31, 0.5, 3), (257, 0.1, 9), (3001, 0.02, 40), (5000, 1, 2), (700, 0.5, 31)])
@pytest.mark.parametrize("k", [2, 5, 7, 8, 16, 36, 64, 128])
@pytest.mark.parametrize("value_type", ["f32", "bf16"])
def test_against_64_bits(h, filled, per, k, value_type):
    coo = _host(h, filled, per)
    dev = F.DeviceMatrix(F.coo2csr(coo))
    packed = None if value_type == "f32" else dev.pack(value_type)
    rng = np.random.default_rng(2)
    X = rng.uniform(-1, 1, (h, k)).astype(np.float32)
    Y0 = rng.uniform(-1, 1, (h, k + 4)).astype(np.float32)
    _, y64, scale = columns_reference(coo, X, 1.5)
    Xd = torch.from_numpy(X).cuda()
    for beta in (0.0, 0.5, 1.0):
        Y = torch.from_numpy(Y0).cuda()
        if beta == 0:
            Y[:, :k] = float("nan")
        dev.spmm(Xd, Y[:, :k], 1.5, beta, packed=packed)
        got = Y.cpu().numpy().astype(np.float64)
        lim = VALUE_RTOL[value_type] * (scale + beta * np.abs(Y0[:, :k])) + 1e-30
        assert (np.abs(got[:, :k] - (y64 + beta * Y0[:, :k])) <= lim).all(), beta
        assert (got[:, k:] == Y0[:, k:]).all()


def test_empty_rows_are_written_in_lines():
    """9 of 10 rows empty at k = 128: beta = 0, which has to write them, took 8.8 times as long as beta = 1, which does not."""
    m = _device(1 << 20, 0.1, 8)
    assert _us(m, 128, 0.0) <= 4 * _us(m, 128, 1.0)


def test_rows_do_not_wait_for_their_y():
    """2^20 rows of 2 at k = 36: beta = 1, without a pass of its own, took 1.31 times as long as beta = 0."""
    m = _device(1 << 20, 1, 2)
    assert _us(m, 36, 1.0) <= 1.15 * _us(m, 36, 0.0)


def test_few_nonzeros_take_more_warps():
    """5,000 rows of 3: k = 128 took 1.8 times as long as k = 16."""
    m = _device(5000, 1, 3)
    first, second = ([_us(m, k, 0.0) for k in (128, 16)] for _ in range(2))   # of calls this short the best of two
    assert min(first[0], second[0]) <= 1.45 * min(first[1], second[1])


@pytest.mark.parametrize("h,per,k", [(30_000, 47, 12), (20_000, 9, 36), (60_000, 20, 5)])
def test_beta_costs_no_more_than_a_pass_over_y(h, per, k):
    """beta = 0.5 beside beta = 1 and a scaling of Y: rows that wait for their Y took up to 1.8 times as long."""
    m = _device(h, 1, per)
    Y = torch.rand((h, k), device="cuda")

    def scaled():
        Y.mul_(0.5)
        m.spmm(X, Y, 0.5, 1.0)

    X = torch.rand((h, k), device="cuda")
    assert _us(m, k, 0.5) <= 1.2 * _median_us(scaled)
