"""Device converters where their kernels change path: runs of empty rows of
every listed length, block rows cut into several items, ranges too long to
stage, arrays off a 16-byte boundary, alignments that leave strips off a
4-value boundary. Each result equals the host converter's, byte for byte.
Released arrays are kept for the next call, given back by device_trim, and
never handed out twice."""
import ctypes as C
import threading

import numpy as np
import pytest

from clspmv_mic_b200 import _abi
from clspmv_mic_b200 import formats as F
from tests.test_device_convert_gpu import check_pair, device_coo, host_raw

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

FORMATS = [("csr", ()), ("ell", ()), ("ell", (6, 0)), ("sell", (4,)), ("sell", (32,)), ("sell", (64,)), ("sell", (128,)),
           ("sell", (12,)), ("b4csr", (4, 4)), ("b4csr", (8, 8)), ("b4csr", (4, 1)), ("b4csr", (4, 2, 5)), ("b4ell", (4, 4)),
           ("b4ell", (8, 1)), ("b4ell", (4, 4, 5, 0)), ("sbell", (4, 4)), ("sbell", (8, 2)), ("sbell", (4, 8, 7))]


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def _rows(h, w, lens, seed):
    """Rows of the given lengths with sorted distinct columns."""
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(len(lens)), lens)
    cols = np.concatenate([np.sort(rng.choice(w, n, replace=False)) for n in lens if n] or [np.zeros(0, int)])
    return F.coo_matrix(h, w, rows, cols, rng.standard_normal(rows.size).astype(np.float32))


def _case(name):
    if name == "gaps":             # empty runs of 31, 32, 33, 64, 4095 .. 4097 and 9000 rows, and before and after
        at, lens = 0, {}
        for gap in (0, 31, 32, 33, 64, 4095, 4096, 4097, 9000):
            at += gap
            lens[at] = 3 + gap % 5
            at += 1
        h = at + 5000
        return _rows(h, 997, [lens.get(r, 0) for r in range(h)], 1)
    if name == "one_late_row":
        return _rows(20000, 501, [0] * 13000 + [7] + [0] * 6999, 2)
    if name == "long_rows":        # block rows of 513 .. 6000 entries beside short ones, skewed and even rows
        lens = [3] * 40 + [1500, 2, 0, 700] + [500] * 4 + [5] * 33 + [127, 128, 129, 130] + [1] * 10 + [2900]
        return _rows(len(lens), 3001, lens, 3)
    if name == "dense_rows":       # 32 rows hold more entries than are staged
        return _rows(130, 400, [100] * 130, 4)
    if name == "mixed":
        rng = np.random.default_rng(5)
        return _rows(1037, 1037, list(rng.integers(0, 40, 1037)), 6)
    raise KeyError(name)


@pytest.mark.parametrize("name", ["gaps", "one_late_row", "long_rows", "dense_rows", "mixed"])
@pytest.mark.parametrize("fmt,args", FORMATS)
def test_paths_match_host(name, fmt, args):
    check_pair(fmt, _case(name), *args)


@pytest.mark.parametrize("n,diagonals", [(31, 3), (33, 31), (127, 45), (4097, 27), (1000, 101)])
@pytest.mark.parametrize("align", [1, 6, 32])
def test_diagonals_match_host(n, diagonals, align):
    r = np.repeat(np.arange(n), diagonals)
    c = r + np.tile(np.arange(diagonals) - diagonals // 2, n)
    keep = (c >= 0) & (c < n) & ((r * 7 + c) % 11 != 0)
    coo = F.coo_matrix(n, n, r[keep], c[keep], np.arange(1, keep.sum() + 1, dtype=np.float32))
    for fmt in ("dia", "bdia"):
        check_pair(fmt, coo, align)


@pytest.mark.parametrize("fmt,args", [("csr", ()), ("dia", ()), ("ell", ()), ("sell", ()), ("b4csr", (4, 4)), ("sbell", (4, 4))])
def test_arrays_off_a_16_byte_boundary(fmt, args):
    coo = _case("mixed") if fmt != "dia" else F.coo_matrix(*__import__("clspmv_mic_b200.synth", fromlist=["x"]).banded(1003, 7))
    dev = device_coo(coo)
    t = {k: torch.cat([v[:1], v])[1:] for k, v in dev.tensors.items()}
    assert all(v.data_ptr() % 16 for v in t.values())
    off = F.DeviceMatrix.from_device_arrays("coo", dict(width=coo.shape[1], height=coo.shape[0], nnz=coo.nnz), t)
    got, (_, host) = F.device_convert(off, fmt, *args), host_raw(fmt, coo, *args)
    for field, _, _ in _abi.FORMATS[fmt][1]:
        assert np.array_equal(got.tensors[field].cpu().numpy().view(np.uint32), host.array(field).view(np.uint32)), field


def test_released_arrays_are_handed_out_once():
    """A struct freed through two copies of itself, and two threads converting
    and dropping at once: every result stays the host's."""
    coo = _case("mixed")
    st, out = F.device_convert_raw(device_coo(coo), "csr")
    assert st == _abi.OK
    twice = _abi.Csr.from_buffer_copy(out)
    F.lib().clspmv_device_free_csr_f32(C.byref(out))
    F.lib().clspmv_device_free_csr_f32(C.byref(twice))
    a, b = (F.device_convert(device_coo(coo), "csr") for _ in range(2))
    ptrs = [t.data_ptr() for m in (a, b) for t in m.tensors.values()]
    assert len(set(ptrs)) == len(ptrs)
    _, host = host_raw("sell", coo)
    wrong = []

    def work():
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            dev = device_coo(coo)
            for _ in range(20):
                m = F.device_convert(dev, "sell")
                if not np.array_equal(m.tensors["sell_data"].cpu().numpy(), host.array("sell_data")):
                    wrong.append(1)
                del m

    threads = [threading.Thread(target=work) for _ in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong
    F.device_trim()
    check_pair("sell", coo)
