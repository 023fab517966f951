"""The list of kept device arrays (csrc/device_pool.cu), compiled against a
stand-in for the CUDA calls it makes (compat/device_pool_check.cpp): no GPU.
An array that a device reset took away or that the caller freed is not handed
out and not freed again; the list's bounds and who leaves it hold; a release
waits for the device without spoiling another thread's stream capture; no
exception leaves a call when the host is out of memory; a matrix may be
released after the library's own destructors."""
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = tmp_path_factory.mktemp("pool") / "device_pool_check"
    src = ROOT / "tests" / "compat" / "device_pool_check.cpp"
    subprocess.run(["g++", "-std=c++17", "-g", "-fsanitize=address", f"-I{ROOT / 'include'}", f"-I{ROOT / 'clspmv_mic_b200' / 'csrc'}",
                    "-I/usr/local/cuda/include", str(src), "-o", str(exe), "-lpthread"], check=True)

    def run(name):
        res = subprocess.run([str(exe), name], capture_output=True, text=True, timeout=60)
        assert res.returncode == 0, res.stdout + res.stderr
    return run


@pytest.mark.parametrize("name", ["reuse", "bounds", "low_memory", "reset", "freed_by_the_caller", "waits", "capture", "host_memory", "at_exit"])
def test_kept_arrays(check, name):
    check(name)
