"""A program that resets its device between calls (compat/device_reset_check.cpp):
uploads get arrays that exist, A^k x in one launch has its limits raised again."""
import subprocess

import pytest

from clspmv_mic_b200 import _abi
from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["upload", "iterate"])
def test_calls_after_a_device_reset(tmp_path, what):
    exe = tmp_path / "device_reset_check"
    subprocess.run(["g++", "-std=c++17", f"-I{ROOT / 'include'}", "-I/usr/local/cuda/include",
                    str(ROOT / "tests" / "compat" / "device_reset_check.cpp"), "-o", str(exe), "-L/usr/local/cuda/lib64",
                    "-lcudart_static", "-ldl", "-lrt", "-lpthread"], check=True)
    res = subprocess.run([str(exe), str(_abi.LIB_PATH), what], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, res.stdout + res.stderr
