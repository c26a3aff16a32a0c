"""The activation's reciprocal against the IEEE division over every float of [1, inf]."""
import ctypes
import os
import subprocess

import pytest

from plugin_navierstokes_gb300 import build

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cuda", "recip_check.cu")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("recip") / "recip_check.so")
    cmd = [build.nvcc_path()] + build._flags() + ["-I", str(build.CSRC), "-shared", SRC, "-o", so]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return so


def test_compiles(lib):
    assert os.path.exists(lib)


@pytest.mark.gpu
def test_reciprocal(lib, cuda):
    out = (ctypes.c_uint * 3)()
    assert ctypes.CDLL(lib).recip_check(out) == 0
    different_bits, largest_ulp, nan = out
    assert different_bits == 0 and largest_ulp <= 1 and nan == 1
