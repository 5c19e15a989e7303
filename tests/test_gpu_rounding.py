"""The straight-line division, reciprocal and square root of csrc/rounding.cuh return the IEEE
results: every mantissa at several exponents, and 4e9 random quotients (tests/rounding_check.cu,
compiled here)."""
import os
import subprocess

import pytest

from conftest import PKG_DIR

pytestmark = pytest.mark.gpu


def test_rounding_helpers_equal_ieee(gpu, tmp_path):
    exe = str(tmp_path / "rounding_check")
    src = os.path.join(os.path.dirname(__file__), "rounding_check.cu")
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", os.path.join(PKG_DIR, "csrc"), "-o", exe, src], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["0", "0", "0", "0"], out
