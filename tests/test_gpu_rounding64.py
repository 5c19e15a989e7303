"""The straight-line double reciprocal and root of csrc/rounding.cuh: a Newton step from a seed of 2^-22
squares the error twice, which leaves the last step's rounding, so they are at most one unit of the last
place from the IEEE results (tests/rounding64_check.cu, compiled here)."""
import os
import subprocess

import pytest

from conftest import PKG_DIR

pytestmark = pytest.mark.gpu


def test_double_helpers_are_within_one_ulp(gpu, tmp_path):
    exe = str(tmp_path / "rounding64_check")
    src = os.path.join(os.path.dirname(__file__), "rounding64_check.cu")
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", os.path.join(PKG_DIR, "csrc"), "-o", exe, src], check=True)
    rcp, root, error = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    assert int(rcp) <= 1 and int(root) <= 1 and error == "0", (rcp, root, error)
