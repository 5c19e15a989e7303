"""The pair tables' attenuator lists (csrc/scatter.cu): a pair's chords stay inside the list that was
sized for it, also when the list is shorter than the chords found (tests/pair_list_check.cu, compiled
here)."""
import os
import subprocess

import pytest

from conftest import PKG_DIR

pytestmark = pytest.mark.gpu


def test_lists_stay_inside_their_size(gpu, tmp_path):
    exe = str(tmp_path / "pair_list_check")
    src = os.path.join(os.path.dirname(__file__), "pair_list_check.cu")
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", os.path.join(PKG_DIR, "csrc"), "-o", exe, src], check=True)
    bad, chords, error = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    # of 6 crystals in a row, those strictly between each ordered pair: 2 (4 * 1 + 3 * 2 + 2 * 3 + 1 * 4)
    assert (bad, chords, error) == ("0", "40", "0")
