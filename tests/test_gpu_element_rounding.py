"""The reference mode's element of a crystal that stands alone against the same float program written out one
rounding at a time (tests/element_rounding.cu, compiled here), bit for bit: crystal sizes whose sub-element
faces and centres do not fit a float, along each axis."""
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR, geometry, sysmat

pytestmark = pytest.mark.gpu

POS, FOV, MU = (np.float32(1.37), np.float32(6.1), np.float32(-2.2)), np.float32(30.0), (0.23, 0.18)
N, PITCH = (6, 5, 4), np.float32([0.5, 0.7, 0.9])
# the last four: thicknesses of which a face's offset from a voxel changes with its product's rounding
SIZES = [1.0, 1.6, 2.3, 2.75, 2.851720094680786, 1.2564748525619507, 2.064007520675659, 2.3938207626342773]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("element") / "element_rounding")
    src = os.path.join(os.path.dirname(__file__), "element_rounding.cu")
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe, src], check=True)
    return exe


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_lone_crystal_equals_the_program_rounding_by_rounding(gpu, program, axis):
    voxels = [np.float32(i - n / 2 + 0.5) * p for z in range(N[2]) for y in range(N[1]) for x in range(N[0])
              for i, n, p in zip((x, y, z), N, PITCH)]
    for s in np.float32(SIZES):
        size = [2.0, 2.0, 2.0]
        size[axis] = float(s)
        det = geometry._detector([POS], size, mu=MU)
        geo = geometry.Geometry("alone", np.zeros(geometry.N_COLLIMATOR, np.float32), det, geometry._image(N, PITCH, FOV),
                                geometry._physics())
        out = gpu.empty((1, geo.n_vox), dtype=gpu.float32, device="cuda")
        sysmat.Context(geo).pe(out)
        args = [POS[0], POS[1] + FOV, POS[2], *size, *MU, *voxels]
        bits = subprocess.run([program, *(repr(float(x)) for x in args)], check=True, capture_output=True, text=True).stdout
        assert np.array_equal(out.cpu().numpy()[0].view(np.uint32), np.array(bits.split(), dtype=np.uint32)), (axis, s)
