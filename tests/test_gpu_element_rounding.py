"""The reference mode's element of a crystal that stands alone against the same float program written out one
rounding at a time (tests/element_rounding.cu, compiled here), bit for bit: crystal sizes whose sub-element
faces and centres do not fit a float, along each axis; and a thin plate in front, whose chord decides which
rays count."""
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


def _compare(gpu, program, collimator, pos, size, n, pitch, fov, plate):
    det = geometry._detector([pos], size, mu=MU)
    image = geometry._image(n, pitch, fov)
    geo = geometry.Geometry("alone", collimator, det, image, geometry._physics())
    out = gpu.empty((1, geo.n_vox), dtype=gpu.float32, device="cuda")
    sysmat.Context(geo).pe(out)
    voxels = [np.float32(i - m / 2 + 0.5) * p for z in range(n[2]) for y in range(n[1]) for x in range(n[0])
              for i, m, p in zip((x, y, z), n, np.float32(pitch))]
    pos = np.float32(pos)
    args = [pos[0], pos[1] + np.float32(fov), pos[2], *size, *MU, *plate, *voxels]
    bits = subprocess.run([program, *(repr(float(x)) for x in args)], check=True, capture_output=True, text=True).stdout
    return np.count_nonzero(out.cpu().numpy()[0].view(np.uint32) != np.array(bits.split(), dtype=np.uint32))


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_lone_crystal_equals_the_program_rounding_by_rounding(gpu, program, axis):
    for s in np.float32(SIZES):
        size = [2.0, 2.0, 2.0]
        size[axis] = float(s)
        none = np.zeros(geometry.N_COLLIMATOR, np.float32)
        assert _compare(gpu, program, none, POS, size, N, PITCH, FOV, [1, 0, 0, 0, 0, 0]) == 0, (axis, s)


@pytest.mark.parametrize("seed", range(6))
def test_thin_plate_equals_the_program_rounding_by_rounding(gpu, program, seed):
    rng = np.random.default_rng(seed)
    thickness = np.float32(rng.uniform(0.03, 0.098))       # chords of 0.1 mm at 13 to 73 degrees
    cb = geometry._CollimatorBuilder()
    cb.add_layer(80.0, thickness, 80.0, 0.0, 0.0, 0.0, 0.0, [])
    half = -thickness / np.float32(2.0)
    plate = [-40.0, half + np.float32(9.0), -40.0, 40.0, -half + np.float32(9.0), 40.0]
    pos = (rng.uniform(-15, 15), rng.uniform(3, 8), rng.uniform(-15, 15))
    assert _compare(gpu, program, cb.build(), pos, (2.0, 5.0, 2.0), (48, 2, 64), (0.53, 0.71, 0.47), 9.0, plate) == 0
