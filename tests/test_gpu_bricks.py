"""Blocks of the matrix whose elements are cut into bricks of 16, 8 or 4 voxels (csrc/pe.cu): single
voxels, part of a row, rows, planes and ragged ends, bit for bit the same elements as in the whole
matrix; and the projector's phases where an element's kept list needs several record arrays."""
import numpy as np
import pytest

from conftest import geometry, sysmat
from test_gpu_pe_phases import SYSTEMS

pytestmark = pytest.mark.gpu

# first detector, detectors, first voxel, voxels of a 30 x 17*9*4 matrix
BLOCKS = [(0, 1, 0, 1), (29, 1, 611, 1), (3, 2, 5, 7), (0, 30, 16, 2), (0, 30, 17, 17), (0, 30, 20, 40), (7, 3, 100, 400),
          (0, 30, 150, 9), (0, 30, 1, 611), (11, 16, 152, 307)]


@pytest.mark.parametrize("mode", [sysmat.MODE_REFERENCE, sysmat.MODE_PRECISE, sysmat.MODE_FP64, sysmat.MODE_LOCAL])
def test_blocks_equal_the_whole_matrix(gpu, mode):
    geo = geometry.mini(seed=12, rotated=True, layers=2, n_rot=8, nvox=(17, 9, 4), ncry=(6, 5))
    ctx = sysmat.Context(geo)
    full = gpu.empty((ctx.n_det, ctx.n_vox), dtype=gpu.float32, device="cuda")
    ctx.pe(full, rotation=3.0, mode=mode)
    for d0, nd, v0, nv in BLOCKS:
        out = gpu.full((nd, nv), -1.0, dtype=gpu.float32, device="cuda")
        ctx.pe(out, rotation=3.0, mode=mode, det_begin=d0, det_count=nd, vox_begin=v0, vox_count=nv)
        assert gpu.equal(out, full[d0:d0 + nd, v0:v0 + nv]), (d0, nd, v0, nv)


@pytest.mark.parametrize("name", ["dense holes", "dense layers", "no holes", "no collimator"])
def test_projector_value_equals_dense_product(gpu, name):
    """u^T A x as the gradient kernel's last entry, at kept lists of one and of several chunks: the
    precise elements are floats of FP64 sums (6e-8 each), the products all FP64."""
    geo = SYSTEMS[name][0]()
    ctx = sysmat.Context(geo)
    dense = gpu.empty((ctx.n_det, ctx.n_vox), dtype=gpu.float32, device="cuda")
    ctx.pe(dense, mode=sysmat.MODE_PRECISE)
    gen = gpu.Generator().manual_seed(3)
    x = gpu.rand(ctx.n_vox, generator=gen).cuda()
    u = gpu.rand(ctx.n_det, generator=gen).cuda()
    want = float(u.double() @ (dense.double() @ x.double()))
    got = float(ctx.vjp(x, u)[sysmat.THETA_N])
    assert abs(got - want) <= 1e-6 * abs(want)
