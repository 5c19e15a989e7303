"""The local mode where a ray runs level with the plates: the voxel at the depth of a layer of sub-elements,
beside the plate.  Its path in the plate's frame is infinite (thickness over cosine), so the ray
contributes nothing; the other layers of sub-elements do.  Against the FP64 oracle."""
import numpy as np
import pytest

from conftest import TOL, geometry, oracle, rel_err, sysmat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [sysmat.MODE_LOCAL, sysmat.MODE_FP64])
@pytest.mark.parametrize("depth", [0.125, 0.25, 1.875])
def test_level_rays_match_fp64_oracle(gpu, mode, depth):
    cb = geometry._CollimatorBuilder()
    cb.add_layer(8.0, 4.0, 24.0, 0.0, 0.002, 0.001, 0.001, [])
    # sub-element depths at odd multiples of 1/8 mm from the crystals' centres
    det = geometry._detector([(20.0, depth, 0.1), (20.0, depth, 3.3)], (2.0, 4.0, 2.0))
    geo = geometry.Geometry("level", cb.build(), det, geometry._image((1, 1, 3), (1.0, 1.0, 1.3), 0.0, shift=(-10.0, 0.0, 0.07)),
                            geometry._physics())
    ctx = sysmat.Context(geo)
    out = gpu.empty((ctx.n_det, ctx.n_vox), dtype=gpu.float32, device="cuda")
    ctx.pe(out, mode=mode)
    ref = oracle.pe(geo, prec=64)
    r = rel_err(out.cpu().numpy(), ref)
    assert ref.min() > 0
    assert r.max() <= TOL, r
