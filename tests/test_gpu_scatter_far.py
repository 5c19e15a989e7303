"""Scatter into a small crystal far from the scatter point.  A voxel whose ray through the scatter point
crosses the crystal has theta_min = 0 (ScatterGen_RayTracing_CircularHole/scatter.cu:1321-1335), and with an
angular width below one step of the Riemann sum its only term is sin(0): the element is 0.  At 900 mm a
cosine's last bit is a tenth of a millimetre at the crystal, so a test of the scattering angle alone
cannot tell such a ray from one that passes by.  One hole, one 0.6 x 0.1 x 0.6 mm crystal, the voxels of
a plane that the hole projects over it."""
import numpy as np
import pytest

from conftest import geometry, oracle, sysmat

pytestmark = pytest.mark.gpu

HOLE, DISTANCE, N, PITCH, SIDE = 63.0, 900.0, 61, 0.0015, 0.6


def _system():
    cb = geometry._CollimatorBuilder()
    cb.add_layer(8.0, 4.0, 8.0, 0.0, 1.1, 0.9, 0.2, [(0.0, 0.0, 1.0)])
    det = geometry._detector([(0.0, DISTANCE, 0.0)], (SIDE, 0.1, SIDE))
    image = geometry._image((N, 1, N), (PITCH, PITCH, PITCH), HOLE)
    return geometry.Geometry("far", cb.build(), det, image, geometry._physics())


def test_rays_through_the_crystal_have_no_term(gpu):
    geo = _system()
    ctx = sysmat.Context(geo)
    bitmap = ctx.bitmap_collimator()
    ctx.scatter_prepare(None, bitmap, parts=sysmat.SCATTER_COLLIMATOR)
    out = gpu.empty((ctx.n_det, ctx.n_vox), dtype=gpu.float32, device="cuda")
    ctx.scatter(out, None, parts=sysmat.SCATTER_COLLIMATOR)
    a = out.cpu().numpy().reshape(N, N)                        # [z][x], one row of voxels in depth
    ref = oracle.scatter(geo, np.zeros((1, geo.n_vox), np.float32), "collimator", bitmap.cpu().numpy().view(np.uint32),
                         prec=64).reshape(N, N)
    # where a voxel's ray meets the crystal's depth, and how far inside its edges that is
    x = -(np.arange(N) - N / 2.0 + 0.5) * PITCH * DISTANCE / HOLE
    inside = 0.5 * SIDE - np.maximum(np.abs(x)[None, :], np.abs(x)[:, None])
    assert (ref[inside > 0.01] == 0.0).all() and (ref[inside < -0.3] > 0.0).all()
    assert (a[inside > 0.01] == 0.0).all(), (a[inside > 0.01] != 0.0).mean()
