"""Grid scatter of stacked plates whose holes reach beyond their plates and are filled: a path that ends on a
plate's face, as from a point at another plate's middle, is not inside it, and its holes do not count.
Against the double definition in the oracle, within the 1e-5 of the largest element that the model is held
to."""
import numpy as np
import pytest

from conftest import TOL, geometry, oracle, sysmat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("thickness,offset", [(0.05, 0.025), (0.3, 0.15)])
def test_paths_that_end_on_a_plate(gpu, thickness, offset):
    cb = geometry._CollimatorBuilder()
    holes = [(x, z, 0.5) for x in (-1.3, 0.0, 1.3) for z in (-1.3, 0.0, 1.3)]
    cb.add_layer(12.0, thickness, 12.0, 0.0, 0.85, 0.5, 0.3, holes)
    cb.add_layer(10.0, 6.0 * thickness, 10.0, offset, 1.1, 0.9, 0.2, holes)
    col = cb.build()
    h = col[100:100 + 9 * 18].reshape(18, 9)
    rng = np.random.default_rng(4)
    h[:, 1] -= rng.uniform(0.1, 1.0, 18)                       # caps
    h[:, 2] += rng.uniform(0.1, 1.0, 18)
    h[:, 5] = rng.uniform(0.0, 0.5, 18)                        # what fills them
    h[:, 6], h[:, 7] = 0.5 * h[:, 5], 0.3 * h[:, 5]
    det = geometry._detector([(0.0, 30.0, 0.0), (15.0, 26.0, 1.0)], (1.0, 2.0, 0.3))
    image = geometry._image((4, 3, 2), (-2.0, -0.5, -0.5), 0.0, shift=(-1.0, 0.125, -1.0))
    geo = geometry.Geometry("plates", col, det, image, geometry._physics())
    ctx = sysmat.Context(geo)
    out = gpu.empty((ctx.n_det, ctx.n_vox), dtype=gpu.float32, device="cuda")
    ctx.scatter_grid(out, parts=sysmat.SCATTER_COLLIMATOR, cell=3.0)
    ref = oracle.scatter_grid(geo, parts=2, cell=3.0)
    assert ref.max() > 0
    assert np.abs(out.cpu().numpy() - ref).max() <= TOL * ref.max()


@pytest.mark.parametrize("exchanged", [False, True])
def test_level_paths(gpu, exchanged):
    """Voxels at the depth of the plate's middle: their paths to its cells run level, and are inside the
    holes whose first cap is the lower one."""
    cb = geometry._CollimatorBuilder()
    cb.add_layer(14.0, 0.5, 14.0, 0.0, 0.2, 0.1, 0.1, [(x, z, 0.6) for x in (-3.0, 0.0, 3.0) for z in (-3.0, 0.0, 3.0)])
    col = cb.build()
    if exchanged:
        h = col[100:100 + 9 * 9].reshape(9, 9)
        h[::2, 1], h[::2, 2] = h[::2, 2].copy(), h[::2, 1].copy()
    det = geometry._detector([(0.3, 9.0, -0.4), (3.0, 9.0, 1.0)], (1.0, 2.0, 1.0))
    geo = geometry.Geometry("level", col, det, geometry._image((3, 1, 2), (1.9, 1.0, 2.3), 0.0, shift=(0.2, 0.0, -0.3)),
                            geometry._physics(lo=40.0))
    ctx = sysmat.Context(geo)
    out = gpu.empty((ctx.n_det, ctx.n_vox), dtype=gpu.float32, device="cuda")
    ctx.scatter_grid(out, parts=sysmat.SCATTER_COLLIMATOR, cell=1.0)
    ref = oracle.scatter_grid(geo, parts=2, cell=1.0)
    assert ref.min() > 0
    assert np.abs(out.cpu().numpy() - ref).max() <= TOL * ref.max()
