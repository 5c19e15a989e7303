"""Grid scatter along paths that run along the holes but for offsets far below a micrometre (csrc/scatter_grid.cu,
seg_cyl64), past a hole whose wall is 1 um away: the path meets no part of the hole.  Against the double
definition in the oracle, within the 1e-5 of the largest element that the model is held to."""
import numpy as np
import pytest

from conftest import TOL, geometry, oracle, sysmat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("elliptical", [False, True])
@pytest.mark.parametrize("offset", [0.0, 1e-28, 1e-20, 3e-17, 1e-13, 1e-9])
def test_axial_paths_match_the_definition(gpu, offset, elliptical):
    cb = geometry._CollimatorBuilder()
    # 1 mm cells of a 3 x 4 x 3 mm plate: centres at x, z = -1, 0, 1; the wall of the hole at x = 0.001
    cb.add_layer(3.0, 4.0, 3.0, 0.0, 1.1, 0.9, 0.2, [(0.501, 0.0, 0.5)])
    det = geometry._detector([(offset, 9.0, 0.0)], (1.0, 4.0, 1.0))
    geo = geometry.Geometry("axial", cb.build(), det, geometry._image((2, 1, 1), (0.7, 1.0, 1.0), 30.0, shift=(0.0, 0.0, 0.2)),
                            geometry._physics())
    ctx = sysmat.Context(geo)
    shapes = [[0.5, 0.4, 0.0]] if elliptical else None
    if elliptical:
        ctx.set_hole_shapes(shapes)
    out = gpu.empty((ctx.n_det, ctx.n_vox), dtype=gpu.float32, device="cuda")
    ctx.scatter_grid(out, parts=sysmat.SCATTER_COLLIMATOR, cell=1.0)
    gpu.cuda.synchronize()
    ref = oracle.scatter_grid(geo, parts=2, cell=1.0, shapes=shapes)
    a = out.cpu().numpy().astype(np.float64)
    assert ref.max() > 0
    assert np.abs(a - ref).max() <= TOL * np.abs(ref).max(), (a, ref)
