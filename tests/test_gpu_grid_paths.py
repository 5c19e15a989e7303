"""Paths of the grid scatter model where its work is split: rotated crystals (the general chord) and
unrotated ones (the path's own reciprocals), several layers, chunks that mix crystal and septal cells,
one voxel and more than a pass of voxels, one detector and more than a tile.  Against the double
definition in the oracle, within the 1e-5 of the largest element that the model is held to."""
import numpy as np
import pytest

from conftest import TOL, geometry, oracle, sysmat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rotated,layers,ncry,nvox,parts", [(False, 1, (3, 3), (1, 1, 1), 3), (True, 2, (3, 2), (2, 1, 1), 3),
                                                            (False, 1, (1, 1), (7, 7, 1), 3), (True, 1, (6, 6), (3, 1, 1), 1),
                                                            (False, 2, (2, 2), (5, 1, 1), 2)])
def test_grid_matches_the_definition(gpu, rotated, layers, ncry, nvox, parts):
    geo = geometry.mini(seed=8, rotated=rotated, layers=layers, ncry=ncry, nvox=nvox, nholes=3)
    ctx = sysmat.Context(geo)
    out = gpu.empty((ctx.n_det, ctx.n_vox), dtype=gpu.float32, device="cuda")
    ctx.scatter_grid(out, parts=parts, cell=1.0)
    gpu.cuda.synchronize()
    ref = oracle.scatter_grid(geo, parts=parts, cell=1.0)
    a = out.cpu().numpy().astype(np.float64)
    assert ref.max() > 0
    assert np.abs(a - ref).max() <= TOL * np.abs(ref).max()
