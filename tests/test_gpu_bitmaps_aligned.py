"""Relationship bitmaps of crystals that lie behind one another but for offsets far below a micrometre, as
rotations and differences of computed positions leave them: directions then differ by less than any
approximate square root resolves; and of crystals in one place or in a hole's, which have no direction.  Every bit equals the
oracle's."""
import numpy as np
import pytest

from conftest import geometry, oracle, sysmat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0.0, 1e-20, 3e-18, 1e-15, 1e-9])
def test_bitmaps_of_aligned_crystals_equal_oracle(gpu, offset):
    cb = geometry._CollimatorBuilder()
    cb.add_layer(8.0, 4.0, 8.0, 0.0, 1.1, 0.9, 0.2, [(0.0, 0.0, 1.0), (2.0, -2.0, 0.5)])
    crystals = [(offset * (k % 3), 10.0 + 6.0 * k, -offset * (k % 2)) for k in range(9)]
    crystals += [(3.0, 20.0, 1.0), (3.0, 20.0, 1.0), (2.0, 0.0, -2.0)]
    det = geometry._detector(crystals, (1.0, 4.0, 1.0))
    geo = geometry.Geometry("aligned", cb.build(), det, geometry._image((2, 2, 1), (1, 1, 1), 40.0), geometry._physics())
    ctx = sysmat.Context(geo)
    want = oracle.bitmap_crystal(geo), oracle.bitmap_collimator(geo)
    assert want[0].any() and want[1].any()
    assert np.array_equal(ctx.bitmap_crystal().cpu().numpy().view(np.uint32), want[0])
    assert np.array_equal(ctx.bitmap_collimator().cpu().numpy().view(np.uint32), want[1])
