"""Relationship bitmaps at crystal counts whose rows do not fill 32-bit words (a word then holds the
end of one row and the start of others) and at a count that fills several words, bit for bit against
the oracle's restatement of the reference kernels."""
import numpy as np
import pytest

from conftest import geometry, oracle, sysmat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncry,nholes,rotated", [((1, 1), 1, False), ((2, 1), 3, True), ((5, 1), 2, True),
                                                 ((11, 3), 3, True), ((8, 8), 2, False), ((13, 7), 4, True)])
def test_bitmaps_equal_oracle(gpu, ncry, nholes, rotated):
    geo = geometry.mini(seed=6, rotated=rotated, ncry=ncry, nholes=nholes)
    ctx = sysmat.Context(geo)
    c = ctx.bitmap_crystal().cpu().numpy().view(np.uint32)
    h = ctx.bitmap_collimator().cpu().numpy().view(np.uint32)
    assert np.array_equal(c, oracle.bitmap_crystal(geo))
    assert np.array_equal(h, oracle.bitmap_collimator(geo))
