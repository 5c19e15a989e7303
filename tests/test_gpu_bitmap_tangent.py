"""The crystal bitmap where a crystal's cone touches another's: radii set so that the directions'
distance equals the radii's sum to the last few bits, on either side, seen from either end.  The
approximate directions of csrc/scatter.cu cannot decide these; every bit equals the oracle's."""
import numpy as np
import pytest

from conftest import geometry, oracle, sysmat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,shuffle", [(0, False), (1, True), (2, True)])
def test_tangent_cones_equal_oracle(gpu, seed, shuffle):
    geo = geometry.mini(seed=3, ncry=(10, 10), nholes=2)
    rng = np.random.default_rng(seed)
    det = geo.detector                                        # 12 floats per crystal: 1-3 centre, 4-6 size
    n = geo.n_det
    order = rng.permutation(n) if shuffle else np.arange(n)
    c = np.array([det[12 * k + 1:12 * k + 4] for k in range(n)], dtype=np.float64)
    c += rng.uniform(-0.3, 0.3, c.shape)
    c = c.astype(np.float32).astype(np.float64)
    size = np.full(n, 0.5)
    for j, i, k in order[:3 * (n // 3)].reshape(-1, 3):       # k touches i, seen from j
        v, w = c[k] - c[j], c[i] - c[j]
        lv, lw = np.linalg.norm(v), np.linalg.norm(w)
        gap = np.linalg.norm(v / lv - w / lw) - 0.5 * 0.5 * 3.0 ** 0.5 / lw
        if gap > 0.0:
            size[k] = 2.0 * gap * lv / 3.0 ** 0.5 * (1.0 + rng.integers(-8, 9) * 3e-8)
    for k in range(n):
        det[12 * k + 1:12 * k + 4] = c[k]
        det[12 * k + 4:12 * k + 7] = size[k]
    ctx = sysmat.Context(geo)
    assert np.array_equal(ctx.bitmap_crystal().cpu().numpy().view(np.uint32), oracle.bitmap_crystal(geo))
