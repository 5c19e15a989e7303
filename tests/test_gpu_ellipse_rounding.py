"""The float chord of elliptical holes is ill-conditioned in the fusion of its sums of products, which are
written out for that reason (csrc/geom.cuh): kernels that inline it in different code have the same chord.
The sampled form at the reference's sampling has the precise mode's contributions in another FP64 order,
so it is equal up to the output's float rounding, and so is the projection of each voxel."""
import numpy as np
import pytest

from conftest import geometry, sysmat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [71, 72])
def test_kernels_share_the_elliptical_chord(gpu, seed):
    geo = geometry.mini(seed=seed, rotated=True, layers=2, nvox=(6, 5, 3), ncry=(5, 4))
    H = geo.n_holes
    rng = np.random.default_rng(seed)
    r = geo.collimator[100:100 + 9 * H].reshape(H, 9)[:, 4].astype(np.float64)
    shapes = np.stack([r * rng.uniform(0.5, 1.0, H), r * rng.uniform(0.5, 1.0, H), rng.uniform(0.0, np.pi, H)], 1)
    ctx = sysmat.Context(geo)
    ctx.set_hole_shapes(shapes.astype(np.float32))
    a = gpu.empty((ctx.n_det, ctx.n_vox), dtype=gpu.float32, device="cuda")
    b = gpu.empty_like(a)
    ctx.pe(a, mode=sysmat.MODE_PRECISE)
    ctx.pe_sampled(b, (8, 16, 8), (1, 1, 1))
    a, b = a.cpu().numpy(), b.cpu().numpy()
    assert a.max() > 0
    assert np.allclose(b, a, rtol=2e-7, atol=0.0), np.abs(b / a - 1.0).max()
    for v in (0, 17, 41):
        x = gpu.zeros(ctx.n_vox, dtype=gpu.float32, device="cuda")
        x[v] = 1.0
        value = np.array([float(ctx.vjp(x, u)[sysmat.THETA_N]) for u in gpu.eye(ctx.n_det, device="cuda")])
        assert np.allclose(value, a[:, v], rtol=2e-7, atol=0.0), (v, np.abs(value / a[:, v] - 1.0).max())
