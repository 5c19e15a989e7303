"""The projection gradient of elements whose kept objects fill several record arrays (csrc/pe_adjoint.cuh): the
partials, and those of the layer that is open at an array's end, are carried from one to the next.
Against central differences of the FP64 oracle with steps that the float parameters represent exactly: hole
centres are multiples of 1/2 below 8, so a step of 2^-20 along (-z, x), the tilt's, is a multiple of their last
bit.  Tolerance: the 1e-3 of test_gpu_adjoint.py, and 1e-4 of the largest geometric partial for those that
nearly cancel; a lost or exchanged carry changes a partial by a good part of itself."""
import numpy as np
import pytest

from conftest import geometry, oracle, sysmat

pytestmark = pytest.mark.gpu

H = 2.0 ** -20
SYSTEMS = {
    # layers, holes along a side, crystal centres, crystal size
    "layers": (3, 21, [(0.3, 18.5, -0.2), (1.1, 18.5, 0.9)], (7.5, 5.0, 7.5)),
    "holes": (1, 25, [(0.4, 9.0, 0.3), (-1.0, 9.0, 0.8)], (10.0, 5.0, 10.0)),
}


def _system(layers, side, crystals, size):
    rng = np.random.default_rng(1)
    cb = geometry._CollimatorBuilder()
    for m in range(layers):
        holes = [(x, z, 0.15 + 0.05 * rng.random()) for x, z, _ in geometry._square_holes(side, 0.5, 0.15)]
        cb.add_layer(24.0, 4.0, 24.0, 4.5 * m, 0.55, 0.4, 0.15, holes)
    image = geometry._image((2, 2, 1), (1.9, 2.1, 2.3), 40.0, shift=(0.13, -0.21, 0.17))
    return geometry.Geometry("dense", cb.build(), geometry._detector(crystals, size), image, geometry._physics())


def _with_holes(geo, edit):
    c = geo.collimator.copy()
    holes = c[100:100 + 9 * geo.n_holes].reshape(-1, 9)
    exact = holes.astype(np.float64)
    edit(exact)
    holes[:] = exact
    assert np.array_equal(holes.astype(np.float64), exact)
    return geometry.Geometry(geo.name, c, geo.detector, geo.image, geo.physics)


@pytest.mark.parametrize("elliptical", [False, True])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_gradient_over_several_record_arrays(gpu, name, elliptical):
    geo = _system(*SYSTEMS[name])
    ctx = sysmat.Context(geo)
    out = gpu.empty((ctx.n_det, ctx.n_vox), dtype=gpu.float32, device="cuda")
    counts = ctx.pe_work(out)
    assert counts["chunked"] == counts["elements"]       # 192 units there, 128 in the gradient
    shapes = None
    if elliptical:
        k = np.arange(geo.n_holes)
        r = geo.collimator[104:104 + 9 * geo.n_holes:9]
        shapes = np.stack([np.where(k % 2 == 0, 0.9 * r, 0.0), 0.7 * r, 0.3 + (0.37 * k) % 3.2], 1).astype(np.float32)
        ctx.set_hole_shapes(shapes)
    rng = np.random.default_rng(5)
    x = rng.uniform(0.5, 2.0, geo.n_vox).astype(np.float32)
    u = rng.uniform(0.5, 2.0, geo.n_det).astype(np.float32)
    got = ctx.vjp(gpu.from_numpy(x).cuda(), gpu.from_numpy(u).cuda()).cpu().numpy()

    def value(g, s=shapes):
        return float(u.astype(np.float64) @ oracle.pe(g, prec=64, shapes=s) @ x.astype(np.float64))

    def slope(side, step=H):
        return (value(*side(step)) - value(*side(-step))) / (2.0 * step)

    theta = geometry.theta_of(geo)

    def along(i):
        def side(h):
            t = theta.copy()
            t[i] += h
            g = geometry.apply_theta(geo, t)             # sets every radius to the mean one: keep the system's
            g.collimator[104:104 + 9 * geo.n_holes:9] = geo.collimator[104:104 + 9 * geo.n_holes:9]
            return g, shapes
        return side

    def radius(h):
        return _with_holes(geo, lambda a: a.__setitem__((slice(None), 4), a[:, 4] + h)), shapes

    def tilt(h):
        def edit(a):
            x0, z0 = a[:, 0].copy(), a[:, 3].copy()
            a[:, 0], a[:, 3] = x0 - h * z0, z0 + h * x0
        s = shapes
        if s is not None:
            s = s.copy()
            s[s[:, 0] > 0, 2] += np.float32(h)
        return _with_holes(geo, edit), s

    want = np.array([slope(along(0)), slope(along(1)), slope(radius), slope(along(3)), slope(along(4)), slope(along(5)),
                     slope(tilt)])
    assert abs(got[sysmat.THETA_N] - value(geo)) <= 1e-5 * value(geo)
    bound = 1e-3 * np.abs(want)
    bound[2:] += 1e-4 * np.abs(want[2:]).max()
    assert (np.abs(got[:sysmat.THETA_N] - want) <= bound).all(), (got, want)
