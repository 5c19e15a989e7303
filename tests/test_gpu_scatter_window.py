"""Scatter with an energy window that is open on one side or on both (infinite or the largest floats as
bounds), against the FP64 oracle with the tolerance of the fresh system in test_gpu_scatter.py."""
import numpy as np
import pytest

from conftest import TOL, geometry, oracle, rel_err, sysmat
from test_oracle import flip_explained

pytestmark = pytest.mark.gpu

MOST = float(np.finfo(np.float32).max)


@pytest.mark.parametrize("lo,hi", [(-np.inf, np.inf), (120.0, np.inf), (-np.inf, 135.0), (-MOST, MOST), (100.0, 1e20)])
def test_open_windows_match_fp64_oracle(gpu, lo, hi):
    base = geometry.mini(seed=21, rotated=True, nvox=(6, 6, 2), ncry=(5, 5))
    geo = geometry.Geometry("open window", base.collimator, base.detector, base.image, geometry._physics(lo=lo, hi=hi))
    ctx = sysmat.Context(geo)
    pe = gpu.empty((ctx.n_det, ctx.n_vox), dtype=gpu.float32, device="cuda")
    ctx.pe(pe)
    maps = ctx.bitmap_crystal(), ctx.bitmap_collimator()
    ctx.scatter_prepare(*maps)
    out = gpu.empty_like(pe)
    pe_h = pe.cpu().numpy()
    for parts, part, bm in ((1, "crystal", maps[0]), (2, "collimator", maps[1])):
        ctx.scatter(out, pe, parts=parts)
        a = out.cpu().numpy()
        bm = bm.cpu().numpy().view(np.uint32)
        ref = oracle.scatter(geo, pe_h, part, bm, prec=64)
        assert np.isfinite(a).all() and np.isfinite(ref).all() and ref.max() > 0
        r = rel_err(a, ref)
        assert np.mean(r > TOL) <= 0.01
        for d, v in np.argwhere(r > 1e-4):
            assert flip_explained(geo, pe_h, part, bm, int(d), int(v))
