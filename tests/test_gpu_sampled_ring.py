"""The sampled form around a ring of crystals without a collimator (csrc/pe_ref.cuh): crystals on every
side of the voxels, so half the elements have no slope filter, and no hole or layer phase.  Divisions
with odd numbers and with the most that an axis and an element take, against the oracle's FP32 twin with
the tolerance of test_gpu_sampled.py, and the reference division against the precise mode."""
import math

import numpy as np
import pytest

from conftest import geometry, oracle, rel_err, sysmat

pytestmark = pytest.mark.gpu


def _ring():
    angles = 2.0 * math.pi * np.arange(24) / 24
    crystals = [(30.0 * math.sin(a), 30.0 * math.cos(a), z) for z in (-1.6, 1.6) for a in angles]
    det = geometry._detector(crystals, (2.0, 4.0, 2.0), rotations=np.tile(angles, 2))
    image = geometry._image((7, 6, 3), (1.5, 1.5, 1.5), 0.0, shift=(0.1, 0.2, 0.3))
    return geometry.Geometry("ring", np.zeros(geometry.N_COLLIMATOR, np.float32), det, image, geometry._physics())


def _sampled(torch, ctx, div, sub):
    out = torch.full((ctx.n_det, ctx.n_vox), -1.0, dtype=torch.float32, device="cuda")
    ctx.pe_sampled(out, div, sub)
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("div,sub", [((1, 1, 1), (1, 1, 1)), ((2, 8, 2), (1, 1, 1)), ((3, 5, 2), (2, 1, 1)),
                                     ((7, 1, 61), (1, 1, 1)), ((64, 8, 8), (1, 1, 1)), ((1, 64, 64), (1, 1, 1))])
def test_ring_matches_oracle(gpu, div, sub):
    geo = _ring()
    a = _sampled(gpu, sysmat.Context(geo), div, sub)
    ref = oracle.pe_sampled(geo, div, sub, prec=32)
    r = rel_err(a, ref)
    assert a.max() > 0
    assert np.median(r) < 1e-6, np.median(r)
    assert np.mean(r > 3e-5) <= 0.005, np.mean(r > 3e-5)
    assert r.max() < 1e-3, r.max()


def test_reference_division_is_the_precise_mode(gpu):
    ctx = sysmat.Context(_ring())
    a = gpu.empty((ctx.n_det, ctx.n_vox), dtype=gpu.float32, device="cuda")
    ctx.pe(a, mode=sysmat.MODE_PRECISE)
    b = _sampled(gpu, ctx, (8, 16, 8), (1, 1, 1))
    assert np.allclose(b, a.cpu().numpy(), rtol=2e-7, atol=0.0)
