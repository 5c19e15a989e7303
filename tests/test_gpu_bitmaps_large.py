"""Relationship bitmaps of systems whose per-object tables need more than 48 KB of shared memory (above
2457 crystals for the crystal bitmap, 3072 for the collimator one), against the oracle; and calls of
several such systems of different sizes at the same time."""
import threading

import numpy as np
import pytest

from conftest import geometry, oracle, sysmat

pytestmark = pytest.mark.gpu


def _subset(geo, ids):
    """The system of the crystals `ids` alone (12 floats each behind the count)."""
    det = np.zeros_like(geo.detector)
    det[0] = len(ids)
    for m, d in enumerate(ids):
        det[1 + 12 * m:13 + 12 * m] = geo.detector[1 + 12 * d:13 + 12 * d]
    return geometry.Geometry("subset", geo.collimator, det, geo.image, geo.physics)


def test_large_crystal_bitmap_equals_oracle_on_sampled_crystals(gpu):
    """A bit belongs to three crystals alone, so the bits of a subset's triples are the subset's bitmap."""
    geo = geometry.mini(seed=6, rotated=True, ncry=(50, 50), nholes=1)
    n = geo.n_det
    rng = np.random.default_rng(3)
    ids = np.unique(np.r_[0, 1, n - 2, n - 1, rng.choice(n, 44, replace=False)])
    bits = sysmat.Context(geo).bitmap_crystal()
    m = len(ids)
    i, j, k = np.meshgrid(np.arange(m), np.arange(m), np.arange(m), indexing="ij")
    upper = i < j
    i, j, k = i[upper].astype(np.int64), j[upper].astype(np.int64), k[upper].astype(np.int64)

    def flat(a, b, c, size):
        return (a * size - a * (a + 1) // 2 + b) * size + c
    big = gpu.from_numpy(flat(ids[i], ids[j], ids[k], n)).cuda()
    got = ((bits[big >> 5].long() >> (big & 31)) & 1).cpu().numpy()
    small = flat(i, j, k, m)
    want = (oracle.bitmap_crystal(_subset(geo, ids))[small >> 5].astype(np.int64) >> (small & 31)) & 1
    assert want.any() and not want.all()
    assert np.array_equal(got, want)


def test_systems_of_different_sizes_at_the_same_time(gpu):
    systems = [geometry.mini(seed=6, ncry=s, nholes=1) for s in ((56, 55), (64, 63), (81, 82))]
    want = [oracle.bitmap_collimator(g) for g in systems]
    failures = []

    def calls(geo, ref):
        try:
            ctx = sysmat.Context(geo)
            stream = gpu.cuda.Stream()
            with gpu.cuda.stream(stream):
                out = ctx.bitmap_collimator()
                for _ in range(3000):                     # bare calls: the threads meet inside the library
                    rc = sysmat.lib().sysmat_bitmap_collimator(ctx.handle, out.data_ptr(), stream.cuda_stream)
                    if rc:
                        failures.append(rc)
                        return
                stream.synchronize()
            if not np.array_equal(out.cpu().numpy().view(np.uint32), ref):
                failures.append("bits differ")
        except Exception as e:                            # the test's thread reports it
            failures.append(str(e))
    threads = [threading.Thread(target=calls, args=a) for a in zip(systems, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
