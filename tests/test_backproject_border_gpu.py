"""Back-projection where samples fall exactly on the image's border: there the
last bit of a coordinate decides between a pixel and the background, so the
coordinates are the reference's products and sums, one by one.  Rotations by
quarter turns about each axis, as cos and sin give them (6e-17 where the exact
matrix has 0), and views on a grid of angles, against the FP64 numpy of the
reference's steps.

Tolerance: as in test_backproject_edges_gpu.py, 5e-6 of the map's norm; one
border row taken for background is off by about 1e-2 of it."""
import math

import numpy as np
import pytest

from tests.test_backproject_edges_gpu import _reference

pytestmark = pytest.mark.gpu


def _turn(axis, deg):
    c, s = math.cos(math.radians(deg)), math.sin(math.radians(deg))
    i, j = [(1, 2), (2, 0), (0, 1)][axis]
    m = np.eye(3)
    m[i, i] = m[j, j] = c
    m[i, j], m[j, i] = -s, s
    return m


@pytest.mark.parametrize("n,N,mag", [(128, 128, 1.0), (64, 64, 1.0), (60, 50, 1.0), (64, 32, 2.0), (32, 64, 0.5)])
def test_border_samples_match_fp64(n, N, mag):
    from bsoft_b200.backproj import BackProjector, BackprojPlan
    from bsoft_b200.geometry import view_to_matrix
    rng = np.random.default_rng(n + N)
    mats = [_turn(a, d) for a in range(3) for d in (90, -90, 180)]
    for th in range(0, 181, 30):
        for ph in range(0, 360, 60):
            t, p = math.radians(th), math.radians(ph)
            v = (math.sin(t) * math.cos(p), math.sin(t) * math.sin(p), math.cos(t))
            mats += [view_to_matrix((*v, math.radians(a))) for a in (0, 90)]
    for m in mats[:9]:                         # one image at a time, so that none hides another
        _compare(BackProjector, BackprojPlan, rng, n, N, mag, [m])
    _compare(BackProjector, BackprojPlan, rng, n, N, mag, mats)


def _compare(BackProjector, BackprojPlan, rng, n, N, mag, mats):
    rec = np.zeros((len(mats), 16))
    rec[:, 0:2] = n // 2
    rec[:, 2:11] = np.asarray(mats).reshape(-1, 9)
    rec[:, 11] = mag
    rec[:, 13] = 1.5
    images = rng.normal(size=(len(mats), n, n)).astype(np.float32)
    plan = BackprojPlan(n=n, map=N, map_sampling=1.5, pixel=1.5, resolution=4.0, records=rec, nmaps=1)
    with BackProjector(plan) as bp:
        bp.add(images, rec)
        got = bp.finish(0)
    ref, = _reference(images, rec, n, N, 4.0, 1)
    assert np.linalg.norm(got - ref) < 5e-6 * np.linalg.norm(ref)
