"""The search's division of tiles on both sides of the line between short and
long panels (20 and 21 tiles of 256 sections), with row tiles in even groups,
groups of 21, seven and four, and runs that hold parts of several row tiles: as
in test_search_runs_gpu.py, how the work is cut changes no bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nimg,norigin,nsec", [
    (2, 25, 5120),      # 20 panel tiles: runs, one row tile
    (60, 25, 5120),     # 12 row tiles
    (150, 25, 5000),    # 30 row tiles, runs across row tiles
    (2, 25, 5121),      # 21: stretches, one row tile
    (60, 25, 5200),     # even groups
    (104, 25, 5377),    # a large group
    (165, 25, 9473),    # 33 row tiles: a large group and fours, 38 panel tiles
    (500, 9, 256),      # one panel tile
    (300, 25, 2000),    # few panel tiles, many row tiles
])
def test_divisions_agree(nimg, norigin, nsec):
    from bsoft_b200.match import Matcher, ctf_record
    rng = np.random.default_rng(nimg + nsec)
    q, _ = np.linalg.qr(rng.normal(size=(nsec, 3, 3)))
    q *= np.linalg.det(q)[:, None, None]
    images = rng.normal(size=(nimg, 32, 32)).astype(np.float32)
    ctf = [ctf_record(200000.0, [-0.07, -400.0 - 3 * i, 0, 0, 500.0]) for i in range(nimg)]
    org = 16 + rng.uniform(-2, 2, (norigin, 2))
    vol = rng.normal(size=(32, 32, 32)).astype(np.float32)
    got = []
    for batch in (0, 1, 7):
        with Matcher(n=32, map=32, map_sampling=1.5, pixel=1.5, hi_res=4.5, batch=batch) as m:
            m.set_reference(vol)
            m.set_panel(q)
            m.set_images(images, ctf)
            got.append(m.search(org))
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
