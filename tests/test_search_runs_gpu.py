"""The search's division of row tiles and panel tiles over the SMs: batches of
one to 53 row tiles (even groups, groups of 21, 7 and 4, a ragged last batch),
panels of one to several tiles, merges of few and many candidates.  How the
work is cut changes no bit, so every division gives the one-image batches'
result, and the best candidate's correlation is the FP64 one's to BF16 rounding
(tested elsewhere)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nimg,norigin,nsec", [
    (1, 1, 5),         # one tile of each
    (7, 25, 700),      # two row tiles, three panel tiles
    (96, 25, 700),     # 19 row tiles
    (104, 25, 1100),   # 21: one large group
    (128, 25, 700),    # 25: a large group and a four
    (270, 25, 1500),   # 53: two large groups, a seven, a four
    (12, 49, 3000),    # many candidates an image
    (5, 25, 38000),    # one row tile over every SM, more panel tiles than stretches
    (150, 9, 300),     # merges of two CTAs per SM
])
def test_divisions_agree(nimg, norigin, nsec):
    from bsoft_b200.match import Matcher, ctf_record
    rng = np.random.default_rng(nimg)
    q, _ = np.linalg.qr(rng.normal(size=(nsec, 3, 3)))
    q *= np.linalg.det(q)[:, None, None]
    images = rng.normal(size=(nimg, 32, 32)).astype(np.float32)
    ctf = [ctf_record(200000.0, [-0.07, -400.0 - 3 * i, 0, 0, 500.0]) for i in range(nimg)]
    org = 16 + rng.uniform(-2, 2, (norigin, 2))
    vol = rng.normal(size=(32, 32, 32)).astype(np.float32)
    got = []
    for batch in (0, 1, 5):
        with Matcher(n=32, map=32, map_sampling=1.5, pixel=1.5, hi_res=4.5, batch=batch) as m:
            m.set_reference(vol)
            m.set_panel(q)
            m.set_images(images, ctf)
            got.append(m.search(org))
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    for r in got[0]:                       # distinct candidates (section -1: fewer than eight exist)
        key = (r[:, 0] * norigin + r[:, 1])[r[:, 0] >= 0]
        assert len(set(key)) == len(key) == min(8, nsec * norigin)
