"""Local search: sections near a proposal, selected for one image or four per
CTA, a panel in one segment and in two, candidate lists that are empty, odd,
and longer than the kernel keeps.  Selection and scores do not depend on the
division, so batches of one image give the same bits; the number selected is
the FP64 trace's but for rounding of the FP32 one (nine products of at most 1:
below 2e-6)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rotations(rng, n):
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], axis=1).reshape(n, 3, 3)


@pytest.mark.parametrize("nimg,nsec,radius,norigin", [
    (1, 1, 180.0, 1),
    (1, 7, 180.0, 9),          # every section: odd
    (3, 33, 2.0, 4),           # mostly none
    (148, 700, 40.0, 5),       # the last size with one image per CTA
    (149, 700, 40.0, 5),       # four per CTA, a ragged last one
    (3, 131105, 3.0, 2),       # two segments
    (151, 131073, 4.0, 2),     # two segments, one section in the second
    (2, 3000, 180.0, 9),       # longer than the list
])
def test_selection_and_picks(nimg, nsec, radius, norigin):
    from bsoft_b200.match import Matcher, ctf_record
    rng = np.random.default_rng(nsec + nimg)
    mats = _rotations(rng, nsec)
    prop = np.zeros((nimg, 11), dtype=np.float32)
    prop[:, :9] = _rotations(rng, nimg).reshape(nimg, 9)
    prop[:, 9:] = rng.uniform(-0.5, 0.5, (nimg, 2))
    org = 16 + rng.uniform(-0.4, 0.4, (norigin, 2))
    images = rng.normal(size=(nimg, 32, 32)).astype(np.float32)
    ctf = [ctf_record(200000.0, [-0.07, -400.0 - 3 * i, 0, 0, 500.0]) for i in range(nimg)]
    vol = rng.normal(size=(32, 32, 32)).astype(np.float32)
    got, selected, whole = [], [], None
    for batch in (0, 1):
        with Matcher(n=32, map=32, map_sampling=1.5, pixel=1.5, hi_res=4.5, batch=batch) as m:
            m.set_reference(vol)
            m.set_panel(mats)
            m.set_images(images, ctf)
            m.reset_stats()
            got.append(m.search_local(prop, org, radius, 3.0, 8))
            selected.append(m.stats()["hypotheses"] / norigin)
            if radius == 180.0 and nsec <= 1024:
                whole = m.search(org)
    assert np.array_equal(got[0], got[1]) and selected[0] == selected[1]
    lo = hi = 0
    for i in range(nimg):
        t = mats.reshape(nsec, 9) @ prop[i, :9].astype(np.float64)
        bound = 1 + 2 * math.cos(math.radians(radius))
        lo += min(1024, int((t >= bound + 2e-6).sum()))
        hi += min(1024, int((t >= bound - 2e-6).sum()))
        for sec in got[0][i, :, 0].astype(int):
            assert sec < 0 or t[sec] >= bound - 2e-6
    assert lo <= selected[0] <= hi
    for r in got[0]:
        keys = [(int(s), int(o)) for s, o in r[:, :2] if s >= 0]
        assert len(set(keys)) == len(keys)
    if whole is not None:                  # every section: the search's best
        assert np.array_equal(got[0][:, 0, :2], whole[:, 0, :2])
        assert np.array_equal(got[0][:, 0, 3], whole[:, 0, 3])
