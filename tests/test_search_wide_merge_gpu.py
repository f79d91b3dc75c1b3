"""The merge of an exhaustive search whose sections x origins do not fit 32 bits
(128-bit candidates).  The origins in two halves, each within 32 bits, hold
every candidate between them: the best of both in (score descending, section,
origin) order are the wide merge's, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nimg", [1, 2])
def test_wide_merge_equals_halves(nimg):
    from bsoft_b200.match import Matcher, ctf_record
    rng = np.random.default_rng(9)
    nsec, norigin = 1 << 20, 4098
    assert nsec * norigin > (1 << 32) > nsec * (norigin // 2)
    q = rng.normal(size=(nsec, 4))
    q /= np.linalg.norm(q, axis=1)[:, None]
    w, x, y, z = q.T
    mats = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], axis=1)
    mats[1] = mats[0]                                      # equal scores: the section decides
    org = 16 + rng.uniform(-3, 3, (norigin, 2))
    org[norigin // 2:] = org[:norigin // 2]                # equal scores across the halves: the origin decides
    with Matcher(n=32, map=32, map_sampling=1.5, pixel=1.5, hi_res=9.0) as m:
        m.set_reference(rng.normal(size=(32, 32, 32)).astype(np.float32))
        m.set_panel(mats, exact_sections=False)
        m.set_images(rng.normal(size=(nimg, 32, 32)).astype(np.float32),
                     [ctf_record(200000.0, [-0.07, -400.0 - 9 * i, 0, 0, 500.0]) for i in range(nimg)])
        wide = m.search(org)
        half = norigin // 2
        first, second = m.search(org[:half]), m.search(org[half:])
    second[:, :, 1] += half
    for got, a, b in zip(wide, first, second):
        both = sorted(np.concatenate([a, b]).tolist(), key=lambda r: (-r[2], r[0], r[1]))[:8]
        assert sorted(got.tolist()) == sorted(both)
