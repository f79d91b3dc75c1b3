"""The particle images' transforms over every box size (even and odd numbers of
stages), cut edges up to the whole transform and not multiples of the columns
per CTA, and batches of one and several images.  The transform is FP64 and each
value is rounded to float once: 2^-24 of the value, and the FP64 stages' own
error, below 1e-14 of the largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [32, 64, 128, 256, 512])
@pytest.mark.parametrize("hi_res", [3.0, 3.75, 9.3])
def test_cut_transforms(box, hi_res):
    from bsoft_b200.match import Matcher, ctf_record
    rng = np.random.default_rng(box)
    nimg = 5
    images = rng.normal(size=(nimg, box, box)).astype(np.float32)
    ctf = [ctf_record(200000.0, [-0.07, -400.0, 20.0, -9.0, 500.0]) for _ in range(nimg)]
    got = []
    for batch in (0, 2):
        with Matcher(n=box, map=box, map_sampling=1.5, pixel=1.5, hi_res=hi_res, batch=batch) as m:
            D = m.diam
            m.set_images(images, ctf, 0.0, 1.0)
            got.append(m.prepared())
    assert np.array_equal(got[0], got[1])
    i = np.arange(D)
    i = np.where(i > (D - 1) // 2, i + box - D, i)
    want = np.fft.fft2(images.astype(np.float64))[:, i][:, :, i]
    want[:, 0, 0] = 0
    err = np.abs(got[0] - want)
    assert (err <= 2.0 ** -23.5 * np.abs(want) + 1e-14 * np.abs(want).max()).all()
