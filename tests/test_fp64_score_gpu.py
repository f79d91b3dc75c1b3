"""The FP64 figure of merit (padded-copy gather, phase tables) against the FP32
one (texture gather, sincos per pixel: other code on every step): kernel widths
that take the general gather, samplings whose sections reach beyond the padded
transform, origins with more distinct slopes than phase tables, one and many
groups, FRC and DPR.

Tolerance: the FP32 form sums ~1e4 FP32 products per figure in a fixed tree of
at most 5 + 40 additions a shell: < 1e-5 (its own bound against the reference
is 2e-5); the DPR's arctangents double it."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n,width,pixel,hi,norg", [
    (32, 32, 8, 1.5, 4.0, 1),
    (64, 64, 8, 1.5, 4.0, 9),        # a 3 x 3 grid: three slopes an axis
    (64, 64, 8, 1.5, 4.0, 25),       # scattered origins: sincos per pixel
    (64, 64, 6, 1.5, 4.0, 9),        # general gather
    (64, 64, 1, 1.5, 4.0, 4),
    (64, 64, 8, 0.8, 4.0, 9),        # particle sampling finer than the map's: positions far outside
    (32, 64, 8, 1.1, 5.0, 2),
])
@pytest.mark.parametrize("dpr", [False, True])
def test_fp64_equals_fp32_scores(N, n, width, pixel, hi, norg, dpr):
    from bsoft_b200.match import Matcher, ctf_record, hypothesis
    rng = np.random.default_rng(N + norg)
    q, _ = np.linalg.qr(rng.normal(size=(7, 3, 3)))
    q *= np.linalg.det(q)[:, None, None]
    q[0] = np.eye(3)
    g = np.arange(N) - N / 2
    vol = sum(np.exp(-((g[:, None, None] - a) ** 2 + (g[None, :, None] - b) ** 2 + (g[None, None, :] - c) ** 2) / 8)
              for a, b, c in rng.uniform(-N / 4, N / 4, (12, 3))).astype(np.float32)
    with Matcher(n=n, map=N, map_sampling=1.5, pixel=pixel, hi_res=hi, kernel_width=width) as m:
        m.set_reference(vol + 0.05 * rng.normal(size=vol.shape).astype(np.float32))
        m.set_images(rng.normal(size=(3, n, n)).astype(np.float32),
                     [ctf_record(200000.0, [-0.07, -600.0, 10.0, 5.0, 900.0]) for _ in range(3)])
        if norg == 9:
            org = [(n / 2 + dx, n / 2 + dy) for dy in (-.4, 0, .4) for dx in (-.4, 0, .4)]
        else:
            org = n / 2 + rng.uniform(-2, 2, (norg, 2))
        hyps = [hypothesis(i % 3, R, o) for i, R in enumerate(q) for o in org]
        f64, c64 = m.score(hyps, fp64=True, dpr=dpr)
        f32, c32 = m.score(hyps, dpr=dpr)
        again = m.score(hyps, fp64=True, dpr=dpr)
    tol = 2e-5 if dpr else 1e-5
    assert np.abs(f64 - f32).max() < tol and np.abs(c64 - c32).max() < tol
    assert np.any(f64 != 0)
    assert np.array_equal(f64, again[0]) and np.array_equal(c64, again[1])
