"""The smallest maps with every tile shape: 8^3 voxels are two tiles of 16 x 16 x 4
and one of the others.  Weights against the FP64 oracle (FP32 contributions,
each rounded once, in sums of some hundred: 1e-6 of the norm)."""
import numpy as np
import pytest

import oracle
from bsoft_b200.plan import P_CTF, P_MAT, P_ORIGIN, P_PIXEL, P_SCALE, P_WEIGHT, ReconPlan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [8, 10, 14])
@pytest.mark.parametrize("shape", range(4))
def test_sums_do_not_depend_on_the_shape(N, shape):
    from bsoft_b200.recon import Reconstructor
    rng = np.random.default_rng(N)
    q, _ = np.linalg.qr(rng.normal(size=(40, 3, 3)))
    rec = np.zeros((40, 32))
    rec[:, P_MAT:P_MAT + 9] = (q * np.linalg.det(q)[:, None, None]).reshape(40, 9)
    rec[:, P_ORIGIN:P_ORIGIN + 2] = N / 2
    rec[:, P_PIXEL] = 1.5
    rec[:, P_SCALE] = rec[:, P_WEIGHT] = 1
    rec[:, P_CTF + 1] = -500.0
    plan = ReconPlan(n=N, ft=32, map=N, map_sampling=1.5, hi_res=1.0, interp=2, ctf_action=0, wiener=0.0, params=rec,
                     nmaps=1)
    images = rng.normal(size=(40, N, N)).astype(np.float32)
    with Reconstructor(plan) as r:
        r.set_tile_shape(shape)
        for _ in range(2):                       # (the replicas' counters are back at zero)
            r.reset()
            r.insert(images, rec)
            v, w = r.accumulators(0)
    ov, ow, _, _ = oracle.insert(plan, images, rec)
    assert np.linalg.norm(w.ravel() - ow) < 1e-6 * np.linalg.norm(ow)
    assert np.linalg.norm(v.ravel() - ov.view(np.complex128)) < 1e-6 * np.linalg.norm(ov)
