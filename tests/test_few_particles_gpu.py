"""Batches of a few particles, whose phase lattices and tile tests come from the
host, and the first sizes that take the kernel: sums against the FP64 oracle
(FP32 contributions rounded once, in sums of some tens: 1e-6 of the norm), half
maps, and spectra, which need neither."""
import numpy as np
import pytest

import oracle
from bsoft_b200.plan import P_CTF, P_MAP, P_MAT, P_ORIGIN, P_PIXEL, P_SCALE, P_WEIGHT, ReconPlan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [32, 50])
@pytest.mark.parametrize("P", [1, 2, 8, 9, 17])
@pytest.mark.parametrize("nmaps", [1, 2])
def test_sums_match_fp64(N, P, nmaps):
    from bsoft_b200.recon import Reconstructor
    rng = np.random.default_rng(N + P)
    q, _ = np.linalg.qr(rng.normal(size=(P, 3, 3)))
    q[0] = np.eye(3)
    rec = np.zeros((P, 32))
    rec[:, P_MAT:P_MAT + 9] = (q * np.linalg.det(q)[:, None, None]).reshape(P, 9)
    rec[:, P_ORIGIN:P_ORIGIN + 2] = N / 2 + rng.uniform(-1, 1, (P, 2))
    rec[:, P_PIXEL] = 1.5
    rec[:, P_SCALE] = rec[:, P_WEIGHT] = 1
    rec[:, P_CTF + 1] = -500.0
    rec[:, P_MAP] = np.arange(P) % nmaps
    plan = ReconPlan(n=N, ft=128, map=N, map_sampling=1.5, hi_res=1.0, interp=2, ctf_action=0, wiener=0.0, params=rec,
                     nmaps=nmaps)
    images = rng.normal(size=(P, N, N)).astype(np.float32)
    with Reconstructor(plan) as r:
        r.insert(images, rec)
        got = [r.accumulators(h) for h in range(nmaps)]
        first = r.spectra(images[:1], rec[:1])
        whole = r.spectra(images, rec)
    assert np.array_equal(first[0], whole[0])
    for h, (v, w) in enumerate(got):
        s = rec[:, P_MAP] == h
        ov, ow, _, _ = oracle.insert(plan, images[s], rec[s])
        assert np.linalg.norm(w.ravel() - ow) <= 1e-6 * np.linalg.norm(ow)
        assert np.linalg.norm(v.ravel() - ov.view(np.complex128)) <= 1e-6 * np.linalg.norm(ov)
