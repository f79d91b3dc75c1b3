"""Ewald-sphere insertion at strong curvature: surfaces that leave the plane by
many voxels reach tiles (and wrap-around aliases) that no pixel of the plane
itself comes near.  Every contribution counts: the weights against the FP64
oracle's, voxel by voxel.

Tolerance: a contribution's trilinear weight is formed in FP32 from tile-relative
coordinates below 100 voxels, each off by a few of their roundings (4e-6): < 1e-5
an axis, so < 3e-5 of the particle weight (0.42) a contribution.  A voxel that n
contributions reach sums to about n / 8 of it (0.05 n) and is off by less than
1.3e-5 n: within 3e-4 (1 + its weight).  A contribution that is left out is
missed by its own weight, up to 0.4."""
import numpy as np
import pytest

import oracle
from bsoft_b200.plan import P_CTF, P_MAT, P_ORIGIN, P_PIXEL, P_SCALE, P_WEIGHT, ReconPlan

pytestmark = pytest.mark.gpu


def _plan(N, lam, interp, views, nmaps=1):
    rng = np.random.default_rng(11)
    q, _ = np.linalg.qr(rng.normal(size=(views, 3, 3)))
    rec = np.zeros((views, 32))
    rec[:, P_MAT:P_MAT + 9] = (q * np.linalg.det(q)[:, None, None]).reshape(views, 9)
    rec[:, P_ORIGIN:P_ORIGIN + 2] = N / 2
    rec[:, P_PIXEL] = 0.5
    rec[:, P_SCALE] = rec[:, P_WEIGHT] = 1
    rec[:, P_CTF + 1] = -500.0
    rec[:, 26] = lam
    plan = ReconPlan(n=N, ft=2 * N, map=N, map_sampling=0.5, hi_res=0.5, interp=interp, ctf_action=0, wiener=0.0,
                     params=rec, nmaps=nmaps)
    return plan, rng.normal(size=(views, N, N)).astype(np.float32)


@pytest.mark.parametrize("lam", [0.1, 0.25, 0.5])          # 3, 8 and 16 voxels at the transform's corners
@pytest.mark.parametrize("shape", range(4))
def test_every_contribution_is_gridded(lam, shape):
    from bsoft_b200.recon import Reconstructor
    plan, images = _plan(64, lam, 2, 48)
    with Reconstructor(plan) as rec:
        rec.set_tile_shape(shape)
        rec.insert(images, plan.params)
        v, w = rec.accumulators(0)
    ov, ow, _, _ = oracle.insert(plan, images, plan.params)
    ow = ow.reshape(w.shape)
    assert (np.abs(w - ow) / (1 + ow)).max() < 3e-4
    ov = ov.view(np.complex128).reshape(v.shape)
    assert (np.abs(v - ov) / (1 + ow)).max() < 3e-4 * np.abs(images).sum(axis=(1, 2)).max() / 128


@pytest.mark.parametrize("interp", [0, 2])
def test_with_figure_of_merit_channels(interp):
    """The path with the FOM channels forms its coordinates in FP64, so nearest
    interpolation takes the oracle's voxels too."""
    from bsoft_b200.recon import Reconstructor
    plan, images = _plan(64, 0.5, interp, 48)
    with Reconstructor(plan, fom=True) as rec:
        rec.insert(images, plan.params)
        _, w = rec.accumulators(0)
    _, ow, _, _ = oracle.insert(plan, images, plan.params)
    ow = ow.reshape(w.shape)
    assert (np.abs(w - ow) / (1 + ow)).max() < 3e-4
