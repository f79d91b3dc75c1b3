"""Finished maps into device memory at any float: the transform's last pass
stores pairs of voxels, so a destination between pairs takes another way.  The
same voxels everywhere, and nothing beside the map is touched."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from bsoft_b200.plan import P_CTF, P_MAT, P_ORIGIN, P_PIXEL, P_SCALE, P_WEIGHT, ReconPlan  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [32, 50])
@pytest.mark.parametrize("offset", range(5))
@pytest.mark.parametrize("rescale", [False, True])
def test_map_lands_where_asked(N, offset, rescale):
    from bsoft_b200.recon import Reconstructor
    rng = np.random.default_rng(7)
    q, _ = np.linalg.qr(rng.normal(size=(12, 3, 3)))
    rec = np.zeros((12, 32))
    rec[:, P_MAT:P_MAT + 9] = (q * np.linalg.det(q)[:, None, None]).reshape(12, 9)
    rec[:, P_ORIGIN:P_ORIGIN + 2] = N / 2
    rec[:, P_PIXEL] = 1.5
    rec[:, P_SCALE] = rec[:, P_WEIGHT] = 1
    rec[:, P_CTF + 1] = -500.0
    plan = ReconPlan(n=N, ft=128, map=N, map_sampling=1.5, hi_res=1.0, interp=2, ctf_action=0, wiener=0.0, params=rec,
                     nmaps=1)
    buf = torch.full((N ** 3 + 8,), 3.5, dtype=torch.float32, device="cuda")
    with Reconstructor(plan) as r:
        r.insert(rng.normal(size=(12, N, N)).astype(np.float32), rec)
        if rescale:
            r.set_rescale(2.0, 5.0)
        ref = r.finish(0)
        r.finish(0, out=buf[offset:offset + N ** 3])
    got = buf.cpu().numpy()
    assert np.array_equal(got[offset:offset + N ** 3].reshape(N, N, N), ref)
    assert (got[:offset] == 3.5).all() and (got[offset + N ** 3:] == 3.5).all()
