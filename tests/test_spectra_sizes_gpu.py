"""The 2-D particle stage at every transform length and at image edges that
leave a line's last threads without pixels (odd, 2, the whole transform),
against FP64 numpy: background fill, padding, transform / ft, origin shift and
the CTF with its odd aberrations, every pixel and mate of the full plane.

Tolerance: 2 log2(ft) FP32 butterfly stages of ~0.6e-7 RMS each plus the
epilogue's products: < 2e-6 of the spectrum's norm (the bound of the
particle-spectrum tests)."""
import math

import numpy as np
import pytest

from bsoft_b200.plan import P_BKG, P_CTF, P_MAT, P_NORM, P_ORIGIN, P_PIXEL, P_SCALE, P_WEIGHT, ReconPlan

pytestmark = pytest.mark.gpu


def _reference(img, r, ft, action, wiener, hi_res):
    n = img.shape[0]
    v = img.astype(np.float64)
    if r[P_NORM]:
        v = (v * r[P_NORM] + r[P_NORM + 1]).astype(np.float32).astype(np.float64)
    g = np.arange(n)
    h = n // 2
    out = ((g[None, :] - r[P_BKG]) / h) ** 2 + ((g[:, None] - r[P_BKG + 1]) / h) ** 2 - 1 > 0
    pad = np.full((ft, ft), v[out].mean() if out.any() else 0.0)
    pad[:n, :n] = v
    F = np.fft.fft2(pad) / ft
    k = np.fft.fftfreq(ft, 1.0 / ft)
    kx, ky = np.meshgrid(k, k)
    F = F * np.exp(2j * math.pi / ft * (kx * r[P_ORIGIN] + ky * r[P_ORIGIN + 1]))
    if action:
        c = r[P_CTF:P_CTF + 7]
        sx, sy = kx / (ft * r[P_PIXEL]), ky / (ft * r[P_PIXEL])
        s2 = sx * sx + sy * sy
        chi = c[0] + c[1] * s2 + c[2] * (sx * sx - sy * sy) + c[3] * 2 * sx * sy + c[4] * s2 * s2
        w = np.sin(chi)
        if action == 1:
            w = np.where(w < 0, -1.0, 1.0)
        elif wiener:
            w = (wiener + 1) * w / (w * w + wiener)
        F = F * np.where(s2 <= 1 / hi_res ** 2, w, 0) * np.exp(-1j * (c[6] * sy + c[5] * sx))
    return F


@pytest.mark.parametrize("ft,n,action", [
    (32, 16, 1), (32, 2, 0), (32, 31, 2), (64, 33, 1), (64, 64, 4), (128, 63, 2), (128, 128, 0), (256, 100, 1),
    (256, 127, 4), (512, 256, 1), (512, 301, 2), (512, 7, 1), (1024, 384, 1), (1024, 513, 4), (1024, 1024, 2)])
def test_spectra_match_fp64(ft, n, action):
    from bsoft_b200.recon import Reconstructor
    rng = np.random.default_rng(ft + n)
    P = 3
    rec = np.zeros((P, 32))
    rec[:, P_MAT:P_MAT + 9] = np.eye(3).reshape(9)
    rec[:, P_ORIGIN:P_ORIGIN + 2] = n / 2 + rng.uniform(-3, 3, (P, 2))
    rec[:, P_BKG:P_BKG + 2] = [[0, 0], [n / 2, n / 2], [n / 3, 1]]
    rec[:, P_PIXEL] = 1.5
    rec[:, P_SCALE] = rec[:, P_WEIGHT] = 1
    rec[:, P_CTF:P_CTF + 7] = [-0.07, -900.0, 40.0, -25.0, 3000.0, 0, 0]
    rec[1, P_CTF + 5:P_CTF + 7] = 3.0, -2.0
    rec[2, P_NORM:P_NORM + 2] = 0.7, -0.2
    hi = 4.1
    wiener = 0.2 if action == 4 else 0.0
    plan = ReconPlan(n=n, ft=ft, map=32 if ft > 32 else 16, map_sampling=1.5, hi_res=hi, interp=2, ctf_action=action,
                     wiener=wiener, params=rec, resolution=1.5)
    images = rng.normal(size=(P, n, n)).astype(np.float32) + 0.5
    with Reconstructor(plan, batch=2) as r:
        got = r.spectra(images, rec)
    for i in range(P):
        ref = _reference(images[i], rec[i], ft, action, wiener, hi)
        assert np.linalg.norm(got[i] - ref) < 2e-6 * np.linalg.norm(ref), i
