"""The back-projection kernel at the edges of its tiles and of the image: map
edges that are no multiple of 16 or smaller than it, axis-aligned views whose
samples fall on pixels, on the last row and column and outside, origins far
off, magnifications, half maps, against FP64 numpy of the reference's steps.

Tolerance: FP32 line transforms (~1e-6 of the filtered image's norm, twice)
and one FP32 rounding per image summed: < 5e-6 of the map's norm."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(images, rec, n, N, res, nmaps):
    k = np.arange(n)
    s = np.where(k > n // 2, n - k, k) / (n * 1.5)
    s2 = s[:, None] ** 2 + s[None, :] ** 2
    ramp = np.where(s2 > 1 / max(res, math.sqrt(2) * 1.5) ** 2, 0, np.sqrt(s2))
    g = np.arange(N) - N // 2
    maps = np.zeros((nmaps, N, N, N))
    for im, r in zip(images, rec):
        f = np.fft.ifft2(np.fft.fft2(im.astype(float)) * ramp).real
        f = (f - f.mean()) / f.std()
        out = ((k[None, :] - r[0]) / (n // 2)) ** 2 + ((k[:, None] - r[1]) / (n // 2)) ** 2 - 1 > 0
        fill = f[out].mean() if out.any() else 0.0
        m = r[2:11].reshape(3, 3) * r[11]
        X, Y = (m[0, c] * g[None, None, :] + m[1, c] * g[None, :, None] + m[2, c] * g[:, None, None] + r[c] for c in (0, 1))
        inside = (X >= 0) & (X < n) & (Y >= 0) & (Y < n)
        ix, iy = np.clip(X, 0, n - 1).astype(int), np.clip(Y, 0, n - 1).astype(int)
        fx, fy, lx, ly = X - ix, Y - iy, ix == n - 1, iy == n - 1
        jx, jy = np.minimum(ix + 1, n - 1), np.minimum(iy + 1, n - 1)
        w = [(1 - fx) * (1 - fy), np.where(lx, 0, fx * (1 - fy)), np.where(ly, 0, np.where(lx, fx, 1 - fx) * fy),
             np.where(lx | ly, 0, fx * fy)]
        v = w[0] * f[iy, ix] + w[1] * f[iy, jx] + w[2] * f[jy, ix] + w[3] * f[jy, jx]
        t = sum(w)
        maps[int(r[12])] += np.where(inside, np.where(t != 0, v / np.where(t != 0, t, 1), fill), fill)
    return maps


@pytest.mark.parametrize("n,N,nmaps,mag", [(16, 8, 1, 1.0), (30, 17, 2, 1.0), (64, 50, 1, 1.3), (60, 100, 2, 0.7),
                                           (128, 33, 1, 3.0)])
def test_maps_match_fp64(n, N, nmaps, mag):
    from bsoft_b200.backproj import BackProjector, BackprojPlan
    rng = np.random.default_rng(n + N)
    q, _ = np.linalg.qr(rng.normal(size=(70, 3, 3)))       # more images than one stage of parameters
    q[:3] = np.eye(3), [[0, -1, 0], [1, 0, 0], [0, 0, 1]], [[0, 0, 1], [0, 1, 0], [-1, 0, 0]]
    rec = np.zeros((70, 16))
    rec[:, 0:2] = n // 2 + rng.uniform(-2, 2, (70, 2))
    rec[:5, 0:2] = n // 2, n // 2
    rec[5, 0:2] = n - 1, 0
    rec[6, 0:2] = 3 * n, -n
    rec[:, 2:11] = q.reshape(70, 9)
    rec[:, 11] = mag
    rec[:, 12] = np.arange(70) % nmaps
    rec[:, 13] = 1.5
    images = rng.normal(size=(70, n, n)).astype(np.float32)
    plan = BackprojPlan(n=n, map=N, map_sampling=1.5, pixel=1.5, resolution=4.0, records=rec, nmaps=nmaps)
    with BackProjector(plan, batch=40) as bp:
        bp.add(images, rec)
        got = [bp.finish(i) for i in ([0] if nmaps == 1 else [1, 2])]
    for a, b in zip(got, _reference(images, rec, n, N, 4.0, nmaps)):
        assert np.linalg.norm(a - b) < 5e-6 * np.linalg.norm(b)
