"""The gridding kernel's pixel walk at the orientations and sizes where its
FP32 row bounds, pair queue and replicas can go wrong: axis-aligned views (an
axis that does not vary along a row), views a hair off them (huge reciprocal
steps, where the FP64 bounds take over), map edges that are no multiple of the
tile, pixel steps from 0.25 to 1 voxel, more pairs than one queue, symmetry
records and half maps; against FP64 trilinear gridding of the context's own
spectra.

Tolerance: a coordinate is off by < 5e-6 voxel, so each corner weight by
< 1.5e-5 of 1; the sums' relative L2 error stays below that."""
import math

import numpy as np
import pytest

from bsoft_b200.plan import P_MAP, P_MAT, P_ORIGIN, P_PIXEL, P_SCALE, P_WEIGHT, ReconPlan

pytestmark = pytest.mark.gpu


def _rot(axis, a):
    c, s = math.cos(a), math.sin(a)
    i, j = [(1, 2), (2, 0), (0, 1)][axis]
    m = np.eye(3)
    m[i, i] = m[j, j] = c
    m[i, j], m[j, i] = -s, s
    return m


def _views(rng, P):
    fixed = [np.eye(3)]
    for axis in range(3):
        fixed += [_rot(axis, a) for a in (math.pi / 2, math.pi, math.pi / 4, 1e-3, 1e-5, 1e-8, math.pi / 2 - 1e-6)]
    q, _ = np.linalg.qr(rng.normal(size=(max(0, P - len(fixed)), 3, 3)))
    q *= np.linalg.det(q)[:, None, None]
    return np.concatenate([np.stack(fixed[:P]), q])


def _grid(F, mats, N, ft, scale, weight, halves):
    """FP64 trilinear sums (2, N, N, N) and weights of spectra in reference order."""
    k = np.fft.fftfreq(ft, 1.0 / ft)
    hh, kk = np.meshgrid(k, k, indexing="xy")
    v = np.zeros((2, N ** 3), complex)
    w = np.zeros((2, N ** 3))
    for f, R, half in zip(F, mats, halves):
        m = (R[:, :1] * hh.ravel() + R[:, 1:2] * kk.ravel()) * scale
        b = np.floor(m)
        r = m - b
        b = b.astype(int)
        for dz in (0, 1):
            for dy in (0, 1):
                for dx in (0, 1):
                    t = weight * (r[0] if dx else 1 - r[0]) * (r[1] if dy else 1 - r[1]) * (r[2] if dz else 1 - r[2])
                    i = (b[0] + dx) % N + N * ((b[1] + dy) % N + N * ((b[2] + dz) % N))
                    np.add.at(v[half], i, f.ravel() * t)
                    np.add.at(w[half], i, t)
    return v.reshape(2, N, N, N), w.reshape(2, N, N, N)


@pytest.mark.parametrize("N,ft,P,nmaps,sym", [
    (16, 32, 70, 1, "C1"),       # more than two batches of 32 particles, every tile reached by all
    (36, 128, 24, 2, "C1"),      # ragged tiles, step 0.28, half maps
    (50, 128, 22, 1, "C1"),
    (64, 64, 24, 1, "C1"),       # whole-voxel steps
    (32, 128, 30, 1, "D2"),      # step 0.25; four records a particle
    (8, 32, 40, 1, "C1"),        # one tile, all aliases
    (42, 128, 24, 2, "C1"),      # rows that are folded a voxel at a time, half maps
    (12, 32, 33, 1, "C1"),       # rows folded by fours, the last tile cut after one
])
def test_sums_match_fp64_gridding(N, ft, P, nmaps, sym):
    from bsoft_b200.recon import Reconstructor
    from bsoft_b200.symmetry import operators
    rng = np.random.default_rng(N + P)
    mats = _views(rng, P)
    rec = np.zeros((P, 32))
    rec[:, P_MAT:P_MAT + 9] = mats.reshape(P, 9)
    rec[:, P_ORIGIN:P_ORIGIN + 2] = N / 2
    rec[:, P_PIXEL] = 1.5
    rec[:, P_SCALE] = rec[:, P_WEIGHT] = 1
    rec[:, P_MAP] = np.arange(P) % 2
    plan = ReconPlan(n=N, ft=ft, map=N, map_sampling=1.5, hi_res=2 * 1.5 / math.sqrt(3), interp=2, ctf_action=0,
                     wiener=0.0, params=rec, nmaps=nmaps, resolution=1.5, symmetry=sym)
    images = rng.normal(size=(P, N, N)).astype(np.float32)
    with Reconstructor(plan) as r:
        F = r.spectra(images, rec)
        r.insert(images, rec)
        got = [r.accumulators(h) for h in range(nmaps)]
        r.reset()
        r.insert(images, rec)
        again = r.accumulators(0)
    ops = operators(sym)
    halves = [int(h) if nmaps == 2 else 0 for h in rec[:, P_MAP]]
    weight = 1.0 if ft == N else 1 / ((ft / N) ** 2 * 0.6)
    v, w = _grid([f for f in F for _ in ops], [S @ R for R in mats for S in ops], N, ft, N / ft, weight,
                 [h for h in halves for _ in ops])
    for h in range(nmaps):
        assert np.linalg.norm(got[h][0] - v[h]) < 1.5e-5 * np.linalg.norm(v[h])
        assert np.linalg.norm(got[h][1] - w[h]) < 1.5e-5 * np.linalg.norm(w[h])
    assert np.array_equal(again[0], got[0][0]) and np.array_equal(again[1], got[0][1])
