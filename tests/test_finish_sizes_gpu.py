"""The finish (weighing, 3-D inverse transform, sinc, half-map FSC) at map
edges that take every radix, more rows than a tile and fewer, against FP64
numpy on the context's own accumulators.

Tolerance: the weighed values are rounded to FP32 once and pass three FP32
transforms of at most five stages each, ~1 ulp (6e-8) a stage: 15 x 6e-8 in
the worst case, < 1e-6 of the map's norm.  The FSC is FP64 sums of products of
the FP32 weighed values: 1e-6 covers their rounding (6e-8 per value)."""
import math

import numpy as np
import pytest

from bsoft_b200.plan import P_CTF, P_MAP, P_MAT, P_ORIGIN, P_PIXEL, P_SCALE, P_WEIGHT, ReconPlan

pytestmark = pytest.mark.gpu


def _context(N, fom=False, interp=2, nmaps=2, P=24, seed=3):
    from bsoft_b200.recon import Reconstructor
    rng = np.random.default_rng(seed)
    rec = np.zeros((P, 32))
    q, _ = np.linalg.qr(rng.normal(size=(P, 3, 3)))
    rec[:, P_MAT:P_MAT + 9] = (q * np.linalg.det(q)[:, None, None]).reshape(P, 9)
    rec[:, P_ORIGIN:P_ORIGIN + 2] = N / 2 + rng.uniform(-1, 1, (P, 2))
    rec[:, P_PIXEL] = 1.5
    rec[:, P_SCALE] = rec[:, P_WEIGHT] = 1
    rec[:, P_CTF + 1] = -500.0
    rec[:, P_MAP] = np.arange(P) % 2
    ft = 32
    while ft < 2 * N and ft < 1024:
        ft *= 2
    plan = ReconPlan(n=N, ft=ft, map=N, map_sampling=1.5, hi_res=2 * 1.5 / math.sqrt(3), interp=interp, ctf_action=1,
                     wiener=0.0, params=rec, nmaps=nmaps, resolution=1.5)
    r = Reconstructor(plan, fom=fom)
    r.insert(rng.normal(size=(P, N, N)).astype(np.float32), rec)
    return r


def _weigh(v, w):
    return np.where(w > 1e-30, v / np.where(w > 1e-30, w, 1), 0)


def _map(F, sinc):
    N = F.shape[0]
    g = np.arange(N)
    odd = (g[:, None, None] + g[None, :, None] + g[None, None, :]) % 2
    m = np.fft.ifftn(F * (1 - 2 * odd)).real * math.sqrt(N ** 3)
    if sinc:
        d = (g - N // 2) / N
        a = math.pi * np.sqrt(d[:, None, None] ** 2 + d[None, :, None] ** 2 + d[None, None, :] ** 2)
        m *= np.where(a > 0, a / np.where(a > 0, np.sin(a), 1), 1) ** 2
    return m


def _fsc(F1, F2, n, maxrad):
    N = F1.shape[0]
    f = np.abs(np.fft.fftfreq(N) * N)
    rad = np.sqrt(f[:, None, None] ** 2 + f[None, :, None] ** 2 + f[None, None, :] ** 2).ravel()
    lo = rad.astype(int)
    ok = lo < maxrad
    s = np.zeros((3, 2 * N))
    for q, t in enumerate(((F1 * F2.conj()).real, np.abs(F1) ** 2, np.abs(F2) ** 2)):
        t = t.ravel()[ok]
        np.add.at(s[q], lo[ok], t * (1 - (rad - lo)[ok]))
        np.add.at(s[q], lo[ok] + 1, t * (rad - lo)[ok])
    with np.errstate(all="ignore"):
        out = np.nan_to_num(s[0] / np.sqrt(s[1] * s[2]), nan=0.0, posinf=0.0, neginf=0.0)
    out[0] = 1
    out[maxrad:] = 0
    return out[:n]


# 8 = 8 (and 4), 10 = 5 2, 14 = 7 2, 18 = 6 3, 32 = 8 4, 36 = 6 6, 50, 70, 98 = 7 7 2,
# 100, 126 = 7 6 3, 144, 162 = 6 3 3 3, 128, 192, 256
@pytest.mark.parametrize("N", [8, 10, 14, 18, 32, 36, 50, 70, 98, 100, 126, 128, 144, 162, 192, 256])
def test_finish_and_fsc_match_fp64(N):
    with _context(N) as r:
        halves = [_weigh(*r.accumulators(h)) for h in (0, 1)]
        both = _weigh(*(a + b for a, b in zip(r.accumulators(0), r.accumulators(1))))
        got = [r.finish(0), r.finish(1), r.finish(2, sinc=False)]
        fsc = r.fsc()
        again = r.fsc(N)
    for g, F, sinc in zip(got, (both, *halves), (True, True, False)):
        ref = _map(F, sinc)
        assert np.linalg.norm(g - ref) < 1e-6 * np.linalg.norm(ref)
    maxrad = int(N * 1.5 / (2 * 1.5 / math.sqrt(3)))
    ref = _fsc(*halves, N, maxrad)
    assert np.abs(again - ref).max() < 1e-6
    assert np.array_equal(fsc, again[:N // 2])


@pytest.mark.parametrize("N", [48, 512])
def test_largest_and_full_map(N):
    """The largest edge (half-space sums), and full-map sums with the SNR
    channels (nearest interpolation)."""
    if N == 512:
        with _context(N, nmaps=1, P=3) as r:
            got, F = r.finish(0), _weigh(*r.accumulators(0))
        ref = _map(F, True)
        assert np.linalg.norm(got - ref) < 1e-6 * np.linalg.norm(ref)
        return
    with _context(N, fom=True, interp=0) as r:
        got, fom = r.finish(1, with_fom=True)
        F = _weigh(*r.accumulators(0))
    ref = _map(F, False)
    assert np.linalg.norm(got - ref) < 1e-6 * np.linalg.norm(ref)
    assert np.isfinite(fom).all() and fom.ravel()[0] == 1
