"""Calls that find the GPU's memory taken by others: what a smaller buffer or
another path can do is done, with the same results."""
import contextlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MB = 1 << 20


@contextlib.contextmanager
def _leave(nbytes):
    """All but about nbytes of the free device memory taken meanwhile, in as
    few pieces as the device gives it."""
    torch.cuda.empty_cache()
    taken, size = [], torch.cuda.mem_get_info()[0]
    while True:
        size = min(size, torch.cuda.mem_get_info()[0] - nbytes) // (2 * MB) * (2 * MB)
        if size <= 0:
            break
        try:
            taken.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            size //= 2
    try:
        yield
    finally:
        del taken
        torch.cuda.empty_cache()


def _matcher():
    from bsoft_b200.match import Matcher, ctf_record
    rng = np.random.default_rng(4)
    m = Matcher(n=128, map=128, map_sampling=1.5, pixel=1.5, hi_res=3.6)
    m.set_reference(rng.normal(size=(128, 128, 128)).astype(np.float32))
    m.set_images(rng.normal(size=(2, 128, 128)).astype(np.float32), [ctf_record(200000.0, [-0.07, -600.0, 0, 0, 900.0])] * 2)
    return m


def _hypotheses(n):
    from bsoft_b200.match import hypothesis
    q, _ = np.linalg.qr(np.random.default_rng(5).normal(size=(n, 3, 3)))
    return [hypothesis(i % 2, r * np.linalg.det(r), (64.3, 63.6)) for i, r in enumerate(q)]


def test_fp64_score_without_the_padded_copies():
    """The FP64 gather's padded copies (40 MB here) do not fit: the gather
    through the texture takes over (FP64 sums of 512 taps in another order:
    1e-12 of the figure)."""
    hyps = _hypotheses(27)
    with _matcher() as m:
        ref = m.score(hyps, fp64=True)                     # (loads the kernels, too)
    with _matcher() as m, _leave(24 * MB):
        got = m.score(hyps, fp64=True)
    assert np.abs(got[0] - ref[0]).max() < 1e-11 and np.abs(got[1] - ref[1]).max() < 1e-11


def test_repeated_fp64_scores_allocate_nothing():
    hyps = _hypotheses(60)
    with _matcher() as m:
        ref = m.score(hyps, fp64=True)
        with _leave(0):
            got = m.score(hyps, fp64=True)
            few = m.score(hyps[:3], fp64=True)
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
    assert np.array_equal(few[0], ref[0][:3])


def test_proposer_goes_back_to_its_batch():
    """The wide pass's activations fit, the copy of the host images beside
    them does not: passes of the context's batch give the same poses."""
    from bsoft_b200.cnn import Proposer
    images = np.random.default_rng(6).normal(size=(1024, 128, 128)).astype(np.float32)
    with Proposer(box=128, batch=8, seed=3) as p:
        free, _ = torch.cuda.mem_get_info()
        ref = p.predict(images)
        used = free - torch.cuda.mem_get_info()[0]
    assert used > 64 * MB                                  # (the images' copy alone)
    with Proposer(box=128, batch=8, seed=3) as p, _leave(used - 32 * MB):
        got = p.predict(images)
    assert np.array_equal(got, ref)


def test_failed_allocations_do_not_fail_the_next_call():
    """A call that ran out of memory leaves nothing behind for the next ones."""
    from bsoft_b200._lib import BsgError
    hyps = _hypotheses(3)
    with _matcher() as m:
        ref = m.score(hyps, fp64=True)
        with _leave(64 * MB), pytest.raises(BsgError):
            m.set_panel(np.tile(np.eye(3), (100000, 1, 1)))
        with _matcher() as other:
            got = other.score(hyps, fp64=True)
        again = m.score(hyps, fp64=True)
    assert np.array_equal(got[0], ref[0]) and np.array_equal(again[0], ref[0])


def test_gridding_without_replicas():
    """Without memory for the replicas' partial sums one warp grids a tile: the
    same contributions in one FP32 sum instead of several (1e-6 of the norm)."""
    from bsoft_b200.recon import Reconstructor
    from bsoft_b200.plan import P_CTF, P_MAT, P_ORIGIN, P_PIXEL, P_SCALE, P_WEIGHT, ReconPlan
    rng = np.random.default_rng(8)
    q, _ = np.linalg.qr(rng.normal(size=(60, 3, 3)))
    rec = np.zeros((60, 32))
    rec[:, P_MAT:P_MAT + 9] = (q * np.linalg.det(q)[:, None, None]).reshape(60, 9)
    rec[:, P_ORIGIN:P_ORIGIN + 2] = 64
    rec[:, P_PIXEL] = 1.5
    rec[:, P_SCALE] = rec[:, P_WEIGHT] = 1
    rec[:, P_CTF + 1] = -500.0
    plan = ReconPlan(n=128, ft=256, map=128, map_sampling=1.5, hi_res=1.0, interp=2, ctf_action=0, wiener=0.0, params=rec,
                     nmaps=1)
    images = rng.normal(size=(60, 128, 128)).astype(np.float32)
    free, _ = torch.cuda.mem_get_info()
    with Reconstructor(plan, batch=64) as r:
        used = free - torch.cuda.mem_get_info()[0]
        r.insert(images, rec)
        v, w = r.accumulators(0)
    assert used > 400 * MB                                 # 16 replicas of 25 MB among it
    with _leave(used - 200 * MB), Reconstructor(plan, batch=64) as r:
        r.insert(images, rec)
        v1, w1 = r.accumulators(0)
    assert np.linalg.norm(w1 - w) < 1e-6 * np.linalg.norm(w)
    assert np.linalg.norm((v1 - v).ravel()) < 1e-6 * np.linalg.norm(v.ravel())
