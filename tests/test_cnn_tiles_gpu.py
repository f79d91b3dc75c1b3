"""The proposer's implicit GEMMs at the edges of their tiles: channel counts
that need padding (to 32) or take the 32-, 64- and 128-column tiles, the
largest and smallest image grids, batches from one image to more rows than
one tile, against the FP64 oracle.

Tolerances.  A product of two split operands keeps 16 bits and a sum its FP32
rounding, so an output is off by a few 2^-16 of the sum of its terms'
magnitudes per layer: 2e-3 of the values' scale, as for the default network.
A gradient changes with every ReLU whose input is within that of zero: of the
~1e5 inputs of a layer here a few flip, each 1 / sqrt(1e5) of a tensor's
norm: 1e-2 per tensor."""
import numpy as np
import pytest

from oracle import cnn_oracle as co

pytestmark = pytest.mark.gpu


def _inputs(box, ch, hid, B, seed):
    rng = np.random.default_rng(seed)
    parts = []
    for name, shape in co.layout(box, ch, hid):
        fan = int(np.prod(shape[1:])) if len(shape) > 1 else 1
        parts.append(rng.normal(scale=np.sqrt(2.0 / fan) if name.endswith(".W") else 0.1, size=shape).ravel())
    q, _ = np.linalg.qr(rng.normal(size=(B, 3, 3)))
    tgt = np.concatenate([q.reshape(B, 9), rng.uniform(-2, 2, (B, 2))], axis=1).astype(np.float32)
    return np.concatenate(parts).astype(np.float32), rng.normal(size=(B, box, box)).astype(np.float32), tgt


@pytest.mark.parametrize("box,ch,hid,B", [
    (64, (32, 64, 64, 128, 128, 128), 1024, 1),      # the default channels, fewest rows
    (64, (32, 64, 64, 128, 128, 128), 96, 33),       # one row more than the 32-row tile
    (64, (3, 33, 65, 40, 160, 31), 70, 5),           # everything padded
    (64, (64, 96, 128, 256, 32, 64), 33, 4),         # two blocks of first-layer channels, 96 and 256 columns
    (128, (8, 32, 16, 64, 16, 16), 32, 2),
    (256, (4, 8, 8, 8, 8, 8), 16, 1),                # first-layer rows of 128 pixels
    (512, (4, 4, 8, 8, 8, 8), 16, 1),                # and of 256: one row per patch
])
def test_network_matches_oracle(box, ch, hid, B):
    from bsoft_b200.cnn import Proposer
    w, imgs, tgt = _inputs(box, ch, hid, B, 11)
    with Proposer(box=box, channels=ch, hidden=hid, batch=8) as net:
        net.set_params(w)
        out = net.predict(imgs)
        loss, g = net.loss_grad(imgs, tgt)
        again = net.loss_grad(imgs, tgt)
    assert loss == again[0] and np.array_equal(g, again[1])
    R, t, L, go = co.forward_backward(w, imgs, tgt, box, ch, hid)
    assert np.abs(out[:, :9].reshape(-1, 3, 3) - R).max() < 2e-3
    assert np.abs(out[:, 9:] - t).max() < 2e-3 * max(1.0, np.abs(t).max())
    assert abs(loss - L) < 2e-3 * max(1.0, abs(L))
    off = 0
    for name, shape in co.layout(box, ch, hid):
        k = int(np.prod(shape))
        a, b = g[off:off + k].astype(np.float64), go[off:off + k]
        off += k
        assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b) + 1e-6, name


def test_predictions_do_not_depend_on_the_pass():
    """One image's pose is the same bits alone, in a small batch and in a
    pass of hundreds (other row tiles), on host and device buffers."""
    import torch
    from bsoft_b200.cnn import Proposer
    rng = np.random.default_rng(5)
    imgs = rng.normal(size=(300, 64, 64)).astype(np.float32)
    with Proposer(box=64, batch=16) as net:
        few = net.predict(imgs[:7])
        one = net.predict(imgs[3:4])
        many = net.predict(imgs)
        dev = torch.empty((300, 11), dtype=torch.float32, device="cuda")
        net.predict(torch.from_numpy(imgs).cuda(), out=dev)
    assert np.array_equal(few, many[:7]) and np.array_equal(one[0], many[3])
    assert np.array_equal(dev.cpu().numpy(), many)
