"""The map decoder's direct kernels (csrc/decoder.cuh) at the shapes where they
can go wrong: one cell and odd numbers of cells a side (a thread takes two), a
last run of cells that is nearly empty, the fewest and the most channels, and
channels that need several blocks of a weight gradient; and a weight that is not
finite, which must not leak through the zero padding."""
import importlib

import numpy as np
import pytest

from oracle.surrogate import MapNetRef

pytestmark = pytest.mark.gpu
S = importlib.import_module("cliffs-src_gb300.surrogate")


def _net(side, ch, seed):
    net = S.MLP(9, 64, 1, 16, seed=seed, map_side=side, map_ch=ch)
    rng = np.random.default_rng(seed)
    Ws, bs = net.weights()
    bs = [rng.normal(0, 0.05, b.shape).astype(np.float32) for b in bs]
    for l, b in enumerate(bs):
        net.set(l, 1, b)
    return net, rng, Ws, bs


@pytest.mark.parametrize("side,ch,batch", [(8, (8, 8, 8), 16), (24, (24, 40, 16), 16), (40, (64, 64, 8), 48),
                                           (56, (32, 24, 64), 16), (72, (64, 16, 8), 16)])
def test_decoder_shapes_against_oracle(side, ch, batch):
    """Forward and every gradient within 5e-3 of the largest magnitude: the BF16
    values of activations and gradients, as in test_gpu_surrogate.py."""
    net, rng, Ws, bs = _net(side, ch, 7)
    x = rng.uniform(-1, 1, (batch, 9)).astype(np.float32)
    t = rng.normal(0, 0.5, (batch, 16 + side * side)).astype(np.float32)
    ref = MapNetRef(Ws, bs, 16, side, ch[0], bf16=True)
    y, yr = net.predict(x), ref.forward(x.astype(np.float64))[-1]
    assert np.abs(y - yr).max() <= 5e-3 * np.abs(yr).max()
    loss, gW, gb = net.gradients(x, t)
    lr, rW, rb = ref.loss_and_grads(x.astype(np.float64), t.astype(np.float64))
    assert abs(loss - lr) <= 1e-3 * lr
    for l in range(net.layers()):
        assert np.abs(gW[l] - rW[l]).max() <= 5e-3 * np.abs(rW[l]).max(), l
        assert np.abs(gb[l] - rb[l]).max() <= 5e-3 * np.abs(rb[l]).max(), l
    net.close()


def test_infinite_weight_stays_off_the_padding():
    """The first row and column of the map read tap (0, 0) of the last level in
    the padding only: with an infinite weight there they keep their values."""
    net, rng, Ws, _ = _net(32, (16, 8, 8), 8)
    x = rng.uniform(-1, 1, (16, 9)).astype(np.float32)
    a = net.predict(x)[:, 16:].reshape(16, 32, 32)
    w = Ws[-1].copy()
    w[0, :8] = np.inf
    net.set(net.layers() - 1, 0, w)
    b = net.predict(x)[:, 16:].reshape(16, 32, 32)
    w[0, :8] = 0.0
    net.set(net.layers() - 1, 0, w)
    c = net.predict(x)[:, 16:].reshape(16, 32, 32)
    assert not np.isfinite(b[:, 1:, 1:]).all()
    assert np.array_equal(a[:, 0], b[:, 0]) and np.array_equal(a[:, :, 0], b[:, :, 0])
    assert np.array_equal(b[:, 0], c[:, 0]) and np.array_equal(b[:, :, 0], c[:, :, 0])
    net.close()
