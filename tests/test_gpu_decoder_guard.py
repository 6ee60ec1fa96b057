"""Infinite weights in the map decoder's direct kernels: what reaches an infinite
tap only through the zero padding stays as it is (0 times infinity is not a
number).  The 8-channel convolution, and the input gradients of each kind: 16, 8
and 4 channels a thread, and the map's level."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
S = importlib.import_module("cliffs-src_gb300.surrogate")


def _tap(w, o, tap, c, channels, value):
    """w [co][9 C] with the weight of output o, tap and input channel c set."""
    w = w.copy()
    w[o, tap * channels + c] = value
    return w


@pytest.mark.parametrize("level,ch", [(0, (16, 8, 8)), (1, (16, 16, 8)), (1, (16, 24, 8))])
def test_forward_of_an_eight_channel_level(level, ch):
    """Tap (0, 0) of the level's first row and column lies in the padding, and so does what the map's first row
    and column read."""
    net = S.MLP(9, 64, 1, 16, seed=8, map_side=32, map_ch=ch)
    rng = np.random.default_rng(8)
    l = net.layers() - 3 + level
    w, x = net.get(l, 0), rng.uniform(-1, 1, (16, 9)).astype(np.float32)
    maps = []
    for value in (np.inf, 0.0):
        net.set(l, 0, _tap(w, 3, 0, 5, ch[level], value))
        maps.append(net.predict(x)[:, 16:].reshape(16, 32, 32))
    assert not np.isfinite(maps[0][:, 4:, 4:]).all()
    for m in maps:
        assert np.isfinite(m[:, 0]).all() and np.isfinite(m[:, :, 0]).all()
    assert np.array_equal(maps[0][:, 0], maps[1][:, 0]) and np.array_equal(maps[0][:, :, 0], maps[1][:, :, 0])
    net.close()


@pytest.mark.parametrize("level,ch,side,batch", [
    (2, (16, 16, 8), 32, 16), (2, (16, 16, 16), 32, 16),  # the map's level
    (1, (16, 16, 8), 64, 96), (1, (16, 24, 8), 64, 96), (1, (16, 24, 8), 32, 16)])  # 16, 8 and 4 channels a thread
def test_input_gradients(level, ch, side, batch):
    """Weights, activations and output gradients above zero: an infinite tap makes the gradients of the level below
    infinite; one product of it with the padding would make them no number."""
    net = S.MLP(9, 64, 1, 16, seed=9, map_side=side, map_ch=ch)
    nd = net.layers() - 3
    for k in range(3):
        net.set(nd + k, 0, np.full(net.shape(nd + k), 0.01, np.float32))
        net.set(nd + k, 1, np.full(net.shape(nd + k)[0], 1.0, np.float32))
    net.set(nd + level, 0, _tap(net.get(nd + level, 0), 0, 0, 5, ch[level], np.inf))
    rng = np.random.default_rng(9)
    x = rng.uniform(-1, 1, (batch, 9)).astype(np.float32)
    t = np.full((batch, 16 + side * side), -1.0, np.float32)
    _, _, gb = net.gradients(x, t)
    assert np.isposinf(gb[nd + level - 1]).all(), gb[nd + level - 1]
    net.close()
