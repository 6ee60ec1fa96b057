"""The map decoder's input gradient at each number of channels a thread takes
(16, 8 and, for the few cells of a small map or batch, 4): the gradients of every
layer are those of the FP64 restatement within 5e-3 of the largest magnitude (the
BF16 values of activations and gradients, as in test_gpu_surrogate.py)."""
import importlib

import numpy as np
import pytest

from oracle.surrogate import MapNetRef

pytestmark = pytest.mark.gpu
S = importlib.import_module("cliffs-src_gb300.surrogate")


@pytest.mark.parametrize("side,ch,batch", [(8, (64, 64, 64), 16), (16, (24, 16, 8), 16), (64, (16, 24, 8), 96)])
def test_gradients_of_every_group(side, ch, batch):
    net = S.MLP(9, 64, 1, 16, seed=3, map_side=side, map_ch=ch)
    rng = np.random.default_rng(3)
    Ws, bs = net.weights()
    x = rng.uniform(-1, 1, (batch, 9)).astype(np.float32)
    t = rng.normal(0, 0.5, (batch, 16 + side * side)).astype(np.float32)
    ref = MapNetRef(Ws, bs, 16, side, ch[0], bf16=True)
    _, gW, gb = net.gradients(x, t)
    _, rW, rb = ref.loss_and_grads(x.astype(np.float64), t.astype(np.float64))
    for l in range(net.layers()):
        assert np.abs(gW[l] - rW[l]).max() <= 5e-3 * np.abs(rW[l]).max(), l
        assert np.abs(gb[l] - rb[l]).max() <= 5e-3 * np.abs(rb[l]).max(), l
    net.close()
