"""The tensor-core products at each tile width that the dispatch takes: 128
columns (512 rows x 8320 columns), 64 (4096 x 512), and 16 for products that
would leave SMs without a block, with column counts that end inside a tile.
Forward and every gradient against the FP64 restatement, within 5e-3 of the
largest magnitude (the BF16 values of activations and gradients, as in
test_gpu_surrogate.py)."""
import importlib

import numpy as np
import pytest

from oracle.surrogate import MLPRef

pytestmark = pytest.mark.gpu
S = importlib.import_module("cliffs-src_gb300.surrogate")


@pytest.mark.parametrize("shape,batch", [((8, 512, 1, 8320), 512), ((8, 512, 2, 64), 4096), ((8, 128, 2, 200), 2048),
                                         ((8, 144, 1, 72), 144)])
def test_products_of_every_width(shape, batch):
    n_in, width, depth, n_out = shape
    net = S.MLP(n_in, width, depth, n_out, seed=5)
    rng = np.random.default_rng(6)
    x = rng.uniform(-1, 1, (batch, n_in)).astype(np.float32)
    t = rng.normal(size=(batch, n_out)).astype(np.float32)
    Ws, bs = net.weights()
    ref = MLPRef(Ws, bs, bf16=True)
    y, yr = net.predict(x), ref.forward(x.astype(np.float64))[-1]
    assert np.abs(y - yr).max() <= 5e-3 * np.abs(yr).max()
    loss, gW, gb = net.gradients(x, t)
    lr, rW, rb = ref.loss_and_grads(x.astype(np.float64), t.astype(np.float64))
    assert abs(loss - lr) <= 1e-3 * lr
    for l in range(depth + 1):
        assert np.abs(gW[l] - rW[l]).max() <= 5e-3 * np.abs(rW[l]).max(), l
        assert np.abs(gb[l] - rb[l]).max() <= 5e-3 * np.abs(rb[l]).max(), l
    net.close()
