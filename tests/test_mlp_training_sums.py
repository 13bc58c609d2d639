"""The training step's ordered sums and in-place packing: after training, both packed images hold
the trained weights (inference and gradient equal those of a solver given the weights afresh, bit for
bit) and training is reproducible, at batch sizes around the tiles of 32 rows, the blocks of 256 and the chunks of 64 partial rows."""
import ctypes

import numpy as np
import pytest

from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import from_scene

pytestmark = pytest.mark.gpu


def gradient(s, feat, target):
    g = np.empty(abi.MLP_PARAMS, np.float32)
    loss = ctypes.c_float()
    fp = ctypes.POINTER(ctypes.c_float)
    s._call("lsp_mlp_gradient", feat.ctypes.data_as(fp), target.ctypes.data_as(fp), feat.shape[0], g.ctypes.data_as(fp),
            ctypes.byref(loss))
    return loss.value, g


def recorded(seed):
    sc = scenes.small_box_scene(n_side=(12, 14, 12), seed=seed)
    s = from_scene(sc)
    s.mlp_record(True)
    for _ in range(3):
        s.update(sc.dt)
    return s


@pytest.mark.parametrize("batch", [1, 31, 33, 256, 257, 1000, 2016])
def test_trained_images_hold_the_weights(batch):
    a, b, c = recorded(3), recorded(3), recorded(3)
    rng = np.random.Generator(np.random.PCG64(batch))
    w0 = rng.uniform(-0.3, 0.3, abi.MLP_PARAMS).astype(np.float32)
    for s in (a, b):
        s.mlp_set_weights(w0)
        loss = s.mlp_train(iterations=3, batch=batch, lr=2e-3, seed=5)
    w = a.mlp_get_weights()
    assert np.isfinite(loss) and not np.array_equal(w, w0)
    assert np.array_equal(w.view(np.uint32), b.mlp_get_weights().view(np.uint32))
    c.mlp_set_weights(w)
    x = rng.normal(0.0, 1.0, (3000, 8)).astype(np.float32)
    t = rng.normal(0.0, 1.0, 3000).astype(np.float32)
    assert np.array_equal(a.mlp_forward(x).view(np.uint32), c.mlp_forward(x).view(np.uint32))
    (la, ga), (lc, gc) = gradient(a, x, t), gradient(c, x, t)
    assert la == lc and np.array_equal(ga.view(np.uint32), gc.view(np.uint32))
    for s in (a, b, c):
        s.close()


@pytest.mark.parametrize("n", [1, 8 * 256, 8 * 256 + 1, 40000, 200000])
def test_row_sums_of_equal_rows(n):
    """Equal rows: the mean gradient is that of one tile of them, up to the rounding of the sums (at most
    2,368 partial rows; relative 2e-3 bounds their FP32 accumulation), and repeats bit for bit."""
    s = recorded(1)
    rng = np.random.Generator(np.random.PCG64(9))
    row = rng.normal(0.0, 1.0, 8).astype(np.float32)
    x = np.tile(row, (n, 1))
    t = np.full(n, 0.25, np.float32)
    loss, g = gradient(s, x, t)
    one_loss, one = gradient(s, np.tile(row, (32, 1)), np.full(32, 0.25, np.float32))
    assert np.linalg.norm(g - one) <= 2e-3 * np.linalg.norm(one)
    assert abs(loss - one_loss) <= 2e-3 * abs(one_loss)
    loss2, g2 = gradient(s, x, t)
    assert loss2 == loss and np.array_equal(g.view(np.uint32), g2.view(np.uint32))
    s.close()
