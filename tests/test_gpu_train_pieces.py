"""An epoch larger than a piece of the gathered samples (32 MB): every sample
is used once with its own target, and the training set's memory is not taken
a second time.
"""
import numpy as np
import pytest

from conftest import has_gpu
from nirnaya_b200 import mlp

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]

BATCH, STEPS = 4096, 98  # 160 bytes a sample: 64 MB, in pieces of 51 and 47 steps


def test_an_epoch_in_pieces():
    import torch

    rng = np.random.default_rng(5)
    X = rng.standard_normal((BATCH * STEPS, 64)).astype(np.float32)
    T = rng.random((BATCH * STEPS, 8)).astype(np.float32)
    # no step changes the weights, so an epoch's loss is that of the predictions, in any order
    with mlp.Mlp(64, 8, width=64, depth=2, seed=2, lr=0.0) as net:
        p = net.get_params()
        net.set_data(X, T)
        free = torch.cuda.mem_get_info()[0]
        losses = net.train(2, BATCH)
        taken = free - torch.cuda.mem_get_info()[0]
        assert np.array_equal(net.get_params(), p)
        want = np.mean((net.predict(X).astype(np.float64) - T) ** 2)
    # sums of 32,768 FP32 terms a step by at most 1024 threads and their tree: 1e-5 is far above their rounding
    assert np.abs(losses - want).max() <= 1e-5 * want
    assert taken < 48 << 20
