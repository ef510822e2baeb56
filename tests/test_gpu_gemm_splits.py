"""Products with few tiles and a long K, whose splits are computed by CTAs of
their own and added from a workspace (k_add_splits of
nirnaya_b200/csrc/mlp.cu): edges of tiles and of splits, every storage, and
every epilogue through the network.
"""
import numpy as np
import pytest

from conftest import has_gpu
from nirnaya_b200 import mlp
from oracle import mlp_oracle as M

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]


@pytest.mark.parametrize("a_kmaj", [True, False])
@pytest.mark.parametrize("b_kmaj", [True, False])
@pytest.mark.parametrize("rows,cols,K", [
    (8, 8, 16 * 256),          # one corner of a tile
    (128, 128, 32 * 256 + 8),  # one tile, a last split of one step
    (136, 72, 16 * 288),       # a second row and column of tiles, splits with half a stage
    (64, 200, 40 * 256 - 24),  # a ragged end of K
    (8, 24, 300 * 256),        # as many splits as there are CTAs wanted
])
def test_splits_in_the_workspace(rows, cols, K, a_kmaj, b_kmaj):
    rng = np.random.default_rng(rows * 131 + cols * 7 + K)
    A = rng.normal(size=(rows, K)).astype(np.float32)
    B = rng.normal(size=(cols, K)).astype(np.float32)
    with mlp.Mlp(8, 8, width=8, depth=1) as net:
        C = net.gemm(a_kmaj, b_kmaj, rows, cols, K, A if a_kmaj else A.T, K if a_kmaj else rows,
                     B if b_kmaj else B.T, K if b_kmaj else cols)
    Al, Bl = M.bf16(A.astype(np.float64)), M.bf16(B.astype(np.float64))
    # exact products added in FP32, at most one rounding (or truncation) for each
    bound = (K + 64) * 2.0 ** -23 * (np.abs(Al) @ np.abs(Bl).T)
    assert np.all(np.abs(C - Al @ Bl.T) <= bound)


def test_odd_columns():
    rng = np.random.default_rng(3)
    A, B = rng.normal(size=(33, 8192)).astype(np.float32), rng.normal(size=(13, 8192)).astype(np.float32)
    with mlp.Mlp(8, 8, width=8, depth=1) as net:
        C = net.gemm(True, True, 33, 13, 8192, A, 8192, B, 8192)
    Al, Bl = M.bf16(A.astype(np.float64)), M.bf16(B.astype(np.float64))
    assert np.all(np.abs(C - Al @ Bl.T) <= (8192 + 64) * 2.0 ** -23 * (np.abs(Al) @ np.abs(Bl).T))


@pytest.mark.parametrize("d_in,d_out,width,rows", [
    (8192, 16, 64, 24),   # bias and ReLU after a long K
    (16, 8192, 64, 24),   # the ReLU's mask after a long K
    (24, 8, 64, 4096),    # the weight gradients as one group, a long K over the samples
])
def test_network(d_in, d_out, width, rows):
    rng = np.random.default_rng(rows)
    with mlp.Mlp(d_in, d_out, width=width, depth=2, seed=4) as net:
        p = net.get_params()
        X = rng.normal(size=(rows, d_in)).astype(np.float32)
        T = rng.normal(size=(rows, d_out)).astype(np.float32)
        loss, g = net.gradients(X, T)
        lo, go = M.loss_and_grads(p, net.dims, X, T)
    # the bounds of the network's other comparisons with this oracle
    assert abs(loss - lo) <= 5e-3 * lo
    assert np.linalg.norm(g - go) <= 1e-2 * np.linalg.norm(go)
