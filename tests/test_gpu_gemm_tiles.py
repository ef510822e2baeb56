"""The GEMM's tiles (128 rows, 64 or 128 columns) and its splits of K at their
edges, against the float64 product of the BF16-rounded operands."""
import numpy as np
import pytest

from conftest import has_gpu
from nirnaya_b200 import mlp
from oracle import mlp_oracle as M

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]


@pytest.mark.parametrize("rows,cols,K", [
    (1, 1, 8),              # one element
    (127, 65, 40),          # a tile less one row, a tile and one column, an odd row length
    (128, 64, 504),         # exactly one tile, one step short of a split K
    (129, 63, 512),         # two splits, ragged and odd
    (130, 130, 552),        # splits of 288: a stage cut in half at each end
    (65, 63, 8 * 256),      # as many splits as a CTA has accumulators
    (64, 65, 9 * 256),      # one more: a cluster
    (17, 33, 16 * 256),     # a split for every rank of the largest cluster
    (64, 63, 17 * 256),     # a second round with a single split
    (5, 64, 33 * 256 + 8),  # a third round, a last split of one step
    (19001, 72, 72),        # enough tiles for 128 columns each
])
def test_tile_and_split_edges(rows, cols, K):
    rng = np.random.default_rng(rows * 131 + cols * 7 + K)
    A = rng.normal(size=(rows, K)).astype(np.float32)
    B = rng.normal(size=(cols, K)).astype(np.float32)
    with mlp.Mlp(8, 8, width=8, depth=1) as net:
        C = net.gemm(True, True, rows, cols, K, A, K, B, K)
    Al, Bl = M.bf16(A.astype(np.float64)), M.bf16(B.astype(np.float64))
    # exact products added in FP32, at most one rounding (or truncation) for each
    bound = (K + 64) * 2.0 ** -23 * (np.abs(Al) @ np.abs(Bl).T)
    assert np.all(np.abs(C - Al @ Bl.T) <= bound)
