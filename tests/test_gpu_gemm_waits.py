"""The waits inside the GEMM kernel are bounded: with loads that never arrive
in full (nir_mlp_wait_test) it ends with an error within seconds, whatever
way the product is cut, and the handle computes the same as before."""
import time

import numpy as np
import pytest

from conftest import has_gpu
from nirnaya_b200 import mlp

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]

LIMIT = 20.0


@pytest.mark.parametrize("M,N,K", [
    (8, 8, 64),          # fewer stages than the ring holds: only the multiplying thread waits
    (128, 128, 640),     # the loading thread waits as well; two accumulators
    (512, 512, 1024),    # clusters
    (128, 128, 8192),    # splits in the workspace
])
def test_a_product_whose_loads_never_arrive(M, N, K):
    rng = np.random.default_rng(M + K)
    A, B = rng.normal(size=(M, K)).astype(np.float32), rng.normal(size=(N, K)).astype(np.float32)
    with mlp.Mlp(8, 8, width=8, depth=1) as net:
        before = net.gemm(True, True, M, N, K, A, K, B, K)
        t = time.perf_counter()
        assert mlp.lib().nir_mlp_wait_test(net._h, M, N, K) == 3
        assert time.perf_counter() - t < LIMIT
        assert b"gave up" in mlp.lib().nir_mlp_last_error()
        assert np.array_equal(net.gemm(True, True, M, N, K, A, K, B, K), before)
