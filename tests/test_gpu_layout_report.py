"""nir_pdhg_get_layout reports the layout of the last PDHG / PDLP solve with
the per-launch kernels, and changes nothing."""
import numpy as np
import pytest

from conftest import has_gpu
from nirnaya_b200 import lp as L
from nirnaya_b200 import pdhg

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]


def facts(eng):
    lo = eng.layout()
    return lo.blocks_a, lo.blocks_at, lo.block_nnz, lo.block_nnz_at


def test_a_reference_solve_leaves_the_layout_in_use_alone():
    lp = L.generate(L.RANDOM_EQ, 4, m=300, n=700)
    for cap in (64, 256):
        with pdhg.Engine(lp) as eng:
            eng.solve(pdhg.default_params(max_iters=64, spmv_block_nnz=cap))
            before = facts(eng)
            assert before[2:] == (cap, cap)
            eng.solve(pdhg.default_params(max_iters=64, algorithm=pdhg.ALGO_REFERENCE, tol=0.0))
            assert facts(eng) == before


def test_clusters_have_no_row_blocks_of_their_own(monkeypatch):
    lp = L.generate(L.RANDOM_EQ, 4, m=300, n=700)
    monkeypatch.setenv("NIR_PDHG_CLUSTER", "4")
    p = pdhg.default_params(max_iters=128)
    with pdhg.Engine(lp) as eng:
        assert facts(eng) == (0, 0, 0, 0)
        x, y, _ = eng.solve(p)
        held = eng.layout().device_bytes
        blocks_a, blocks_at, nnz_a, nnz_at = facts(eng)
        x1, y1, _ = eng.solve(p)
        assert np.array_equal(x1, x) and np.array_equal(y1, y) and eng.layout().device_bytes == held
        # the same once they are built
        eng.time_iteration(pdhg.PREC_FP64, 2)
        assert facts(eng) == (blocks_a, blocks_at, nnz_a, nnz_at) and blocks_a > 0 and blocks_at > 0
