"""The CTA-block layout against the warp row blocks: iterations whose kernels
start early, over LPs with fewer blocks than CTAs, a row longer than a block,
empty rows and columns, and several blocks per CTA.

The two differ in the order of a row's sum alone, so after a few hundred
iterations the points agree far below 1e-9 relative (each sum's rounding is
1e-16 of its terms, and the iteration does not expand differences).
"""
import pytest

from conftest import has_gpu
from nirnaya_b200 import lp as L
from nirnaya_b200 import pdhg
from test_gpu_cluster import TOL, one_row_lp, rel
from test_gpu_parity import dense_row_lp

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]

CASES = {
    "one_row": one_row_lp,
    "dense_row": dense_row_lp,
    "random": lambda: L.generate(L.RANDOM_EQ, 3, m=301, n=753),
    "blocks": lambda: L.generate(L.MULTIPERIOD, 3, m=2011, n=5003),
    "several_blocks_per_cta": lambda: L.generate(L.RANDOM_EQ, 5, m=40001, n=100003),
}


@pytest.mark.parametrize("prec", [pdhg.PREC_FP64, pdhg.PREC_MIXED])
@pytest.mark.parametrize("name", CASES)
def test_cta_blocks_match_warp_blocks(name, prec):
    with pdhg.Engine(CASES[name]()) as eng:
        (x0, y0, i0), (x1, y1, i1) = (
            eng.solve(pdhg.default_params(tol=1e-7, max_iters=256, precision=prec, spmv_block_nnz=b)) for b in (256, 1024))
    assert (i1.status, i1.iterations, i1.restarts) == (i0.status, i0.iterations, i0.restarts)
    assert rel(x1, x0) <= TOL and rel(y1, y0) <= TOL
    assert abs(i1.objective - i0.objective) <= TOL * (1 + abs(i0.objective))
