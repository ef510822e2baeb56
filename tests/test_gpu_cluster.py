"""Solves in thread-block clusters (nirnaya_b200/csrc/k_cluster.cuh) against
the per-launch kernels (NIR_PDHG_CLUSTER=0), through the C ABI.

Both run the same iteration in FP64 arithmetic and differ in the order of a
row's sum alone, so after a few hundred iterations the points agree far
below 1e-9 relative (each sum's rounding is 1e-16 of its terms, and the
iteration does not expand differences).
"""
import numpy as np
import pytest

from conftest import has_gpu
from nirnaya_b200 import batch as B
from nirnaya_b200 import lp as L
from nirnaya_b200 import pdhg
from test_gpu_parity import dense_row_lp

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]

TOL = 1e-9


def one_row_lp():
    """Fewer rows than ranks, one-entry columns, a free and a fixed column."""
    lp = L.LP.from_rows(5, [([0, 1, 2, 3, 4], [1.0, 2.0, -1.0, 3.0, 1.0])], cost=[1.0, -1.0, 0.5, 2.0, 0.0],
                        collo=[0.0, 0.0, -np.inf, 0.0, 1.5], colup=[4.0, 3.0, np.inf, np.inf, 1.5], rowlo=[2.0],
                        rowup=[6.0])
    return lp


CASES = {
    "one_row": (one_row_lp, {}),
    "dense_row": (dense_row_lp, {}),  # a 9,000-entry row, empty rows and columns
    "random": (lambda: L.generate(L.RANDOM_EQ, 3, m=301, n=753), {}),
    "zipf": (lambda: L.generate(L.ZIPF, 2, m=1500, n=3700, target_nnz=36000), {}),
    "blocks": (lambda: L.generate(L.MULTIPERIOD, 3, m=2011, n=5003), {}),
    "each_iteration_checked": (lambda: L.generate(L.RANDOM_EQ, 4, m=120, n=300), dict(check_every=1, max_iters=60)),
    "more_weights_than_tabulated": (lambda: L.generate(L.RANDOM_EQ, 4, m=120, n=300), dict(check_every=101)),
    "plain_pdhg": (lambda: L.generate(L.RANDOM_EQ, 9, m=300, n=700), dict(algorithm=pdhg.ALGO_PDHG)),
}


def rel(a, b):
    return np.linalg.norm(a - b) / (1e-300 + np.linalg.norm(b))


def solve(monkeypatch, lp, size, kw):
    monkeypatch.setenv("NIR_PDHG_CLUSTER", str(size))
    with pdhg.Engine(lp) as eng:
        return eng.solve(pdhg.default_params(**{**dict(tol=1e-7, max_iters=320), **kw}))


@pytest.mark.parametrize("prec", [pdhg.PREC_FP64, pdhg.PREC_MIXED])
@pytest.mark.parametrize("name", CASES)
def test_clusters_match_the_per_launch_kernels(monkeypatch, name, prec):
    make, kw = CASES[name]
    lp = make()
    x0, y0, i0 = solve(monkeypatch, lp, 0, dict(kw, precision=prec))
    for size in (1, 2, 8, 16):
        x, y, i = solve(monkeypatch, lp, size, dict(kw, precision=prec))
        assert i.kernel_launches < i0.kernel_launches  # the clusters ran
        assert (i.status, i.iterations, i.restarts) == (i0.status, i0.iterations, i0.restarts)
        assert rel(x, x0) <= TOL and rel(y, y0) <= TOL
        assert abs(i.objective - i0.objective) <= TOL * (1 + abs(i0.objective))


def test_new_vectors_warm_start_and_a_mixed_hand_over(monkeypatch):
    # one handle: a cold solve, new vectors, a start, and the FP64 phase (forced by polish_switch_kkt)
    a = L.generate(L.BLEND_FAMILY, 1, m=600, n=1500, target_nnz=12000)
    b = L.generate(L.BLEND_FAMILY, 2, m=600, n=1500, target_nnz=12000)
    got = []
    for size in (0, 4):
        monkeypatch.setenv("NIR_PDHG_CLUSTER", str(size))
        with pdhg.Engine(L.LP(a.nrow, a.ncol, a.col_start, a.row_index, a.value, a.cost, a.collo, a.colup, a.rowlo,
                              a.rowup)) as eng:
            x, y, _ = eng.solve(pdhg.default_params(max_iters=256))
            eng.update_vectors(cost=b.cost, rowlo=b.rowlo, rowup=b.rowup, collo=b.collo, colup=b.colup)
            got.append(eng.solve(pdhg.default_params(max_iters=448, polish_switch_kkt=1e-2), x_init=x, y_init=y))
    (x0, y0, i0), (x1, y1, i1) = got
    assert i0.iterations_fp64 > 0 and i1.iterations_fp64 == i0.iterations_fp64
    assert rel(x1, x0) <= TOL and rel(y1, y0) <= TOL


@pytest.mark.parametrize("prec", [pdhg.PREC_FP64, pdhg.PREC_MIXED])
@pytest.mark.parametrize("size", [None, 1, 8])
def test_batch_clusters_match_the_per_launch_kernels(monkeypatch, size, prec):
    # uneven instances; the last one fits no cluster and stays with the per-launch kernels
    lps = [L.generate(L.RANDOM_EQ, 11, m=300, n=750), one_row_lp(), L.generate(L.MULTIPERIOD, 12, m=700), dense_row_lp(),
           L.generate(L.RANDOM_EQ, 13, m=13000, n=32000)]
    out = []
    for s in (0, size):
        if s is None:
            monkeypatch.delenv("NIR_PDHG_CLUSTER")
        else:
            monkeypatch.setenv("NIR_PDHG_CLUSTER", str(s))
        with B.BatchEngine(lps) as eng:
            out.append(eng.solve(pdhg.default_params(max_iters=320, tol=1e-7, precision=prec))[0])
    for (x0, y0, i0), (x1, y1, i1) in zip(*out):
        assert (i1.status, i1.iterations, i1.restarts) == (i0.status, i0.iterations, i0.restarts)
        assert rel(x1, x0) <= TOL and rel(y1, y0) <= TOL
