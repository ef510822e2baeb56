"""The reported objective is c'x + obj_offset on every path of a solve
(the reference's Model::eval_objective, src/model/model.hpp:73-98), through
the C ABI.

The engine adds in double-double, numpy's dot in FP64: they differ by at
most n rounding errors of the terms' magnitudes.
"""
import numpy as np
import pytest

from conftest import has_gpu
from nirnaya_b200 import batch as B
from nirnaya_b200 import lp as L
from nirnaya_b200 import pdhg

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]

OFFSET = -1234.5


def with_offset(lp, offset=OFFSET):
    return L.LP(lp.nrow, lp.ncol, lp.col_start, lp.row_index, lp.value, lp.cost, lp.collo, lp.colup, lp.rowlo, lp.rowup,
                obj_offset=offset)


def check(lp, x, objective):
    terms = lp.cost * x
    slack = 2.0 ** -52 * lp.ncol * (np.abs(terms).sum() + abs(lp.obj_offset))
    assert abs(objective - (terms.sum() + lp.obj_offset)) <= slack


def parallel_lp():
    """Column 0 twice, the second time doubled: solved as the equivalent LP."""
    return L.LP.from_rows(3, [([0, 1, 2], [1.0, 2.0, 1.0]), ([0, 1, 2], [-1.0, -2.0, 2.0])], cost=[1.0, 2.5, 0.5],
                          collo=[0.0, 0.0, 0.0], colup=[4.0, 3.0, 5.0], rowlo=[2.0, -3.0], rowup=[6.0, np.inf])


SOLVES = {
    "pdlp_fp64": dict(precision=pdhg.PREC_FP64),
    "pdlp_mixed": dict(precision=pdhg.PREC_MIXED),
    "pdlp_fp32": dict(precision=pdhg.PREC_FP32),
    "pdhg": dict(algorithm=pdhg.ALGO_PDHG),
    "reference": dict(algorithm=pdhg.ALGO_REFERENCE),
    "no_iteration": dict(max_iters=0),
}


@pytest.mark.parametrize("cluster", [0, 8])
@pytest.mark.parametrize("solve", SOLVES)
def test_one_lp(monkeypatch, solve, cluster):
    monkeypatch.setenv("NIR_PDHG_CLUSTER", str(cluster))
    for lp in (L.generate(L.RANDOM_EQ, 5, m=120, n=300), parallel_lp()):
        lp = with_offset(lp)
        with pdhg.Engine(lp) as eng:
            x, _, info = eng.solve(pdhg.default_params(**{**dict(max_iters=192), **SOLVES[solve]}))
        check(lp, x, info.objective)


@pytest.mark.parametrize("cluster", [0, 1])
def test_batch(monkeypatch, cluster):
    monkeypatch.setenv("NIR_PDHG_CLUSTER", str(cluster))
    lps = [with_offset(L.generate(L.RANDOM_EQ, 5 + k, m=60 + 7 * k, n=150), OFFSET * (k + 1)) for k in range(3)]
    with B.BatchEngine(lps) as eng:
        res, _ = eng.solve(pdhg.default_params(max_iters=192))
    for lp, (x, _, info) in zip(lps, res):
        check(lp, x, info.objective)
