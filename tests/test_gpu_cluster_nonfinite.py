"""A column that overflows touches only the rows it occurs in, in the
thread-block clusters (nirnaya_b200/csrc/k_cluster.cuh) as in the per-launch
kernels: a slice's padding entries multiply nothing of the iterate.
"""
import numpy as np
import pytest

from conftest import has_gpu
from nirnaya_b200 import lp as L
from nirnaya_b200 import pdhg

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]

TOL = 1e-9  # as between the two paths on finite data (test_gpu_cluster.py)
OWN = 14    # rows of the block with the overflowing column, its only column of that many entries


def two_blocks(seed):
    """Rows 0 .. 13 share the free column 0, whose cost is near the largest
    double; the other rows and columns are an LP of their own, with rows of
    1 to 9 and columns of at most 12 entries."""
    rng = np.random.default_rng(seed)
    m, n = 150, 260
    rows = [([0, 1 + i % 3], [1.0, 0.5 + 0.1 * i]) for i in range(OWN)]
    for _ in range(m):
        cols = np.sort(rng.choice(np.arange(4, n), int(rng.integers(1, 10)), replace=False))
        rows.append((cols.tolist(), rng.uniform(0.5, 1.5, len(cols)).tolist()))
    cost = rng.uniform(0.1, 1.0, n)
    cost[0] = -1.7e308
    collo = np.zeros(n)
    collo[0] = -np.inf
    return L.LP.from_rows(n, rows, cost=cost, collo=collo, colup=np.where(np.arange(n) == 0, np.inf, 10.0),
                          rowlo=np.full(OWN + m, 1.0), rowup=np.full(OWN + m, 5.0))


@pytest.mark.parametrize("prec", [pdhg.PREC_FP64, pdhg.PREC_MIXED])
@pytest.mark.parametrize("size", [1, 2, 8])
def test_an_overflow_stays_in_its_block(monkeypatch, size, prec):
    lp = two_blocks(3)
    assert np.diff(lp.col_start).argmax() == 0
    got = []
    for s in (0, size):
        monkeypatch.setenv("NIR_PDHG_CLUSTER", str(s))
        with pdhg.Engine(lp) as eng:
            x, y, _ = eng.solve(pdhg.default_params(max_iters=64, precision=prec, omega_init=1e-3))
        got.append((x, y))
    (x0, y0), (x, y) = got
    assert not np.isfinite(y0[:OWN]).all()  # it did overflow
    assert np.isfinite(x0[4:]).all() and np.isfinite(y0[OWN:]).all()
    for a, b in ((x[4:], x0[4:]), (y[OWN:], y0[OWN:])):
        assert np.linalg.norm(a - b) <= TOL * (1.0 + np.linalg.norm(b))
