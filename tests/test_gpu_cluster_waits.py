"""The waits inside a thread-block cluster are bounded: persistent=3 makes
rank 0 wait for bytes that nobody sends.  The solve has to end with an
internal error within the bounds of the waits (about a second each, ranks
that wait for a rank that gave up give up after it), and the same handle has
to solve as if nothing had happened.
"""
import time

import numpy as np
import pytest

from conftest import has_gpu
from nirnaya_b200 import batch as B
from nirnaya_b200 import lp as L
from nirnaya_b200 import pdhg

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]

LIMIT = 20.0


def expect_internal_error(solve):
    t = time.perf_counter()
    with pytest.raises(RuntimeError, match="internal_error"):
        solve(pdhg.default_params(persistent=3, max_iters=5000))
    assert time.perf_counter() - t < LIMIT


@pytest.mark.parametrize("size", [1, 2, 16])
def test_one_lp(monkeypatch, size):
    monkeypatch.setenv("NIR_PDHG_CLUSTER", str(size))
    lp = L.generate(L.RANDOM_EQ, 4, m=300, n=700)
    p = pdhg.default_params(max_iters=256)
    with pdhg.Engine(lp) as eng:
        x0, y0, _ = eng.solve(p)
    with pdhg.Engine(lp) as eng:
        expect_internal_error(eng.solve)
        x, y, _ = eng.solve(p)
    assert np.array_equal(x, x0) and np.array_equal(y, y0)


def test_batch(monkeypatch):
    monkeypatch.setenv("NIR_PDHG_CLUSTER", "4")
    lps = [L.generate(L.MULTIPERIOD, 3, m=500), L.generate(L.RANDOM_EQ, 4, m=300, n=700)]
    p = pdhg.default_params(max_iters=256)
    with B.BatchEngine(lps) as eng:
        want, _ = eng.solve(p)
        expect_internal_error(eng.solve)
        got, _ = eng.solve(p)
    for (x0, y0, _), (x, y, _) in zip(want, got):
        assert np.array_equal(x, x0) and np.array_equal(y, y0)


def test_the_per_launch_kernels_have_no_such_wait(monkeypatch):
    monkeypatch.setenv("NIR_PDHG_CLUSTER", "0")
    with pdhg.Engine(L.generate(L.RANDOM_EQ, 4, m=300, n=700)) as eng:
        assert eng.solve(pdhg.default_params(persistent=3))[2].status == pdhg.OPTIMAL
