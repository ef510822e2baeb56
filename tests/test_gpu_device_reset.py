"""A program may reset the device between two handles: what the libraries
keep of host memory that kernels write to (nirnaya_b200/csrc/mapped_host.hpp)
is valid for the next handle all the same.  In a process of its own, for the
reset takes the whole context.
"""
import os
import subprocess
import sys

import pytest

from conftest import ROOT, has_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA device")]

PROGRAM = """
import ctypes, sys
import numpy as np
from nirnaya_b200 import lp as L, mlp, pdhg

lp = L.generate(L.RANDOM_EQ, 4, m=120, n=300)
X = np.linspace(-1.0, 1.0, 16 * 16, dtype=np.float32).reshape(16, 16)

def work(handles):
    engines = [pdhg.Engine(lp) for _ in range(handles)]
    nets = [mlp.Mlp(16, 8, width=64, depth=2, seed=3) for _ in range(handles)]
    out = [e.solve(pdhg.default_params(max_iters=128))[0] for e in engines] + [n.predict(X) for n in nets]
    for h in engines + nets:
        h.close()
    return out

driver = ctypes.CDLL("libcuda.so.1")
device = ctypes.c_int()
first = work(20)  # more handles than blocks are kept
assert driver.cuInit(0) == 0 and driver.cuDeviceGet(ctypes.byref(device), 0) == 0
for handles in (1, 20):
    assert driver.cuDevicePrimaryCtxReset_v2(device) == 0
    again = work(handles)
    assert np.array_equal(again[0], first[0]) and np.array_equal(again[-1], first[-1])
print("ok")
"""


def test_handles_after_a_device_reset():
    out = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
