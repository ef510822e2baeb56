"""Device buffers that grow on demand (nirnaya_b200/csrc/grown.hpp): after an
allocation that failed, nothing is served from memory already given back.
Built and run on the CPU with a memory that fails on demand; the sources are
checked for buffers that are released and allocated by hand.
"""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "nirnaya_b200", "csrc")


def test_a_failed_growth_leaves_an_empty_buffer(tmp_path):
    exe = str(tmp_path / "grown")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, os.path.join(ROOT, "tests", "native", "grown_harness.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout


def test_no_buffer_of_a_handle_is_regrown_by_hand():
    # h->release(h->x) ... h->x = h->alloc(...) leaves h->x dangling when the allocation throws
    for name in ("mlp.cu", "engine.cu", "engine_batch.cuh", "engine_cluster.cuh"):
        with open(os.path.join(CSRC, name)) as f:
            assert not re.findall(r"release\(h->\w+\)|release\(\*q\);\s*\*?q = h->alloc", f.read()), name
