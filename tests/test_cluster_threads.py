"""The worker threads of a cluster plan (nirnaya_b200/csrc/cluster_plan.hpp):
a thread that cannot be started, for want of memory too, leaves its work to
the others; it must not end the process with the started ones unjoined.
"""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include"


def test_a_thread_that_cannot_be_started(tmp_path):
    exe = str(tmp_path / "threads")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "nirnaya_b200", "csrc"), "-I", CUDA_INC,
                    os.path.join(ROOT, "tests", "native", "cluster_threads_harness.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", (out.returncode, out.stdout, out.stderr)
