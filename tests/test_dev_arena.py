"""The engine's device memory (nirnaya_b200/csrc/dev_arena.hpp): allocations
carved from chunks stay inside a block, whatever was given back by rewinding
before them.  An address outside of its block is an illegal access on the
device, so this runs on the CPU with a host allocator.
"""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include"


def test_allocations_stay_in_their_blocks(tmp_path):
    exe = str(tmp_path / "arena")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "nirnaya_b200", "csrc"), "-I", CUDA_INC,
                    os.path.join(ROOT, "tests", "native", "dev_arena_harness.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
