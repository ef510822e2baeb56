"""Where clusters cannot run, a solve falls back to a smaller size or to the
per-launch kernels instead of failing: the host's part of that choice
(nirnaya_b200/csrc/cluster_plan.hpp), and that a device out of memory is
reported as such (dev_arena.hpp), on the CPU.
"""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "nirnaya_b200", "csrc")
CUDA_INC = os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include"


def test_sizes_and_memory(tmp_path):
    exe = str(tmp_path / "choice")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-I", CUDA_INC,
                    os.path.join(ROOT, "tests", "native", "cluster_choice_harness.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout


NO_MEMORY = r"""
#include "dev_arena.hpp"
#include <cstdio>
static int g_last = 0;
extern "C" {
cudaError_t cudaMalloc(void**, size_t) { g_last = cudaErrorMemoryAllocation; return cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "out of memory"; }
cudaError_t cudaGetLastError() { const int e = g_last; g_last = 0; return cudaError_t(e); }
}
int main() {
    nir::DevArena m;
    try {
        m.alloc(100);
    } catch (const std::bad_alloc& e) {
        // nothing left for the next launch's check to find
        std::printf("%s\n", g_last == 0 && std::string(e.what()).find("out of memory") != std::string::npos ? "ok" : "left");
        return 0;
    }
    return 1;
}
"""


def test_a_device_out_of_memory_can_be_told_apart(tmp_path):
    src, exe = tmp_path / "no_memory.cpp", str(tmp_path / "no_memory")
    src.write_text(NO_MEMORY)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", CUDA_INC, str(src), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
