"""Kernels of nirnaya_b200/csrc/mlp.cu that start while the kernel before them
still runs (they call pdl_wait) must not take what that one writes as
`const T* __restrict__`: the qualifiers promise the compiler that nobody
writes the memory while the kernel runs, and let it load through the
read-only path, which may hold what was there before.  No run can show this
reliably, so the signatures are checked.
"""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# complete before the chain of early launches begins: targets and output weights
BEFORE_THE_CHAIN = {"tgt", "w"}


def functions(src):
    """name -> (parameters, body) of the device functions at the top level."""
    src = re.sub(r"__launch_bounds__\([^)]*\)", "", src)
    out = {}
    for m in re.finditer(r"^(?:__global__|__device__)[^;{]*?\b(\w+)\(([^{;]*)\)\s*\{", src, re.M):
        depth, k = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(src[k], 0)
            k += 1
        out[m.group(1)] = (m.group(2), src[m.end():k])
    return out


def test_early_kernels_promise_nothing_about_a_neighbours_output():
    with open(os.path.join(ROOT, "nirnaya_b200", "csrc", "mlp.cu")) as f:
        fn = functions(f.read())
    early = {k for k, (_, body) in fn.items() if "pdl_wait();" in body}
    assert {"k_gemm", "k_loss", "k_colsum_part", "k_adam"} <= early
    # and what they call
    reached, todo = set(), set(early)
    while todo:
        k = todo.pop()
        reached.add(k)
        todo |= {c for c in fn if c not in reached and re.search(r"\b%s\b\s*[(<]" % c, fn[k][1])}
    for k in sorted(reached):
        promised = set(re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", fn[k][0]))
        assert promised <= BEFORE_THE_CHAIN, (k, promised)
