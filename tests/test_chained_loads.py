"""Loads in kernels launched before their predecessor has ended
(launch_chained): such a kernel reads what that predecessor wrote, so nothing
in it may be loaded through the non-coherent path, which CUDA defines only for
data that is read-only for the whole life of the kernel.  That path is
__ldg, and what the compiler may choose for a `const T* __restrict__`.

Read from the sources, on the CPU: the chained kernels, and every device
function of the files that hold them."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nextla.jl_gb300", "csrc")


def _functions(text):
    """(name, is_kernel, source) of every __global__ and __device__ function definition."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__(global|device)__", text):
        body = text.find("{", m.end())
        if body < 0 or ";" in text[m.end():body]:
            continue  # a declaration or a variable
        head = text[m.end():body]
        name = re.search(r"(\w+)\s*\((?!.*__launch_bounds__)", re.sub(r"__launch_bounds__\([^)]*\)", "", head), re.S)
        depth, end = 1, body + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        if name:
            yield name.group(1), m.group(1) == "global", text[m.start():end]


def test_chained_kernels_load_coherently():
    seen = set()
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith(".cu"):
            continue
        with open(os.path.join(CSRC, f)) as fh:
            text = fh.read()
        calls = re.findall(r"launch_chained\(([^;]*);", text)
        chained = {k for c in calls for k in re.findall(r"\b(\w+_kernel)\b", c)}
        if not chained:
            continue
        for name, kernel, source in _functions(text):
            if kernel and name not in chained:
                continue
            assert "__ldg" not in source, (f, name)
            assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", source), (f, name)
            if kernel:
                assert "chain_begin()" in source, (f, name)
                seen.add(name)
    assert {"crt_gemm_kernel", "crt_finish_kernel", "crt_split_kernel", "split_kernel", "umma_gemm_kernel",
            "umma_f32_kernel", "stage_f32_kernel", "leaf_pair_kernel"} <= seen, seen
