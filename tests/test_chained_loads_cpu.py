"""Kernels launched as programmatic dependents read what their predecessor wrote.  Their wait orders those
loads only while the compiler may not take the memory for unwritten: no __restrict__ pointer and no
non-coherent load in a chained kernel, nor in the helpers that such a kernel calls.  Checked on the source."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hpcsharp_b200", "csrc")
FORBIDDEN = re.compile(r"__restrict__|__ldg\s*\(|\bldg_stream_v4\s*\(|\bld\.global\.nc\b")


def _functions():
    """name -> text (signature and body) of every __global__ and __device__ function of csrc/."""
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
        for m in re.finditer(r"__(?:global|device)__[^;{}()]*?\b(\w+)\s*\([^;{}]*\)\s*(?:const\s*)?\{", text):
            at = m.end() - 1
            depth, end = 0, at
            for end in range(at, len(text)):
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                if depth == 0:
                    break
            out.setdefault(m.group(1), "")
            out[m.group(1)] += text[m.start():end + 1]
    return out


FUNCTIONS = _functions()
CHAINED = sorted(n for n, t in FUNCTIONS.items() if "__global__" in t and "chain_wait()" in t)


def test_chained_kernels_are_found():
    assert {"lookback_pass_kernel", "finalize_kernel", "select_sample_kernel", "select_window_kernel", "select_level_kernel",
            "select_compact_kernel", "select_finish_kernel", "partition_count_kernel", "partition_scan_kernel",
            "partition_scatter_kernel", "topk_gather_kernel", "topk_small_sort_kernel"} <= set(CHAINED)


@pytest.mark.parametrize("kernel", CHAINED)
def test_chained_kernel_loads_are_ordered(kernel):
    seen, todo = set(), [kernel]
    while todo:
        name = todo.pop()
        if name in seen:
            continue
        seen.add(name)
        text = FUNCTIONS[name]
        bad = FORBIDDEN.search(text)
        assert bad is None, f"{kernel}: {bad.group(0)} in {name}"
        todo += [c for c in set(re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\s*\(", text)) if c in FUNCTIONS]
