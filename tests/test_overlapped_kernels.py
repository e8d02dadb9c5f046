"""Kernels that start while the kernel before them runs (launch_overlapped in
csrc/common.cuh) make no __restrict__ promise in their parameters, which would
hold before they have waited for that kernel's writes."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "shiokaze_b200", "csrc")


def test_overlapped_kernels_take_no_restrict_parameters():
    names, bad = set(), []
    sources = {f: open(os.path.join(CSRC, f)).read() for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))}
    for text in sources.values():
        names |= set(re.findall(r"launch_overlapped\((k_\w+),", text))
    assert len(names) >= 10, names
    found = set()
    for text in sources.values():
        for kernel, params in re.findall(r"__global__ void (?:__launch_bounds__\([^)]*\)\s*)?(k_\w+)\(([^{;]*?)\)\s*\{", text):
            if kernel in names:
                found.add(kernel)
                if "__restrict__" in params:
                    bad.append(kernel)
    assert found == names
    assert not bad, bad
