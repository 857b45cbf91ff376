"""Kernels that overlap their predecessor (launch_dependent) must not load through the read-only path: its
data has to stay unchanged for the kernel's whole lifetime, and the predecessor may still be writing."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sd3.c_b200", "csrc")


def _sources():
    return {f: re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
            for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}


def test_no_read_only_loads_in_dependent_kernels():
    src = _sources()
    dependent = [f for f, s in src.items() if "launch_dependent(" in s]
    assert len(dependent) >= 6
    for f in dependent + [f for f in src if f.endswith(".cuh")]:  # the headers' functions are inlined into them
        assert "__ldg(" not in src[f] and "ld.global.nc" not in src[f], f
    for f in dependent:
        # a kernel that waits for its predecessor takes no __restrict__ pointers (the compiler may turn loads
        # from const ones into read-only ones)
        for m in re.finditer(r"__global__.*?\{(.*?)\n\}", src[f], flags=re.S):
            if "grid_dep_wait()" in m.group(0):
                assert "__restrict__" not in m.group(0).split("{", 1)[0], (f, m.group(0)[:120])
