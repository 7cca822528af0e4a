"""A block's barrier has to be met by every thread at the same statement.  The filters'
kernels split a block into causal and anticausal warps, so their helpers are entered by some
warps only and hold no barrier; it stands in the kernel itself, outside the split."""
import os

from conftest import ROOT


def test_filter_barriers_stand_in_the_kernels():
    with open(os.path.join(ROOT, "itk_gb300", "csrc", "gb_filters.cu")) as f:
        lines = f.read().split("\n")
    found = 0
    function = ""
    for line in lines:
        if line[:1] not in ("", " ", "}", "/") and ("__device__" in line or "__global__" in line):
            function = line
        if "__syncthreads()" in line.split("//")[0]:
            found += 1
            assert "__global__" in function, f"barrier in a helper: {function}"
    assert found > 0
