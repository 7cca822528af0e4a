"""Orderings that a run on the GPU does not show to be missing, read from the source.

A block's barrier has to be met by every thread at the same statement.  The filters'
kernels split a block into causal and anticausal warps, so their helpers are entered by some
warps only and hold no barrier; it stands in the kernel itself, outside the split.

A kernel that follows a join of two streams is an ordinary launch: one that may start before
the stream's last kernel has ended is ordered by that kernel alone."""
import os
import re

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


def test_batched_kernels_after_a_join_are_ordinary_launches():
    with open(os.path.join(ROOT, "itk_gb300", "csrc", "gb_batch.cu")) as f:
        source = f.read()
    # an evaluation ends in the join; the step, or the next evaluation's clear, follows it
    assert "cudaStreamWaitEvent(st, b->fork_ev[1]" in source
    assert not re.search(r"launch_dep\(\s*st,\s*k_batch_clear", source)
    assert re.search(r"if \(step && fork\) \{\s*k_batch_step<<<", source)
