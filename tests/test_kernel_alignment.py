"""Shared memory that 16-byte asynchronous copies or vector loads go to is declared so."""
import glob
import os
import re

from conftest import ROOT


def test_tiles_of_wide_copies_are_declared_at_16_bytes():
    with open(os.path.join(ROOT, "itk_gb300", "csrc", "gb_filters.cu")) as f:
        tiles = re.findall(r"extern __shared__ ([^;]*)tile\[\];", f.read())
    assert tiles and all("__align__(16)" in t for t in tiles)
    # nodes behind another array in the same dynamic shared memory
    for path in glob.glob(os.path.join(ROOT, "itk_gb300", "csrc", "*.cuh")):
        with open(path) as f:
            for kernel in f.read().split("__global__")[1:]:
                if "node_offset(B)" in kernel.split("\n}\n")[0]:
                    assert "extern __shared__ __align__(16)" in kernel, path
