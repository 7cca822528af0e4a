"""Lengths of plain FP32 sums, read from the source.

The B-spline derivative's sums over a cell's samples are plain FP32 in up to 16 additions, then
pairwise and compensated: the rounding of longer runs is a few per cent of the derivative's error,
below what one input's error varies by, so no comparison of outputs shows it."""
import os
import re

from conftest import ROOT


def test_chunk_sums_make_at_most_sixteen_plain_additions():
    with open(os.path.join(ROOT, "itk_gb300", "csrc", "gb_bspline.cuh")) as f:
        source = f.read()
    constants = {k: int(v) for k, v in re.findall(r"constexpr int (\w+) = (\d+);", source)}
    plain = constants.get("kFoldBatches", constants["kChunkLen"] // constants["kChunkBatch"]) * constants["kChunkBatch"]
    assert plain <= 16 * constants.get("kChunkSlices", 64)
    kernel = source[source.index("k_bspline_chunks(EvalArgs a)"):]
    assert "batch % kFoldBatches == kFoldBatches - 1" in kernel
    assert re.search(r"j \+= kChunkSlices", kernel)
