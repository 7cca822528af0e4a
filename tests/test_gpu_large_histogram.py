"""Mattes' joint histogram of blocks that flush it many times.

A block of pass 1 empties its shared histogram every 16384 samples; its column sums (the moving
marginal) are emptied with it.  Kept in 32-bit words to the block's end they wrap from about
4096 rows times flushes on: with 159 bins from 0.4 to 0.9 million samples in a block.  The
batched engine, told to put any number of samples into a block, spreads a registration over 80
blocks: 464^3 voxels are 1.25 million a block, 76 flushes of 155 rows."""
import numpy as np
import pytest

import itk_gb300 as gb

pytestmark = pytest.mark.gpu


def mi_of_pdf(p):
    pf, pm = p.sum(1, keepdims=True), p.sum(0, keepdims=True)
    ok = p > np.finfo(np.float64).eps
    return float(-(p[ok] * np.log(p[ok] / (pf * pm)[ok])).sum())


def test_marginal_is_the_histograms_after_many_flushes():
    n, bins = 464, 159
    rng = np.random.default_rng(11)
    # unrelated images: each column holds every row, and the weights' low bits are spread evenly
    fixed, moving = (gb.Image(rng.random((n, n, n), dtype=np.float32)) for _ in range(2))
    t = gb.AffineTransform()
    t.SetCenter((np.array([n, n, n]) - 1.0) / 2.0)
    m = gb.MattesMutualInformationImageToImageMetricv4()
    m.SetFixedImage(fixed)
    m.SetMovingImage(moving)
    m.SetMovingTransform(t)
    m.SetNumberOfHistogramBins(bins)
    m.SetUseMovingImageGradientFilter(False)
    m.Initialize()
    o = gb.RegularStepGradientDescentOptimizerv4()
    o.SetNumberOfIterations(1)
    o.SetMetric(m)
    b = gb.RegistrationBatch()
    b.SetSamplesPerBlock(1 << 27, 1 << 27, 1 << 27)
    b.Add(o)
    b.Run()
    # the value formed from the marginal is the one that the joint PDF's own sums give: pf is a
    # count there and a sum of weights within 3 / 2^27 of 1 each here; the rest is FP64
    want = mi_of_pdf(m.GetJointPDF())
    assert abs(o.GetValue() - want) <= 1e-7 + 1e-6 * abs(want)
