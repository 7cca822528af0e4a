"""A registration among many: pass 1 of Mattes spreads over fewer blocks there, with the same bits."""
import numpy as np
import pytest

import itk_gb300 as gb
from cases import perturbed, small_pair

pytestmark = pytest.mark.gpu


def optimizer(k):
    size = (40 + k % 3, 39, 41 - k % 2)
    fixed, moving, t = small_pair(size, config=1, multimodal=True, seed_shift=k % 4)
    t = perturbed(t, k)
    m = gb.MattesMutualInformationImageToImageMetricv4()
    m.SetFixedImage(fixed)
    m.SetMovingImage(moving)
    m.SetMovingTransform(t)
    m.SetNumberOfHistogramBins([50, 20, 64][k % 3])
    m.Initialize()
    o = gb.RegularStepGradientDescentOptimizerv4()
    o.SetMetric(m)
    o.SetNumberOfIterations(4)
    o.SetScales(np.array([1.0] * 9 + [1.0 / 50.0] * 3))
    return t, o


def run(indices, persistent):
    b = gb.RegistrationBatch()
    b.SetPersistent(persistent)
    members = [optimizer(k) for k in indices]
    for _, o in members:
        b.Add(o)
    b.Run()
    return [(t.GetParameters().copy(), o.GetValue()) for t, o in members]


@pytest.mark.parametrize("persistent", [False, True])
def test_alone_equals_among_sixty(persistent):
    # alone 80 blocks or more; of 60 such registrations 8 (persistent) to 26 blocks
    among = run(range(60), persistent)
    for k in (0, 1, 2, 31, 59):
        (p, v), = run([k], persistent)
        assert np.array_equal(p, among[k][0]) and v == among[k][1]
