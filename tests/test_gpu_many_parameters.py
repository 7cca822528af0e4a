"""The host call's results of one block of the epilogue kernel (up to 1024) and of several."""
import numpy as np
import pytest

import itk_gb300 as gb
from cases import small_pair
from itk_gb300 import data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [3, 4, 8, 30])  # 650, 1031, 3995 and 107813 results
@pytest.mark.parametrize("kind", ["msq", "jhmi"])
def test_host_call_gives_the_device_calls_bits(mesh, kind):
    torch = pytest.importorskip("torch")
    fixed, moving, a = small_pair((40, 36, 32), config=1, multimodal=True)
    b = gb.BSplineTransform()
    b.SetTransformDomain(np.zeros(3), np.array([39.0, 35.0, 31.0]), (mesh,) * 3)
    b.SetParameters(np.random.default_rng(mesh).uniform(-0.5, 0.5, b.GetNumberOfParameters()))
    t = gb.CompositeTransform()
    t.AddTransform(a)
    t.AddTransform(b)
    m = {"msq": gb.MeanSquaresImageToImageMetricv4, "jhmi": gb.JointHistogramMutualInformationImageToImageMetricv4}[kind]()
    m.SetFixedImage(fixed)
    m.SetMovingImage(moving)
    m.SetMovingTransform(t)
    m.SetMovingImageGradientImage(data.gradient_image(moving))
    m.Initialize()
    v, d = m.GetValueAndDerivative()
    p = torch.tensor(np.asarray(t.GetParameters()), dtype=torch.float64, device="cuda")
    out = torch.full((2 + d.size,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    m.evaluate_device(p.data_ptr(), out.data_ptr(), True)
    assert m.synchronize() == 0
    o = out.cpu().numpy()
    assert o[0] == v and o[1] == m.GetNumberOfValidPoints() and np.array_equal(o[2:], d)
