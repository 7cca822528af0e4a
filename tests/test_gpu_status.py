"""gb_metric_synchronize returns the status of the last evaluation, whoever asked for it."""
import numpy as np
import pytest

import itk_gb300 as gb
from cases import small_pair
from itk_gb300 import _capi, data

pytestmark = pytest.mark.gpu

METRICS = {"msq": gb.MeanSquaresImageToImageMetricv4, "mattes": gb.MattesMutualInformationImageToImageMetricv4,
           "jhmi": gb.JointHistogramMutualInformationImageToImageMetricv4, "corr": gb.CorrelationImageToImageMetricv4}


@pytest.mark.parametrize("kind", list(METRICS))
@pytest.mark.parametrize("derivative", [False, True])
def test_status_follows_the_last_evaluation(kind, derivative):
    torch = pytest.importorskip("torch")
    fixed, moving, t = small_pair((40, 36, 32), config=1, multimodal=True)
    m = METRICS[kind]()
    m.SetFixedImage(fixed)
    m.SetMovingImage(moving)
    m.SetMovingTransform(t)
    m.SetMovingImageGradientImage(data.gradient_image(moving))
    m.Initialize()
    near = np.asarray(t.GetParameters(), np.float64)
    far = near + np.array([0.0] * 9 + [1e4] * 3)
    out = torch.zeros(2 + near.size, dtype=torch.float64, device="cuda")

    def on_host(p, expected):
        t.SetParameters(p)
        for _ in range(2):  # captured, then replayed
            try:
                m.GetValueAndDerivative() if derivative else m.GetValue()
            except gb.ExceptionObject:
                pass
            assert m.synchronize() == expected

    def on_device(p, expected):
        d = torch.tensor(p, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        m.evaluate_device(d.data_ptr(), out.data_ptr(), derivative)
        assert m.synchronize() == expected

    none = _capi.GB_ERR_NO_VALID_POINTS
    on_device(near, 0)
    on_host(far, none)
    on_host(near, 0)
    on_device(far, none)
    on_host(near, 0)
    on_device(near, 0)
    on_host(far, none)
    on_device(near, 0)
