"""B-spline grids of many small cells, where a warp sums a cell: against the FP64 oracle."""
import numpy as np
import pytest

import itk_gb300 as gb
from cases import run_oracle
from conftest import MATTES_VALUE_ATOL, assert_deriv_close, assert_value_close
from itk_gb300 import data

pytestmark = pytest.mark.gpu

SIZE, MESH = (60, 56, 52), (16, 15, 17)


def points_of(form):
    rng = np.random.default_rng(5)
    last = np.array(SIZE) - 1.0
    if form == "dense":  # 27 to 64 samples to a cell
        return None
    few = rng.uniform(0.0, 1.0, (15000, 3)) * last  # none to a dozen
    if form == "few":
        return few.astype(np.float32)
    # and cells of 31, 32, 33, 127, 129, 512, 513 and 3000 samples, one side of a batch, a fold and a chunk each
    spots = rng.choice(14 * 13 * 15, 8, replace=False)
    cell = last / np.array(MESH)
    many = [(np.array([1 + s % 14, 1 + s // 14 % 13, 1 + s // 182]) + rng.uniform(0.01, 0.99, (n, 3))) * cell
            for s, n in zip(spots, (31, 32, 33, 127, 129, 512, 513, 3000))]
    return np.concatenate([few] + many).astype(np.float32)


def make_metric(kind, fixed, moving, transform, gradient, points, bins):
    m = {"msq": gb.MeanSquaresImageToImageMetricv4, "mattes": gb.MattesMutualInformationImageToImageMetricv4,
         "jhmi": gb.JointHistogramMutualInformationImageToImageMetricv4}[kind]()
    m.SetFixedImage(fixed)
    m.SetMovingImage(moving)
    m.SetMovingTransform(transform)
    m.SetMovingImageGradientImage(gradient)
    if kind != "msq":
        m.SetNumberOfHistogramBins(bins)
    if points is not None:
        m.SetVirtualSampledPointSet(points)
        m.SetUseSampledPointSet(True)
    m.Initialize()
    return m


@pytest.mark.parametrize("kind", ["msq", "mattes", "jhmi"])
@pytest.mark.parametrize("form", ["dense", "few", "uneven"])
def test_small_cells_match_the_oracle(kind, form):
    fixed, moving, _, _ = data.pair_bspline(SIZE, (4, 4, 4), instance=1, multimodal_map=kind != "msq")
    gradient = data.gradient_image(moving)
    b = data.random_bspline_coefficients(data.bspline_over_image(fixed, MESH), 3, 1.0)
    points = points_of(form)
    bins = 20 if kind == "jhmi" else 50
    m = make_metric(kind, fixed, moving, b, gradient, points, bins)
    v, d = m.GetValueAndDerivative()
    r = run_oracle(kind, fixed, moving, b, gradient=gradient, points=points, bins=bins)
    assert r["status"] == 0 and m.GetNumberOfValidPoints() == r["nvalid"]
    assert_value_close(v, r["value"], atol=MATTES_VALUE_ATOL if kind == "mattes" else 0.0)
    assert_deriv_close(d, r["derivative"])
    v2, d2 = m.GetValueAndDerivative()
    assert v2 == v and np.array_equal(d2, d)
