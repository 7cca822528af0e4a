"""Fixed values of single sample points, bit for bit.

Initialize interpolates the fixed image at every sample point in FP64 and keeps the value as a
float; most points take FP32 pairs whose error bound says that the float is the same.  A metric
of one point over an empty moving image has that float's square as its value, in FP32."""
import numpy as np
import pytest

import itk_gb300 as gb

pytestmark = pytest.mark.gpu


def point_to_index(image):
    """ImageBase's physical-to-index matrix, in the order of the library's own inverse."""
    a = (image.direction * image.spacing[None, :]).ravel()
    c = [a[4] * a[8] - a[5] * a[7], a[5] * a[6] - a[3] * a[8], a[3] * a[7] - a[4] * a[6]]
    i = 1.0 / (a[0] * c[0] + a[1] * c[1] + a[2] * c[2])
    return np.array([c[0] * i, (a[2] * a[7] - a[1] * a[8]) * i, (a[1] * a[5] - a[2] * a[4]) * i,
                     c[1] * i, (a[0] * a[8] - a[2] * a[6]) * i, (a[2] * a[3] - a[0] * a[5]) * i,
                     c[2] * i, (a[1] * a[6] - a[0] * a[7]) * i, (a[0] * a[4] - a[1] * a[3]) * i]).reshape(3, 3)


def interpolated(image, point):
    """The FP64 trilinear value at an inner point, rounded to float."""
    m, p = point_to_index(image), point.astype(np.float64)
    v = image.array.astype(np.float64)
    c = np.zeros(3)
    for r in range(3):
        for k in range(3):
            c[r] = c[r] + m[r, k] * (p[k] - image.origin[k])
    b = np.floor(c).astype(int)
    v = v[b[2]:b[2] + 2, b[1]:b[1] + 2, b[0]:b[0] + 2]
    for t in c - b:  # x, y, z: the last axis of what is left
        v = v[..., 0] + (v[..., 1] - v[..., 0]) * t
    return np.float32(v)


def initialized_square(image, moving, point):
    t = gb.AffineTransform()
    m = gb.MeanSquaresImageToImageMetricv4()
    m.SetFixedImage(image)
    m.SetMovingImage(moving)
    m.SetMovingTransform(t)
    m.SetUseMovingImageGradientFilter(False)
    m.SetVirtualSampledPointSet(point)
    m.SetUseSampledPointSet(True)
    m.Initialize()
    return m.GetValue()


def check(image, moving, point):
    f = interpolated(image, point)
    assert initialized_square(image, moving, point) == float(f * f)


# An oblique grid and a point of it whose pair index is off by 2.2, 2.4 and 1.1e-12 along the
# three axes, and corners with a slope of 1 along each: the value is off by 5.7e-12, and for
# these values of the near corner a boundary between two floats lies in between.
DIRECTION = [[0.19202969208283716, -0.02074640819995066, -0.9811698038083785],
             [-0.8917186732061274, -0.4211993854935796, -0.1656166824789549],
             [-0.40983216712951487, 0.9067307561821383, -0.09938274789566526]]
SPACING = (2.9477452643605653, 1.6690043751817292, 1.1858999535559578)
POINT = np.array([float.fromhex("-0x1.acd968p+6"), float.fromhex("-0x1.fc4a52p+8"), float.fromhex("0x1.bf8b8ap+5")],
                 np.float32)


@pytest.mark.parametrize("near,far", [("6d59d639", 1.0), ("efa2a93a", 1.0), ("47e6c1ba", 1.0), ("b16ec0b9", 1.0),
                                      ("2ad8fab9", -1.0), ("4c0e8d3a", -1.0), ("9ae8c23a", -1.0), ("b802313a", -1.0)])
def test_value_next_to_a_rounding_boundary(near, far):
    a = np.zeros((158, 163, 142), np.float32)
    a[155:157, 160:162, 139:141] = far
    a[155, 160, 139] = np.frombuffer(bytes.fromhex(near), "<f4")[0]
    image, moving = (gb.Image(x, SPACING, direction=DIRECTION) for x in (a, np.zeros_like(a)))
    check(image, moving, POINT)


@pytest.mark.parametrize("spacing,oblique", [(1.0, False), (0.7, True), (1e35, False), (1e-33, True)])
def test_values_of_random_points(spacing, oblique):
    rng = np.random.default_rng(3)
    a = rng.uniform(-1.0, 1.0, (24, 24, 24)).astype(np.float32)
    kw = dict(spacing=(spacing,) * 3, direction=DIRECTION if oblique else None)
    image, moving = gb.Image(a, **kw), gb.Image(np.zeros_like(a), **kw)
    for index in rng.uniform(1.0, 22.0, (100, 3)):
        check(image, moving, image.TransformIndexToPhysicalPoint(index).astype(np.float32))
