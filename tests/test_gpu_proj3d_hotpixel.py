"""GENERAL 3D back projection beside detector pixels far above their neighbours,
infinite ones and ones of float32's size: every voxel against the float32 model
with 64-bit sums.

With non-negative data a voxel is a sum of positive products: each product and
each interpolation rounds a few times, each view's addition once, so voxel by
voxel the error is at most (views + 16) units of 2^-24 of the value itself,
whatever the pixels that the voxel does not touch."""

import numpy as np
import pytest
import torch

from oracle import ctref
from scico_gb300 import linop

pytestmark = pytest.mark.gpu
X3 = linop.XRayTransform3D

SHAPE, DET, NV = (20, 27, 22), (40, 44), 6


def _op(vs):
    ang = np.random.default_rng(5).uniform(0, np.pi, (NV, 3))
    M = X3.matrices_from_euler_angles(SHAPE, DET, "XYZ", ang, voxel_spacing=vs).astype(np.float32)
    H = X3(SHAPE, M, DET)
    assert H.kind == "general"
    return H, M


# staged tiles; tiles that hang over the detector's edge; views that gather from memory
SPACINGS = [None, [1.1, 1.2, 1.3], [2.0, 2.5, 3.0]]


@pytest.mark.parametrize("vs", SPACINGS, ids=str)
@pytest.mark.parametrize("hot", [3e4, 1e9])
def test_hot_pixels(cuda, vs, hot):
    H, M = _op(vs)
    rng = np.random.default_rng(3)
    y = rng.uniform(0.001, 1.0, H.output_shape).astype(np.float32)
    y[:, 18, 20] = hot
    y[:, 23, 25] = hot
    got = H.back_project(torch.from_numpy(y).to(cuda)).cpu().numpy()
    want = ctref.xray3d_back_project(y, M, SHAPE, np.float32, np.float64)
    assert np.all(np.abs(got - want) <= (NV + 16) * 2.0**-24 * want)


@pytest.mark.parametrize("vs", SPACINGS, ids=str)
def test_infinite_pixel(cuda, vs):
    H, M = _op(vs)
    y = np.random.default_rng(4).uniform(0.5, 1.0, H.output_shape).astype(np.float32)
    y[1, 19, 22] = np.inf
    got = H.back_project(torch.from_numpy(y).to(cuda)).cpu().numpy()
    with np.errstate(invalid="ignore"):
        want = ctref.xray3d_back_project(y, M, SHAPE, np.float32)
    assert np.isposinf(want).any()
    assert np.array_equal(np.isposinf(got), np.isposinf(want))
    assert np.array_equal(np.isnan(got), np.isnan(want))


@pytest.mark.parametrize("vs", SPACINGS, ids=str)
def test_large_pixels_stay_finite(cuda, vs):
    H, M = _op(vs)
    y = np.zeros(H.output_shape, np.float32)
    y[2] = np.random.default_rng(6).choice([-3e38, 3e38], DET)
    assert torch.isfinite(H.back_project(torch.from_numpy(y).to(cuda))).all()
