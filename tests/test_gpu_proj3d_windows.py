"""GENERAL 3D projections with nearly parallel matrix rows, which the forward's
windows leave to the march: against the float32 oracle (rel l2 <= 1e-5, the
projector's own tolerance), alone and beside ordinary views."""

import numpy as np
import pytest
import torch

from oracle import ctref
from scico_gb300 import linop

pytestmark = pytest.mark.gpu
X3 = linop.XRayTransform3D

SHAPE, DET = (97, 128, 111), (128, 181)
PARALLEL = [[1.1872672e-01, 1.5680777e-01, -1.2382731e-01, 5.1078472e01],
            [2.5399225, 3.3546038, -2.6490467, -1.3085880e02]]


@pytest.mark.parametrize("beside", [0, 2])
def test_nearly_parallel_rows(cuda, beside):
    M = np.array([PARALLEL])
    if beside:
        ang = np.random.default_rng(1).uniform(0, np.pi, (beside, 3))
        M = np.concatenate([X3.matrices_from_euler_angles(SHAPE, DET, "XYZ", ang), M])
    M = M.astype(np.float32)
    H = X3(SHAPE, M, DET)
    assert H.kind == "general"
    rng = np.random.default_rng(2)
    x = rng.random(SHAPE).astype(np.float32)
    y = rng.random(H.output_shape).astype(np.float32)
    got = H.project(torch.from_numpy(x).to(cuda)).cpu().numpy()
    want = ctref.xray3d_project(x, M, DET, np.float32, np.float64)
    for v in range(len(M)):
        assert ctref.rel_l2(got[v], want[v]) <= 1e-5
    got = H.back_project(torch.from_numpy(y).to(cuda)).cpu().numpy()
    assert ctref.rel_l2(got, ctref.xray3d_back_project(y, M, SHAPE, np.float32)) <= 1e-5
