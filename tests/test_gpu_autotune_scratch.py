"""The 3D tuner stays inside the scratch it is given: with no more than the
forward's, view splits whose partial volumes do not fit are no candidates.  The
bytes after the scratch keep their values."""

import ctypes

import numpy as np
import pytest
import torch

from scico_gb300 import _lib, linop

pytestmark = pytest.mark.gpu
X3 = linop.XRayTransform3D


@pytest.mark.parametrize("shape,det,nv,seq", [((64, 128, 128), (64, 182), 20, "X"), ((40, 33, 57), (60, 60), 12, "XYZ")])
def test_tuner_keeps_to_its_scratch(cuda, shape, det, nv, seq):
    ang = np.linspace(0.1, 3, nv)
    H = X3(shape, X3.matrices_from_euler_angles(shape, det, seq, ang[:, None] if seq == "X" else np.stack([ang] * 3, 1)), det)
    volume = 4 * int(np.prod(shape))
    # what a call needs: the forward's scratch (general: none), and for this few views one split
    given = H.workspace_bytes()[0] if H.kind == "axis0" else 0
    assert given < 2 * volume
    whole = torch.full((given + 5 * volume + 4096,), 0x5A, dtype=torch.uint8, device=cuda)
    vol, proj = torch.zeros(shape, device=cuda), torch.zeros(H.output_shape, device=cuda)
    out = _lib.Proj3dSchedule()
    lib = _lib.load()
    try:
        _lib.call("ct_proj3d_autotune", ctypes.addressof(H.geometry()), vol.data_ptr(), proj.data_ptr(), whole.data_ptr(),
                  given, 2, torch.cuda.current_stream().cuda_stream, ctypes.addressof(out))
        assert out.tuned == 1 and out.adj_splits >= 1
        assert bool((whole[given:] == 0x5A).all())
    finally:
        lib.ct_proj3d_schedule_clear()


def test_query_does_not_depend_on_the_schedule(cuda):
    """The scratch asked for after tuning is the scratch asked for before."""
    shape, nv = (64, 64, 64), 20
    M = X3.matrices_from_euler_angles(shape, (112, 112), "XYZ", np.stack([np.linspace(0.1, 3, nv)] * 3, 1))
    H = X3(shape, M, (112, 112))
    before = H.workspace_bytes()
    try:
        assert H.autotune()["tuned"]
        assert X3(shape, M, (112, 112)).workspace_bytes() == before
    finally:
        _lib.load().ct_proj3d_schedule_clear()
