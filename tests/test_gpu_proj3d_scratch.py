"""What a general 3D projection allocates: no scratch where no view's windows
use it, no copy of the volume where no view marches along axis 2, and none at
all where that much memory is not free; the projections stay the oracle's
(rel l2 <= 1e-5) or, scratch to scratch, the same bits."""

import ctypes

import numpy as np
import pytest
import torch

from oracle import ctref
from scico_gb300 import _device, _lib, linop

pytestmark = pytest.mark.gpu
X3 = linop.XRayTransform3D
SLACK = 1 << 20  # the allocator's rounding


def _op(shape, det, angles, seq="XYZ", vs=None):
    M = X3.matrices_from_euler_angles(shape, det, seq, angles, voxel_spacing=vs).astype(np.float32)
    H = X3(shape, M, det)
    assert H.kind == "general"
    return H, M


def _allocated(H, x):
    """Bytes that a projection allocates at its peak, and the projection."""
    H.project(x)  # tables on the device
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    y = H.project(x)
    return torch.cuda.max_memory_allocated() - before, y


def _fwd(H, x, nbytes):
    ws = _device.workspace(nbytes)
    out = torch.empty(H.output_shape, device=x.device)
    _lib.call("ct_proj3d_fwd", ctypes.addressof(H.geometry()), x.data_ptr(), out.data_ptr(), 1, ws.data_ptr(), nbytes,
              torch.cuda.current_stream().cuda_stream)
    return out


def test_no_scratch_where_no_view_uses_it(cuda):
    ang = np.random.default_rng(1).uniform(0, np.pi, (4, 3))
    H, M = _op((40, 44, 36), (90, 100), ang, vs=[2.0, 2.5, 3.0])
    x = torch.rand(H.input_shape, generator=torch.Generator().manual_seed(1)).to(cuda)
    used, y = _allocated(H, x)
    assert used <= 4 * y.numel() + SLACK
    assert ctref.rel_l2(y.cpu().numpy(), ctref.xray3d_project(x.cpu().numpy(), M, H.det_shape, np.float32)) <= 1e-5


def test_no_copy_of_the_volume_where_no_view_marches_along_axis_2(cuda):
    shape = (120, 120, 120)
    # small turns: the rays run close to the axis that the matrix drops first (axis 2 without a turn)
    ang = np.stack([np.linspace(1.2, 1.9, 3), np.full(3, 0.2)], axis=1)
    H, M = _op(shape, (140, 180), ang, seq="XY")
    assert not (H.view_table[:, 8] == 2).any()
    x = torch.rand(shape, generator=torch.Generator().manual_seed(2)).to(cuda)
    full = H.workspace_bytes()[0]
    volume = 4 * x.numel()
    used, y = _allocated(H, x)
    assert used <= 4 * y.numel() + full - volume + SLACK
    assert torch.equal(y, _fwd(H, x, full))


@pytest.mark.parametrize("less", [1, 256])
def test_views_along_axis_2_without_their_copy(cuda, less):
    ang = np.random.default_rng(3).uniform(0, np.pi, (8, 3))
    H, M = _op((33, 40, 28), (60, 64), ang)
    along = torch.from_numpy(H.view_table[:, 8] == 2)
    assert along.any() and not along.all()
    x = torch.rand(H.input_shape, generator=torch.Generator().manual_seed(4)).to(cuda)
    full = H.workspace_bytes()[0]
    want, got = _fwd(H, x, full), _fwd(H, x, full - less)
    assert torch.equal(got.cpu()[~along], want.cpu()[~along])
    assert ctref.rel_l2(got.cpu().numpy(), ctref.xray3d_project(x.cpu().numpy(), M, H.det_shape, np.float32)) <= 1e-5


def test_projects_where_the_scratch_does_not_fit(cuda, monkeypatch):
    ang = np.random.default_rng(5).uniform(0, np.pi, (4, 3))
    H, M = _op((24, 30, 26), (50, 50), ang)
    x = torch.rand(H.input_shape, generator=torch.Generator().manual_seed(6)).to(cuda)

    def none_free(nbytes):
        raise torch.cuda.OutOfMemoryError("no memory for the scratch")

    monkeypatch.setattr(_device, "workspace", none_free)
    y = H.project(x)
    assert ctref.rel_l2(y.cpu().numpy(), ctref.xray3d_project(x.cpu().numpy(), M, H.det_shape, np.float32)) <= 1e-5
