"""AXIS0 projections of a view table that ct_proj3d_views would not write: one
view's columns so far apart that a tile's bins pass the forward's 8 bits.  The
forward leaves that view out, as zeros, and says so in the error word; the other
views keep their bits."""

import ctypes

import numpy as np
import pytest
import torch

from scico_gb300 import _device, _lib, linop

pytestmark = pytest.mark.gpu
X3 = linop.XRayTransform3D


@pytest.mark.parametrize("shape", [(33, 20, 22), (130, 40, 36)])
def test_wide_view_is_left_out_and_reported(cuda, shape):
    lib = _lib.load()
    det = (shape[0], 60)
    H = X3(shape, X3.matrices_from_euler_angles(shape, det, "X", np.linspace(0, 3, 5)[:, None]), det)
    assert H.kind == "axis0"
    x = torch.rand(shape, generator=torch.Generator().manual_seed(1)).to(cuda)
    want = H.project(x)
    assert lib.ct_proj3d_errflag() == 0
    table = H.view_table.copy()
    table[2, 5:7] *= 16.0 / np.abs(table[2, 5:7]).sum()  # 240 bins a tile: still held
    table[3, 5:7] *= 17.0 / np.abs(table[3, 5:7]).sum()  # 255 and the bins beside them: not
    dev = torch.from_numpy(table).to(cuda)
    g = _lib.Geom3D()
    ctypes.memmove(ctypes.addressof(g), ctypes.addressof(H.geometry()), ctypes.sizeof(g))
    g.views = dev.data_ptr()
    fwd, _ = H.workspace_bytes()
    ws = _device.workspace(fwd)
    got = torch.full_like(want, float("nan"))
    _lib.call("ct_proj3d_fwd", ctypes.addressof(g), x.data_ptr(), got.data_ptr(), 1, ws.data_ptr(), ws.numel(),
              _device.stream())
    torch.cuda.synchronize()
    assert lib.ct_proj3d_errflag() == 1
    assert torch.count_nonzero(got[3]) == 0
    for v in (0, 1, 4):
        assert torch.equal(got[v], want[v])
    assert torch.isfinite(got[2]).all()
