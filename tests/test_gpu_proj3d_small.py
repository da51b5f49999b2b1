"""GENERAL 3D back projection of small and thin volumes, which a voxel per thread
serves, and of the sizes around the rule that chooses it: against the float32
oracle (rel l2 <= 1e-5), with hot pixels voxel by voxel ((views + 16) units of
2^-24 of the value, as each product, interpolation and sum rounds once or
twice), and with scratch for fewer splits."""

import ctypes

import numpy as np
import pytest
import torch

from oracle import ctref
from scico_gb300 import _device, _lib, linop

pytestmark = pytest.mark.gpu
X3 = linop.XRayTransform3D


def _op(shape, nv, vs=None):
    ang = np.random.default_rng(nv).uniform(0, np.pi, (nv, 3))
    det = (int(np.linalg.norm(shape) * max(vs or [1])) + 1,) * 2
    M = X3.matrices_from_euler_angles(shape, det, "XYZ", ang, voxel_spacing=vs).astype(np.float32)
    H = X3(shape, M, det)
    assert H.kind == "general"
    return H, M


@pytest.mark.parametrize("shape,nv,vs", [((1, 1, 1), 1, None), ((8, 8, 8), 3, None), ((15, 17, 1), 40, None),
                                         ((24, 28, 20), 12, None), ((4, 100, 90), 33, None), ((24, 24, 24), 12, [2.0] * 3),
                                         ((40, 40, 40), 20, None), ((48, 48, 48), 20, None), ((200, 20, 20), 65, None)])
def test_small_volumes(cuda, shape, nv, vs):
    H, M = _op(shape, nv, vs)
    y = np.random.default_rng(1).uniform(0.001, 1.0, H.output_shape).astype(np.float32)
    y[:, H.det_shape[0] // 2, H.det_shape[1] // 2] = 1e7
    want = ctref.xray3d_back_project(y, M, shape, np.float32, np.float64)
    dev = torch.from_numpy(y).to(cuda)
    got = H.back_project(dev)
    assert torch.equal(got, H.back_project(dev))
    got = got.cpu().numpy()
    assert ctref.rel_l2(got, want) <= 1e-5
    assert np.all(np.abs(got - want) <= (nv + 16) * 2.0**-24 * want)
    # two splits' scratch, or as much as a call of so few views may need
    splits = H.schedule()["adj_splits"]
    if splits > 2:
        nbytes = 2 * 4 * int(np.prod(shape)) + 256
        ws = _device.workspace(nbytes)
        out = torch.empty(shape, device=cuda)
        st = _lib.load().ct_proj3d_adj(ctypes.addressof(H.geometry()), dev.data_ptr(), out.data_ptr(), 1, ws.data_ptr(),
                                       nbytes, torch.cuda.current_stream().cuda_stream)
        assert st in (_lib.CT_OK, _lib.CT_ERR_WORKSPACE)
        if st == _lib.CT_OK:
            assert ctref.rel_l2(out.cpu().numpy(), want) <= 1e-5


def _us(fn):
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(20):
            fn()
    best = float("inf")
    for _ in range(8):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        graph.replay()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 50.0)
    return best


@pytest.mark.parametrize("shape,nv,vs", [((16, 16, 16), 6, None), ((24, 24, 24), 12, [2.0] * 3)])
def test_small_volumes_are_not_served_by_bricks(cuda, shape, nv, vs):
    """A view's chain through a brick takes these volumes 10 and 42 us, a voxel per
    thread 2.5 and 5 us; the forward, whose work is several times the adjoint's,
    is the yardstick (14 and 44 us)."""
    H, _ = _op(shape, nv, vs)
    x, y = torch.rand(shape, device=cuda), torch.rand(H.output_shape, device=cuda)
    assert _us(lambda: H.back_project(y)) <= 0.5 * _us(lambda: H.project(x))
