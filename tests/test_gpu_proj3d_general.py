"""The GENERAL 3D kernels where their windows, bricks and fallbacks meet:
against the float32 oracle (rel l2 <= 1e-5, the projector's own tolerance:
bit-identical weights, another order of the sums).

Cases: sides around the 16-voxel windows and bricks, every marching axis, views
that need two or four phases of lanes, views outside the tile bounds (coarse
and fine voxels: the march and the global gathers), detectors smaller than the
shadow and off to one side, a single plane, and calls with no scratch or less
than the query asks for.
"""

import ctypes

import numpy as np
import pytest
import torch

from oracle import ctref
from scico_gb300 import _device, _lib, linop

pytestmark = pytest.mark.gpu
X3 = linop.XRayTransform3D


def _angles(seq, nv, seed):
    if len(seq) == 1:
        return np.linspace(0, np.pi, nv, endpoint=False)[:, None] + 0.1
    return np.random.default_rng(seed).uniform(0, np.pi, (nv, len(seq)))


CASES = [
    dict(shape=(15, 16, 17), det=(33, 31), seq="XYZ", nv=9),
    dict(shape=(1, 33, 40), det=(40, 52), seq="XYZ", nv=5),
    dict(shape=(33, 1, 18), det=(40, 40), seq="XYZ", nv=5),
    dict(shape=(20, 47, 1), det=(50, 21), seq="ZXY", nv=5),
    dict(shape=(48, 31, 65), det=(70, 70), seq="YZX", nv=12),
    dict(shape=(33, 40, 36), det=(17, 9), seq="XYZ", nv=6),  # cuts the shadow
    dict(shape=(24, 24, 24), det=(30, 30), seq="XYZ", nv=6, vs=[0.7, 0.6, 0.8]),  # two phases
    dict(shape=(24, 24, 24), det=(20, 20), seq="XYZ", nv=6, vs=[0.4, 0.4, 0.4]),  # four phases, or the march
    dict(shape=(20, 20, 20), det=(20, 20), seq="XYZ", nv=6, vs=[0.2, 0.2, 0.2]),  # the march
    dict(shape=(12, 14, 10), det=(40, 40), seq="XYZ", nv=6, vs=[2.0, 2.5, 3.0]),  # the march, global gathers
    dict(shape=(12, 40, 10), det=(40, 60), seq="XYZ", nv=6, vs=[1.0, 1.5, 1.2]),  # some of each
]


def _op(c):
    M = X3.matrices_from_euler_angles(c["shape"], c["det"], c["seq"], _angles(c["seq"], c["nv"], c["nv"]),
                                      voxel_spacing=c.get("vs"))
    H = X3(c["shape"], M, c["det"])
    assert H.kind == "general"
    return H, M.astype(np.float32)


@pytest.mark.parametrize("c", CASES, ids=lambda c: f"{c['shape']}-{c['seq']}-{c.get('vs')}")
def test_windows_and_bricks(cuda, c):
    H, M = _op(c)
    rng = np.random.default_rng(1)
    x = rng.random((2,) + c["shape"]).astype(np.float32)
    y = H.project(torch.from_numpy(x).to(cuda))
    assert torch.equal(y, H.project(torch.from_numpy(x).to(cuda)))
    ys = rng.standard_normal((2,) + H.output_shape).astype(np.float32)
    b = H.back_project(torch.from_numpy(ys).to(cuda))
    for k in range(2):
        assert ctref.rel_l2(y[k].cpu().numpy(), ctref.xray3d_project(x[k], M, c["det"], np.float32)) <= 1e-5
        assert ctref.rel_l2(b[k].cpu().numpy(), ctref.xray3d_back_project(ys[k], M, c["shape"], np.float32)) <= 1e-5


def _call(name, H, src, out_shape, ws, nbytes):
    g = H.geometry()
    out = torch.empty(out_shape, device=src.device)
    st = getattr(_lib.load(), name)(ctypes.addressof(g), src.data_ptr(), out.data_ptr(), 1,
                                    ws.data_ptr() if ws is not None else None, nbytes,
                                    torch.cuda.current_stream().cuda_stream)
    return st, out


def test_scratch_limits(cuda):
    """No scratch, too little and what the query reports: the same projections
    (a general geometry never needed forward scratch); the adjoint is refused
    below the scratch it always needed and takes fewer splits below the query."""
    c = dict(shape=(40, 33, 57), det=(60, 60), seq="XYZ", nv=32)
    H, M = _op(c)
    x = torch.rand(c["shape"], generator=torch.Generator().manual_seed(1)).to(cuda)
    y = torch.rand(H.output_shape, generator=torch.Generator().manual_seed(2)).to(cuda)
    fwd, adj = H.workspace_bytes()
    ws = _device.workspace(max(fwd, adj))
    want = ctref.xray3d_project(x.cpu().numpy(), M, c["det"], np.float32)
    for w, n in ((None, 0), (ws, fwd - 1), (ws, fwd)):
        st, out = _call("ct_proj3d_fwd", H, x, H.output_shape, w, n)
        assert st == _lib.CT_OK
        assert ctref.rel_l2(out.cpu().numpy(), want) <= 1e-5
    want = ctref.xray3d_back_project(y.cpu().numpy(), M, c["shape"], np.float32)
    voxels = int(np.prod(c["shape"]))
    least = (2 * voxels * 4 + 255) // 256 * 256  # 295 blocks of 256 voxels: three splits asked, 2 or more kept
    st, _ = _call("ct_proj3d_adj", H, y, c["shape"], None, 0)
    assert st == _lib.CT_ERR_WORKSPACE
    st, _ = _call("ct_proj3d_adj", H, y, c["shape"], ws, least // 2)
    assert st == _lib.CT_ERR_WORKSPACE
    for n in (adj, (3 * voxels * 4 + 255) // 256 * 256):
        st, out = _call("ct_proj3d_adj", H, y, c["shape"], ws, n)
        assert st == _lib.CT_OK
        assert ctref.rel_l2(out.cpu().numpy(), want) <= 1e-5


def test_capture(cuda):
    """The forward's launches replay inside a stream capture."""
    H, M = _op(CASES[4])
    x = torch.rand(H.input_shape, generator=torch.Generator().manual_seed(1)).to(cuda)
    want = H.project(x).clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = H.project(x)
    out.zero_()
    g.replay()
    assert torch.equal(out, want)
