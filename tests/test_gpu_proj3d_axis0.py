"""The AXIS0 3D kernels at slice counts around their 32 / 64 / 128-slice groups,
tile edges of 16 pixels, short view runs, detectors that cut the shadow or
leave slices off it, and reduced scratch, against the float32 oracle (rel l2 <=
1e-5: bit-identical weights, another order of the sums)."""

import ctypes

import numpy as np
import pytest
import torch

from oracle import ctref
from scico_gb300 import _device, _lib, linop

pytestmark = pytest.mark.gpu
X3 = linop.XRayTransform3D

CASES = [
    dict(shape=(1, 16, 16), det=(1, 24), nv=3),
    dict(shape=(31, 17, 15), det=(31, 25), nv=5),
    dict(shape=(33, 15, 40), det=(33, 44), nv=9),
    dict(shape=(64, 33, 16), det=(64, 38), nv=17),
    dict(shape=(65, 20, 20), det=(65, 12), nv=33),  # cuts the shadow
    dict(shape=(128, 16, 48), det=(128, 52), nv=4),
    dict(shape=(131, 34, 18), det=(131, 40), nv=66),
    dict(shape=(40, 20, 22), det=(44, 31), nv=7),  # rows off the slices (offset 2)
    dict(shape=(260, 16, 17), det=(260, 25), nv=40),
    dict(shape=(33, 21, 19), det=(33, 29), nv=80),  # view splits of a volume that is no whole number of quads
]


def _op(c, angles=None):
    a = np.linspace(0, np.pi, c["nv"], endpoint=False) if angles is None else angles
    M = X3.matrices_from_euler_angles(c["shape"], c["det"], "X", a[:, None])
    H = X3(c["shape"], M, c["det"])
    assert H.kind == "axis0"
    return H, M.astype(np.float32)


@pytest.mark.parametrize("c", CASES, ids=lambda c: f"{c['shape']}-{c['det']}-{c['nv']}")
def test_slice_groups_and_tiles(cuda, c):
    H, M = _op(c)
    rng = np.random.default_rng(c["nv"])
    x = rng.random((2,) + c["shape"]).astype(np.float32)
    y = H.project(torch.from_numpy(x).to(cuda))
    ys = rng.standard_normal((2,) + H.output_shape).astype(np.float32)
    b = H.back_project(torch.from_numpy(ys).to(cuda))
    for k in range(2):
        assert ctref.rel_l2(y[k].cpu().numpy(), ctref.xray3d_project(x[k], M, c["det"], np.float32)) <= 1e-5
        assert ctref.rel_l2(b[k].cpu().numpy(), ctref.xray3d_back_project(ys[k], M, c["shape"], np.float32)) <= 1e-5


def test_adjoint_splits_and_scratch(cuda):
    """Every view-split count gives the same back projection to rounding, the
    scratch a call always needed is enough, and less is refused."""
    c = dict(shape=(40, 40, 40), det=(40, 57), nv=96)
    H, M = _op(c)
    y = torch.rand(H.output_shape, generator=torch.Generator().manual_seed(2)).to(cuda)
    want = ctref.xray3d_back_project(y.cpu().numpy(), M, c["shape"], np.float32)
    g = H.geometry()
    one = 4 * int(np.prod(c["shape"]))
    _, adj = H.workspace_bytes()
    ws = _device.workspace(adj)
    ok = _lib.load().ct_proj3d_adj
    for n, status in ((0, _lib.CT_ERR_WORKSPACE), (2 * one, _lib.CT_ERR_WORKSPACE), (6 * one, _lib.CT_OK),
                      (adj, _lib.CT_OK)):
        out = torch.empty(c["shape"], device=cuda)
        st = ok(ctypes.addressof(g), y.data_ptr(), out.data_ptr(), 1, ws.data_ptr() if n else None, n,
                torch.cuda.current_stream().cuda_stream)
        assert st == status
        if st == _lib.CT_OK:
            assert ctref.rel_l2(out.cpu().numpy(), want) <= 1e-5
