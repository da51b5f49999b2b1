"""The 2D adjoint with two images a CTA (batches) against one image at a time:
the same sums in the same order for the same view splits, so a batch differs
from its images by the split order alone (rel l2 <= 2e-6, a few float32
roundings of a sum of hundreds of terms); against the float64 oracle rel l2 <=
1e-5 as the projector's own tests; odd batches, sides and views, large |Px|
(general floor path), and reduced scratch."""

import ctypes

import numpy as np
import pytest
import torch

from oracle import ctref
from scico_gb300 import _device, _lib, linop

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize("shape,nv,batch,kw", [
    ((64, 64), 33, 2, {}), ((65, 63), 40, 3, {}), ((130, 200), 96, 5, {}), ((128, 96), 180, 16, {}),
    ((301, 300), 64, 4, {}), ((303, 303), 40, 4, {}),  # the split sum in quads, and too odd for them
   
    ((40, 30), 64, 7, dict(det_count=20)), ((50, 50), 48, 4, dict(y0=-3.0e6, det_count=71)),
    ((64, 70), 17, 2, dict(dx=0.4))], ids=str)
def test_batch_matches_single(cuda, shape, nv, batch, kw):
    ang = np.linspace(0, np.pi, nv, endpoint=False)
    A = linop.XRayTransform2D(shape, ang, **kw)
    y = torch.rand((batch,) + A.output_shape, generator=torch.Generator().manual_seed(batch)).to(cuda)
    got = A.back_project(y)
    assert torch.equal(got, A.back_project(y))
    for k in range(batch):
        one = A.back_project(y[k].contiguous())
        assert _rel(got[k], one) <= 2e-6 if float(one.abs().max()) > 0 else torch.equal(got[k], one)
    if "y0" not in kw:
        g = ctref.xray2d_defaults(shape, ang, dx=kw.get("dx"), det_count=kw.get("det_count"))
        ref = ctref.xray2d_back_project(y[-1].cpu().numpy(), g, np.float64)
        assert ctref.rel_l2(got[-1].cpu().numpy(), ref) <= 1e-5


def test_reduced_scratch(cuda):
    """The scratch that a call has always needed is enough; less is refused."""
    A = linop.XRayTransform2D((96, 96), np.linspace(0, np.pi, 180, endpoint=False))
    batch, img = 16, 16 * 96 * 96 * 4
    y = torch.rand((batch,) + A.output_shape, generator=torch.Generator().manual_seed(1)).to(cuda)
    want = A.back_project(y)
    g = A.geometry()
    _, adj = A.workspace_bytes(batch)
    ws = _device.workspace(adj)
    for n, ok in ((adj, True), (11 * img, True), (10 * img, False), (0, False)):
        out = torch.empty((batch, 96, 96), device=cuda)
        st = _lib.load().ct_proj2d_adj(ctypes.addressof(g), y.data_ptr(), out.data_ptr(), batch,
                                       ws.data_ptr() if n else None, n, torch.cuda.current_stream().cuda_stream)
        assert st == (_lib.CT_OK if ok else _lib.CT_ERR_WORKSPACE)
        if ok:
            assert _rel(out, want) <= 2e-6


@pytest.mark.parametrize("shape,nv,batch", [((70, 100), 60, 100), ((300, 200), 91, 8), ((33, 66), 7, 900), ((40, 70), 1, 2000),
                                            ((64, 64), 45, 90), ((500, 257), 200, 1), ((90, 80), 23, 120)], ids=str)
def test_forward_runs_of_views(cuda, shape, nv, batch):
    """Long and short runs of views a CTA (large problems) against one round of even runs: no sum depends on the
    runs, so each image's projections are the same bits as alone, and each view's as in a scan of a few views."""
    ang = np.linspace(0, np.pi, nv, endpoint=False)
    A = linop.XRayTransform2D(shape, ang)
    x = torch.rand((batch,) + shape, generator=torch.Generator().manual_seed(nv)).to(cuda)
    got = A.project(x if batch > 1 else x[0]).reshape((batch,) + A.output_shape)
    for k in {0, batch // 2, batch - 1} if batch > 1 else ():
        assert torch.equal(got[k], A.project(x[k].contiguous()))
    few = sorted({0, nv // 2, nv - 2, nv - 1} - {-1})
    B = linop.XRayTransform2D(shape, ang[few])
    assert torch.equal(got[-1][few], B.project(x[-1].contiguous()))
