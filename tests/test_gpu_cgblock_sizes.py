"""The element passes of inverse.cg_block at the sizes where they change form: images whose size is and is not a
multiple of four, several groups a thread, arrays off a 16-byte boundary, many view splits, no step at all, and
vectors so small or so large that a dot product leaves the range of its float32 splitting.

Values agree with the autograd recurrence to 1e-5, gradients to 1e-4 (the well-conditioned setting of the block's
other tests: lam comparable to the operator's scale, three steps).  Scaling b, z by a power of two scales every
float32 vector exactly and leaves the step sizes alone, so results then agree to the float64 sums' rounding as it
shows in a float32 step size: 1e-6."""

import numpy as np
import pytest
import torch

from scico_gb300 import inverse, linop

pytestmark = pytest.mark.gpu


def _op(shape, nv):
    return (1.0 / max(shape)) * linop.XRayTransform2D(shape, np.linspace(0, np.pi, nv, endpoint=False))


def _run(H, b, x0, w, lam_val, iters, native=True):
    b = b.detach().requires_grad_()
    x0 = x0.detach().requires_grad_()
    lam = torch.full((1,), lam_val, device=b.device, requires_grad=True)
    if native:
        x = inverse.cg_block(H, b, lam, x0=x0, maxiter=iters)
    else:
        x = inverse.cg_solver(lambda v: inverse.back_project(H, inverse.project(H, v)) + lam * v, b, x0=x0,
                              maxiter=iters, batch_dims=1)
    return (x.detach(), *torch.autograd.grad((w * x).sum(), (b, x0, lam)))


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize("shape,batch,nv", [((5, 5), 2, 9), ((17, 19), 3, 24), ((64, 64), 1, 45), ((90, 70), 4, 30),
                                            ((181, 183), 1, 40), ((400, 404), 1, 30), ((32, 32), 40, 12)])
@pytest.mark.parametrize("shift", [0, 1])
def test_cg_block_sizes(cuda, shape, batch, nv, shift):
    H, g = _op(shape, nv), torch.Generator().manual_seed(5)
    n = batch * shape[0] * shape[1]
    b, x0, w = ((torch.randn(n + 1, generator=g).to(cuda))[shift: shift + n].view(batch, *shape) for _ in range(3))
    x, gb, gx0, gl = _run(H, b, x0, w, float(nv), 3)
    xr, gbr, gx0r, glr = _run(H, b, x0, w, float(nv), 3, native=False)
    assert _rel(x, xr) < 1e-5
    assert _rel(gb, gbr) < 1e-4
    # lam's gradient is a sum over all pixels that nearly cancels: measured by its terms, |gb| |x|
    assert float((gl - glr).abs() / (gb.norm() * x.norm())) < 1e-4
    # what is left of x0's influence after three steps is small against the gradient it starts from
    assert float((gx0 - gx0r).norm() / w.norm()) < 1e-4


def test_cg_block_no_step(cuda):
    H, g = _op((24, 20), 15), torch.Generator().manual_seed(6)
    b, x0, w = (torch.randn((2, 24, 20), generator=g).to(cuda) for _ in range(3))
    x, gb, gx0, _ = _run(H, b, x0, w, 2.0, 0)
    assert torch.equal(x, x0) and torch.equal(gx0, w) and not gb.any()


@pytest.mark.parametrize("power", [-70, -45, 45])
def test_cg_block_scale(cuda, power):
    H, g = _op((48, 52), 40), torch.Generator().manual_seed(7)
    b, x0, w = (torch.randn((2, 48, 52), generator=g).to(cuda) for _ in range(3))
    c = 2.0 ** power
    x, gb, gx0, gl = _run(H, b, x0, w, 40.0, 3)
    xs, gbs, gx0s, gls = _run(H, b * c, x0 * c, w, 40.0, 3)
    assert _rel(xs / c, x) < 1e-6
    assert _rel(gbs, gb) < 1e-6
    assert _rel(gls / c, gl) < 1e-6
    assert float((gx0s - gx0).norm() / w.norm()) < 1e-6


def test_cg_block_gradient_over_its_input(cuda):
    """ct_cg_block_bwd with a gradient written over gx: the bits of separate arrays."""
    import ctypes

    from scico_gb300 import _device, _lib

    A = linop.XRayTransform2D((40, 36), np.linspace(0, np.pi, 20, endpoint=False))
    gen = torch.Generator().manual_seed(8)
    b, x0, w = (torch.randn((2, 40, 36), generator=gen).to(cuda) for _ in range(3))
    d = _lib.CgBlockDesc(A.geometry(), 2, 3, 0, 1.0 / 1600.0)
    tb, wb = _lib.c_size_t(), _lib.c_size_t()
    at = ctypes.addressof
    _lib.call("ct_cg_block_workspace", at(d), at(tb), at(wb))
    tape, ws = _device.workspace(tb.value), _device.workspace(wb.value)
    x = torch.empty_like(b)
    st = _device.stream()
    _lib.call("ct_cg_block_fwd", at(d), b.data_ptr(), 20.0, x0.data_ptr(), x.data_ptr(), tape.data_ptr(),
              tape.numel(), ws.data_ptr(), ws.numel(), st)

    def grads(gx, gb, gx0):
        gl = torch.zeros(1, dtype=torch.float64, device=cuda)
        _lib.call("ct_cg_block_bwd", at(d), gx.data_ptr(), b.data_ptr(), 20.0, x0.data_ptr(), tape.data_ptr(),
                  tape.numel(), gb.data_ptr(), gx0.data_ptr(), gl.data_ptr(), ws.data_ptr(), ws.numel(), st)
        return gb, gx0, gl

    want = grads(w, torch.empty_like(w), torch.empty_like(w))
    for over in (0, 1):
        g = w.clone()
        got = grads(g, g if over == 0 else torch.empty_like(w), g if over == 1 else torch.empty_like(w))
        assert all(torch.equal(a, c) for a, c in zip(got, want))
