"""The one-pass regulariser kernels against the oracle at the sizes where they
can go wrong: blocks that end inside a row, sides of one, odd sides, axis
subsets and orders, batches, and infinities.

Same-shape finite differences, their adjoint and the L2,1 prox perform the
oracle's float32 operations in its order: equal bits.  The one-pass TV prox
equals the composition of ct_haar_fwd, the norm's prox and ct_haar_adj bit for
bit (a base norm of another type takes that composition).
"""

import numpy as np
import pytest
import torch

from oracle import ctref
from scico_gb300 import functional, linop

pytestmark = pytest.mark.gpu

MODES = [dict(append=0), dict(append=1), dict(prepend=0), dict(prepend=1), dict(circular=True)]
SHAPES = [((1023,), None), ((1025,), None), ((1, 7), None), ((33, 31), (1, 0)), ((7, 1, 151), None),
          ((5, 37, 29), (2, 0)), ((16, 64, 4), (0, 1, 2)), ((5, 37, 29), (1,)),
          ((1024,), None), ((12, 40), (1, 0)), ((3, 5, 260), None), ((6, 9, 8), (2, 0)), ((1, 3, 4), None)]  # whole quads


@pytest.mark.parametrize("kw", MODES, ids=str)
@pytest.mark.parametrize("shape,axes", SHAPES, ids=str)
def test_same_shape_differences(cuda, shape, axes, kw):
    rng = np.random.default_rng(sum(shape))
    x = rng.standard_normal((2,) + shape).astype(np.float32)
    x.reshape(2, -1)[0, -1] = np.inf
    ax = tuple(range(len(shape))) if axes is None else axes
    D = linop.FiniteDifference(shape, axes=axes, **kw)
    y = D._eval(torch.from_numpy(x).to(cuda)).cpu().numpy()
    d = rng.standard_normal((2, len(ax)) + shape).astype(np.float32)
    back = D._adj(torch.from_numpy(d).to(cuda)).cpu().numpy()
    for b in range(2):
        with np.errstate(invalid="ignore"):
            ref = [ctref.fd_eval(x[b], axes=(a,), **kw)[0] for a in ax]
        np.testing.assert_array_equal(y[b], np.stack(ref))
        want = ctref.fd_adj(d[b], shape, axes=ax, **kw)
        np.testing.assert_array_equal(back[b], want)


@pytest.mark.parametrize("kw", MODES, ids=str)
@pytest.mark.parametrize("shape", [(6, 40), (3, 5, 64)], ids=str)
def test_differences_off_a_quad_boundary(cuda, shape, kw):
    """Arrays that start off a 16-byte boundary: the bits of aligned ones."""
    D, n = linop.FiniteDifference(shape, **kw), int(np.prod(shape))
    v = torch.from_numpy(np.random.default_rng(n).standard_normal((1 + len(shape)) * n).astype(np.float32)).to(cuda)
    x, d = v[:n].clone().view((1,) + shape), v[n:].clone().view((1, len(shape)) + shape)
    xs, ds = (torch.empty(t.numel() + 1, device=cuda)[1:].view(t.shape).copy_(t) for t in (x, d))
    assert xs.is_contiguous() and xs.data_ptr() % 16
    assert torch.equal(D._eval(xs), D._eval(x)) and torch.equal(D._adj(ds), D._adj(d))


@pytest.mark.parametrize("ncomp", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 255, 1024, 1025, 5001])
def test_l21_prox_sizes(cuda, ncomp, n):
    v = np.random.default_rng(n).standard_normal((ncomp, n)).astype(np.float32)
    v[:, 0] = 0.0
    got = functional.L21Norm().prox(torch.from_numpy(v).to(cuda), 0.7).cpu().numpy()
    np.testing.assert_array_equal(got, ctref.l21_prox(v, np.float32(0.7)))


class _L21(functional.L21Norm):
    """A base norm of another type: the TV prox takes the composed path."""


class _L1(functional.L1Norm):
    pass


@pytest.mark.parametrize("iso", [True, False])
@pytest.mark.parametrize("circular", [True, False])
@pytest.mark.parametrize("shape,axes", SHAPES + [((1,), None), ((2, 3, 2), (1, 2))], ids=str)
def test_tv_prox_one_pass(cuda, iso, circular, shape, axes):
    v = torch.from_numpy(np.random.default_rng(3).standard_normal(shape).astype(np.float32)).to(cuda)
    v.view(-1)[0] = float("inf")
    one = (functional.IsotropicTVNorm if iso else functional.AnisotropicTVNorm)(circular=circular, axes=axes)
    two = functional.TVNorm(_L21() if iso else _L1(), circular=circular, axes=axes)
    np.testing.assert_array_equal(one.prox(v, 0.05).cpu().numpy(), two.prox(v, 0.05).cpu().numpy())
    t = torch.empty((3,) + shape, device=cuda).transpose(0, -1)  # not contiguous
    t.copy_(torch.randn(t.shape, generator=torch.Generator().manual_seed(1)).to(cuda))
    if t.ndim <= 3:
        np.testing.assert_array_equal(one.prox(t, 0.05).cpu().numpy(), two.prox(t, 0.05).cpu().numpy())
