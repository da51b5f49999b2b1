"""The ramp filter's row kernel at the lengths where its blocks of eight taps
and eight outputs end unevenly, and the masked back projection, against the
oracle.

Tolerance of the rows: each output is a sum of at most n/2 + 1 products of
float32 numbers accumulated in float32; with unit-variance data the rounding
of the running sum is below n/2 half-ulps of the largest partial sum, so
rel l2 <= n/4 * 2^-24 + 2^-23 (taps and products), at least 4e-7.
"""

import numpy as np
import pytest
import torch

from oracle import ctref
from scico_gb300 import _lib, linop

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("det", [1, 2, 3, 4, 15, 16, 17, 18, 31, 32, 33, 34, 35, 63, 257, 1001, 1090, 4099, 20600])
def test_ramp_rows_lengths(cuda, det):
    rows = 3
    y = np.random.default_rng(det).standard_normal((rows, det)).astype(np.float32)
    out = torch.full((rows + 1, det), 7.0, device=cuda)
    _lib.call("ct_fbp_filter", torch.from_numpy(y).to(cuda).data_ptr(), out.data_ptr(), rows, det,
              torch.cuda.current_stream().cuda_stream)
    got = out.cpu().numpy()
    assert np.all(got[rows] == 7.0)  # nothing past the last row
    n, off = np.arange(-(det - 1), det), (det - 1) // 2
    h = np.where(n == 0, 0.25, np.where(n % 2 != 0, -1.0 / (np.pi * np.where(n == 0, 1, n)) ** 2, 0.0))
    h[(n < -off) | (n > det - 1 - off)] = 0.0
    if det <= 4099:
        want = np.stack([np.convolve(r.astype(np.float64), h)[det - 1:2 * det - 1] for r in y])
    else:
        m = 4 * det
        F = np.fft.rfft(h, m) * np.fft.rfft(y.astype(np.float64), m)
        want = np.fft.irfft(F, m)[:, det - 1:2 * det - 1]
    assert ctref.rel_l2(got[:rows], want) <= max(4e-7, det / 4 * 2.0**-24 + 2.0**-23)


def test_ramp_rows_reach(cuda):
    """An infinite sample reaches the outputs within its taps and no others."""
    det = 61
    y = torch.zeros((1, det), device=cuda)
    y[0, 40] = float("inf")
    out = torch.empty_like(y)
    _lib.call("ct_fbp_filter", y.data_ptr(), out.data_ptr(), 1, det, torch.cuda.current_stream().cuda_stream)
    i = np.arange(det)
    d = np.abs(i - 40)
    hit = (d == 0) | ((d % 2 == 1) & (d <= (det - 1) // 2))
    np.testing.assert_array_equal(~np.isfinite(out.cpu().numpy()[0]), hit)


@pytest.mark.parametrize("n,nv,det", [(48, 90, 40), (700, 8, 991)])
def test_masked_back_projection(cuda, n, nv, det):
    """One pass = mask times scale times the back projection, bit for bit
    (several view splits, and one with a detector that cuts corners)."""
    A = linop.XRayTransform2D((n, n), np.linspace(0, np.pi, nv, endpoint=False), det_count=det)
    y = torch.rand((2,) + A.output_shape, generator=torch.Generator().manual_seed(1)).to(cuda)
    got = A.fbp(y)
    assert A.fbp_mask.dtype == torch.bool
    A.fbp_mask = A.fbp_mask.to(torch.uint8)  # a caller's own mask: composed expression
    assert torch.equal(got, A.fbp(y))
