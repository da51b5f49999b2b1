"""The float64 dot products (ct_dot) against exact sums, at sizes and scales where their float32 splitting changes
form: sizes with and without whole quads, products below and above the range it covers, cancelling sums, zeros.

A float64 product of two float32 values is exact and math.fsum is exactly rounded, so the reference has no error of
its own.  Bound: at most 32 float64 roundings lie between a product and the total at these sizes (7 of a thread's
four groups, 8 + 5 of the block, 2 + 8 + 5 of the grid and its last rounding), 32 x 2^-53 = 2^-48 of sum |a b|; the splitting adds
less than 2^-60."""

import math

import numpy as np
import pytest
import torch

from scico_gb300 import _device, _lib

pytestmark = pytest.mark.gpu


def _dot(a, b):
    a, b = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    out = torch.empty(1, dtype=torch.float64, device="cuda")
    ws = torch.zeros(256 + 8 * 4 * 304, dtype=torch.uint8, device="cuda")
    _lib.call("ct_dot", a.data_ptr(), b.data_ptr(), a.numel(), out.data_ptr(), ws.data_ptr(), ws.numel(),
              _device.stream())
    return out.item()


@pytest.mark.parametrize("n", [1, 4, 7, 64, 4096, 262144, 311300, 1 << 20])
@pytest.mark.parametrize("kind", ["plain", "square", "wide", "tiny", "huge", "cancel", "holes"])
def test_dot_against_exact_sum(cuda, n, kind):
    rng = np.random.default_rng(n)
    a, b = (rng.standard_normal(n).astype(np.float32) for _ in range(2))
    if kind == "square":
        b = a
    elif kind == "wide":
        a = (a * np.exp(rng.uniform(-60, 60, n))).astype(np.float32)
    elif kind == "tiny":  # products down to 2^-240, where a float32 product is zero
        a, b = a * np.float32(2.0 ** -110), b * np.float32(2.0 ** -110)
        b[: n // 2] *= np.float32(2.0 ** 60)
    elif kind == "huge":  # products up to 2^240, where a float32 product is infinite
        a, b = a * np.float32(2.0 ** 120), b * np.float32(2.0 ** 110)
        b[: n // 2] *= np.float32(2.0 ** -115)
    elif kind == "cancel" and n > 1:
        h = n // 2
        a[h: 2 * h], b[h: 2 * h] = a[:h], -b[:h]
    elif kind == "holes":
        a[rng.random(n) < 0.7] = 0.0
    p = a.astype(np.float64) * b.astype(np.float64)
    assert abs(_dot(a, b) - math.fsum(p)) <= 2.0 ** -48 * math.fsum(np.abs(p))


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_dot_passes_non_finite_on(cuda, bad):
    a, b = np.zeros(4096, np.float32), np.ones(4096, np.float32)
    a[5] = bad
    assert not math.isfinite(_dot(a, b))
    b[5] = 0.0
    assert math.isnan(_dot(a, b)) and math.isnan(_dot(b, a))
