"""The regulariser kernels around the size up to which a thread takes one
element (eight blocks of 256 an SM) and past which it takes four: the oracle's
bits on either side.  Small arrays take no longer than their one launch: the
L2,1 prox of 3 x 12288 against the L1 prox of the same array (2.1 and 1.5 us; 3.1
with four vectors a thread)."""

import numpy as np
import pytest
import torch

from oracle import ctref
from scico_gb300 import functional, linop

pytestmark = pytest.mark.gpu


def _edge():
    return torch.cuda.get_device_properties(0).multi_processor_count * 8 * 256


@pytest.mark.parametrize("ncomp", [1, 2, 3])
@pytest.mark.parametrize("past", [0, 1, 1023])
def test_l21_prox_around_the_edge(cuda, ncomp, past):
    n = _edge() + past
    v = np.random.default_rng(n).standard_normal((ncomp, n)).astype(np.float32)
    got = functional.L21Norm().prox(torch.from_numpy(v).to(cuda), 0.7).cpu().numpy()
    np.testing.assert_array_equal(got, ctref.l21_prox(v, np.float32(0.7)))


@pytest.mark.parametrize("kw", [dict(append=0), dict(prepend=1), dict(circular=True)], ids=str)
@pytest.mark.parametrize("rows", [-1, 1])
def test_short_rows_around_the_edge(cuda, kw, rows):
    shape = (10, _edge() // 310 + rows, 31)  # rows too short for a warp and no whole number of quads
    rng = np.random.default_rng(3)
    D = linop.FiniteDifference(shape, **kw)
    x = rng.standard_normal((1,) + shape).astype(np.float32)
    d = rng.standard_normal((1, 3) + shape).astype(np.float32)
    y = D._eval(torch.from_numpy(x).to(cuda)).cpu().numpy()[0]
    np.testing.assert_array_equal(y, np.stack([ctref.fd_eval(x[0], axes=(a,), **kw)[0] for a in range(3)]))
    back = D._adj(torch.from_numpy(d).to(cuda)).cpu().numpy()[0]
    np.testing.assert_array_equal(back, ctref.fd_adj(d[0], shape, axes=(0, 1, 2), **kw))


def _us(fn):
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(50):
            fn()
    best = float("inf")
    for _ in range(8):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        graph.replay()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 20.0)
    return best


def test_small_prox_is_one_short_launch(cuda):
    v = torch.randn((3, 64, 64, 3), device=cuda)
    l21, l1 = functional.L21Norm(), functional.L1Norm()
    assert _us(lambda: l21.prox(v, 0.05)) <= 1.75 * _us(lambda: l1.prox(v, 0.05))
