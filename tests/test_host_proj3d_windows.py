"""Which views the GENERAL 3D forward's windows take (ct_proj3d_window_views, the
test that the device makes): every voxel of a view that they take writes inside
its window's tile, and every pixel finds the windows that cover it.  The
positions, shifts, tiles and the gather's window index are evaluated here in
float32 as the kernels do, for nearly parallel matrix rows (accepted down to a
sine of 1e-6, where the shear per plane has few digits left) and for rotations."""

import ctypes

import numpy as np
import pytest

from scico_gb300 import _lib, linop

X3 = linop.XRayTransform3D
F = np.float32
WIN, SLACK = 16, F(0.0625)

# Nearly parallel rows: row sines 1.6e-6 and 3.1e-5.
PARALLEL = [
    ((97, 128, 111), [[1.1872672e-01, 1.5680777e-01, -1.2382731e-01, 5.1078472e01],
                      [2.5399225, 3.3546038, -2.6490467, -1.3085880e02]]),
    ((256, 256, 256), [[-2.04851621, 1.18603859, 1.69305127, 128.0],
                       [-0.26546947, 0.15369791, 0.21938796, 128.0]]),
]


def taken(shape, M):
    """(view table, windows' choice per view) of a GENERAL geometry."""
    M = np.ascontiguousarray(M, dtype=F)
    views = np.zeros((len(M), _lib.CT_VIEW3D_STRIDE), F)
    n = np.asarray(shape, np.int32)
    kind, off = ctypes.c_int32(), ctypes.c_int32()
    lib = _lib.load()
    assert lib.ct_proj3d_views(M.ctypes.data, len(M), n.ctypes.data, np.array([64, 64], np.int32).ctypes.data,
                               views.ctypes.data, None, ctypes.addressof(kind), ctypes.addressof(off)) == _lib.CT_OK
    out = np.full(len(M), -1, np.int32)
    assert lib.ct_proj3d_window_views(views.ctypes.data, len(M), n.ctypes.data, out.ctypes.data) == _lib.CT_OK
    return views, out


def worst(m, shape):
    """Of one view by windows: the furthest that a voxel's slot lies outside its
    tile, and the furthest that a window lies outside a pixel's candidates."""
    ax = int(m[8])
    p, q = (1 if ax == 0 else 0), (1 if ax == 2 else 2)
    na, n_p, n_q = shape[ax], shape[p], shape[q]
    ma, mp, mq, c = ([m[r * 4 + k] for r in (0, 1)] for k in (ax, p, q, 3))
    det = F(mp[0] * mq[1]) - F(mq[0] * mp[1])
    d = [-F(F(mq[1] * ma[0]) - F(mq[0] * ma[1])) / det, -F(F(mp[0] * ma[1]) - F(mp[1] * ma[0])) / det]
    w = F(1.0 / WIN)
    inv = [[F(w * mq[1]) / det, -F(w * mq[0]) / det], [-F(w * mp[1]) / det, F(w * mp[0]) / det]]
    fw = F(WIN)
    T = [int(np.ceil(fw * abs(mp[r]) + fw * abs(mq[r]) + 2 * SLACK)) + 1 for r in (0, 1)]
    base = [((c[r] + F(0.5) * ma[r]) + (F(-0.25) - SLACK)) + (fw * min(mp[r], F(0)) + fw * min(mq[r], F(0)))
            for r in (0, 1)]
    xp, xq = (np.arange(n, dtype=F) + F(0.5) for n in (n_p, n_q))
    prod_p, prod_q = [mp[r] * xp for r in (0, 1)], [mq[r] * xq for r in (0, 1)]
    out, far = 0, 0.0
    for ia in range(na):
        s = [int(np.floor(F(d[k] * F(ia)) + F(0.5))) for k in (0, 1)]
        I, J = np.floor_divide(np.arange(n_p) - s[0], WIN), np.floor_divide(np.arange(n_q) - s[1], WIN)
        u, lo = [], []
        for r in (0, 1):
            a = ma[r] * (F(ia) + F(0.5))
            if ax == 2:
                px = (prod_p[r][:, None] + prod_q[r][None, :]) + a
            else:
                px = (a + prod_p[r])[:, None] + prod_q[r][None, :]
            u.append(np.floor((px + c[r]) - F(0.25)))
            b = base[r] + (mp[r] * (fw * I.astype(F))[:, None] + mq[r] * (fw * J.astype(F))[None, :])
            lo.append(u[r] - np.floor(b))
            out = max(out, int(-lo[r].min()), int(lo[r].max()) - (T[r] - 1))
        y = [u[r] - (c[r] + F(0.5) * ma[r] - F(0.25)) for r in (0, 1)]
        for k, W in ((0, I[:, None]), (1, J[None, :])):
            x = inv[k][0] * y[0] + inv[k][1] * y[1]
            margin = F(1.25) * (abs(inv[k][0]) + abs(inv[k][1])) + F(0.01)
            for step in (0, 1):  # both pixels of a footprint along both axes
                e = step * (inv[k][0] + inv[k][1])
                far = max(far, float((np.floor(x + e - margin) - W).max()), float((W - np.floor(x + e + margin)).max()))
    return out, far


@pytest.mark.parametrize("shape,m", PARALLEL)
def test_nearly_parallel_rows_take_the_march(ctlib, shape, m):
    views, how = taken(shape, [m])
    assert worst(views[0], shape)[0] > 0  # a window's tile would not hold them
    assert how[0] == 0


def _parallel(rng, count, lo, hi):
    """Matrices whose rows enclose an angle of lo..hi, one row several times the
    other (else two voxels of a step share a slot and no window takes the view)."""
    out = []
    while len(out) < count:
        a = rng.standard_normal(3)
        a /= np.linalg.norm(a)
        e = np.cross(a, rng.standard_normal(3))
        b = a + np.exp(rng.uniform(np.log(lo), np.log(hi))) * e / np.linalg.norm(e)
        rows = np.stack([a * rng.uniform(0.05, 1.0), b * rng.uniform(2.0, 5.0)])
        out.append(np.concatenate([rows[:: rng.choice([-1, 1])], rng.uniform(20, 80, (2, 1))], axis=1))
    return out


@pytest.mark.parametrize("lo,hi", [(4e-6, 1e-5), (1e-5, 1e-3), (1e-3, 1e-1)])
def test_voxels_stay_inside_their_tiles(ctlib, lo, hi):
    rng = np.random.default_rng(7)
    shape = (61, 48, 55)
    M = _parallel(rng, 40, lo, hi)
    views, how = taken(shape, M)
    for v in np.flatnonzero(how):
        slot, window = worst(views[v], shape)
        assert slot <= 0 and window <= 0, (M[v], slot, window)


@pytest.mark.parametrize("shape,vs", [((61, 48, 55), None), ((97, 128, 111), None), ((40, 45, 64), [0.7, 0.6, 0.8]),
                                      ((2000, 24, 30), None)])
def test_rotations_take_the_windows(ctlib, shape, vs):
    ang = np.random.default_rng(3).uniform(0, np.pi, (6, 3))
    M = X3.matrices_from_euler_angles(shape, (64, 64), "XYZ", ang, voxel_spacing=vs)
    views, how = taken(shape, M)
    assert np.all(how > 0)
    assert np.array_equal(how == 2, views[:, 8] == 2)
    for v in range(len(M) if np.prod(shape) < 1e6 else 2):
        slot, window = worst(views[v], shape)
        assert slot <= 0 and window <= 0


@pytest.mark.parametrize("vs,want", [([0.1, 0.1, 0.1], 0), ([3.0, 3.0, 3.0], 0)])
def test_fine_and_coarse_voxels_take_the_march(ctlib, vs, want):
    M = X3.matrices_from_euler_angles((20, 20, 20), (40, 40), "XYZ", [[0.3, 0.5, 0.2]], voxel_spacing=vs)
    assert taken((20, 20, 20), M)[1][0] == want


def test_window_views_rejects_bad_input(ctlib):
    out = np.zeros(1, np.int32)
    n = np.array([4, 4, 4], np.int32)
    t = np.zeros((1, _lib.CT_VIEW3D_STRIDE), F)
    f = ctlib.ct_proj3d_window_views
    assert f(None, 1, n.ctypes.data, out.ctypes.data) == _lib.CT_ERR_INVALID_ARG
    assert f(t.ctypes.data, 0, n.ctypes.data, out.ctypes.data) == _lib.CT_ERR_SHAPE
    t[0, 8] = 3.0
    assert f(t.ctypes.data, 1, n.ctypes.data, out.ctypes.data) == _lib.CT_ERR_INVALID_ARG
