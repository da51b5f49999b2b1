"""Scratch that the 3D projector's query reports for general geometries (host
code; the view table is not read): bounded by the volume's own size or a
gigabyte for a view's tiles, and none where the tiles would outgrow that."""

import ctypes

import pytest

from scico_gb300 import _lib


def _query(shape, views):
    g = _lib.Geom3D()
    g.shape[:] = list(shape)
    g.det_shape[:] = [64, 64]
    g.n_views = views
    g.kind = _lib.CT_PROJ3D_GENERAL
    g.views = 256  # never dereferenced by the query
    fwd, adj = _lib.c_size_t(), _lib.c_size_t()
    assert _lib.load().ct_proj3d_workspace(ctypes.addressof(g), 1, ctypes.addressof(fwd),
                                           ctypes.addressof(adj)) == _lib.CT_OK
    return fwd.value


@pytest.mark.parametrize("shape", [(1, 20000, 20000), (20000, 1, 20000), (12000, 12000, 1), (1, 1, 500_000_000)])
def test_no_windows_where_tiles_would_outgrow_the_volume(ctlib, shape):
    assert _query(shape, 60) == 0


@pytest.mark.parametrize("shape", [(16, 16, 16), (97, 128, 111), (256, 256, 256), (1024, 1024, 1024), (8, 4096, 4096),
                                   (1, 6000, 6000), (3000, 7, 3000)])
@pytest.mark.parametrize("views", [1, 60, 2000])
def test_scratch_is_bounded(ctlib, shape, views):
    volume = 4 * shape[0] * shape[1] * shape[2]
    fwd = _query(shape, views)
    assert volume < fwd <= volume + max(volume, 1 << 30) + 512 * views + 4096
