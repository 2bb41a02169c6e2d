"""Gridding through tiles: supports on both sides of its range, grids that are
not multiples of a tile, empty channels, visibilities beyond the edges and
kernel tables smaller than the support, bit for bit against the restatement of
do_gridding."""

import numpy as np
import pytest

import grid_oracle as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("table_shape,support", [((3, 3), (1, 1)), ((7, 7), (3, 3)), ((9, 9), (4, 4)),
                                                 ((5, 3), (2, 1)), ((5, 5), (3, 4)),
                                                 ((11, 11), (5, 5)), ((1, 1), (0, 0)),
                                                 ((3, 1), (1, 0))])
@pytest.mark.parametrize("M,N", [(64, 64), (37, 51), (8, 16)])
def test_tiles(table_shape, support, M, N):
    import gpuvmem_gb300 as gv
    rng = np.random.default_rng([M, N, *support])
    counts = (700, 0, 1, 333)
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    V, cell = int(off[-1]), 0.05 / 3600.0
    freqs = np.linspace(220e9, 240e9, len(counts)).astype(np.float32)
    uvw = rng.normal(0, 0.25 * 1.3e-3 / (cell * np.pi / 180.0), (V, 3))  # some beyond the edges
    uvw[::50] *= 100.0
    vo = rng.normal(0, 1, (V, 2)).astype(np.float32)
    w = rng.uniform(0.5, 2.0, V).astype(np.float32)
    w[::7] = 0.0
    w[3::31] *= -1.0
    table = rng.uniform(-0.2, 1.0, table_shape).astype(np.float32)
    goff, guvw, gvo, gw = gv.grid_visibilities(table, support, M, N, -cell, cell, freqs, off, uvw,
                                               vo, w)
    for c in range(len(counts)):
        o, e, a, b = off[c], off[c + 1], goff[c], goff[c + 1]
        ruvw, rvo, rw = G.grid_channel(table, support, uvw[o:e], vo[o:e], w[o:e], freqs[c], M, N,
                                       -cell, cell)
        np.testing.assert_array_equal(guvw[a:b], ruvw)
        np.testing.assert_array_equal(gw[a:b].view(np.uint32), rw.view(np.uint32))
        np.testing.assert_array_equal(np.ascontiguousarray(gvo[a:b]).view(np.uint32).ravel(),
                                      np.ascontiguousarray(rvo).view(np.uint32).ravel())
