"""The ghost ring that the fast-arithmetic step pushes from a block's rim cells
(outflow, walls, kept ghosts, neighbour blocks, corners) against the ring that
setGhostLayer forms from the same cells, bit for bit: one-cell, one-row and
one-column blocks, blocks of several tiles, every boundary type on every side."""
import numpy as np
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu

OUT, WALL, INFLOW, CONNECT, PASSIVE = 0, 1, 2, 3, 5


@pytest.mark.parametrize("solver", ["HLLE", "FWAVE"])
@pytest.mark.parametrize("nx_cols,ny_rows", [([1], [1]), ([5], [1]), ([1], [70]), ([40], [259]), ([33, 20], [64, 31]),
                                             ([1, 2], [3, 1])])
@pytest.mark.parametrize("boundary", [[OUT, WALL, WALL, OUT], [WALL, OUT, PASSIVE, WALL], [INFLOW, WALL, OUT, CONNECT],
                                      [OUT, PASSIVE, WALL, WALL]])
def test_pushed_ring_equals_recomputed_ring(swe, solver, nx_cols, ny_rows, boundary):
    n = sum((x + 2) * (y + 2) for x in nx_cols for y in ny_rows)
    r = np.random.default_rng(n)
    st = [10 + r.random(n), r.random(n) - 0.5, r.random(n) - 0.5, -10 + 0.1 * r.random(n)]
    st = [a.astype(np.float32) for a in st]

    def make(state):
        D = swe.Domain(nx_cols, ny_rows, 10.0, 12.0, boundary=boundary, solver=getattr(swe, solver), arithmetic=swe.FAST)
        D.upload(*state)
        return D

    D = make(st)
    D.exchange_bathymetry()
    st[3] = D.download()[3]
    D.step(3)
    D.set_ghost_layer()
    pushed = D.download()
    assert D.status() == 0
    D.close()
    E = make(pushed)
    E.set_ghost_layer()
    ref = E.download()
    E.close()
    for a, b, k in zip(pushed, ref, "h hu hv b".split()):
        assert_bitwise(a, b, k)
