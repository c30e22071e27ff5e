"""The ghost ring that the exact update pass pushes from a block's rim cells
(outflow, walls, kept ghosts, neighbour blocks, corners) against the ring that
setGhostLayer forms from the same cells, bit for bit: both step semantics, one
row, one column, tiles of the four-team kernel and of the plain one."""
import numpy as np
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu

OUT, WALL, INFLOW, CONNECT, PASSIVE = 0, 1, 2, 3, 5


@pytest.mark.parametrize("speed_pass", [0, 1])  # small domains: their own kernel, and the two passes
@pytest.mark.parametrize("semantics,nx_cols,ny_rows", [
    (0, [1], [1]), (0, [5], [1]), (0, [1], [70]), (0, [40], [259]), (0, [33, 20], [64, 31]), (0, [700, 520], [256, 512]),
    (1, [1], [1]), (1, [1], [70]), (1, [40], [259]),
])
@pytest.mark.parametrize("solver", ["HLLE", "HYBRID"])
@pytest.mark.parametrize("boundary", [[OUT, WALL, WALL, OUT], [WALL, OUT, PASSIVE, WALL], [INFLOW, WALL, OUT, CONNECT]])
def test_pushed_ring_equals_recomputed_ring(swe, solver, semantics, nx_cols, ny_rows, boundary, speed_pass):
    n = sum((x + 2) * (y + 2) for x in nx_cols for y in ny_rows)
    r = np.random.default_rng(n)
    st = [10 + r.random(n), r.random(n) - 0.5, r.random(n) - 0.5, -10 + 0.1 * r.random(n)]
    st = [a.astype(np.float32) for a in st]

    def make(state):
        D = swe.Domain(nx_cols, ny_rows, 10.0, 12.0, boundary=boundary, solver=getattr(swe, solver), semantics=semantics,
                       speed_pass=speed_pass)
        D.upload(*state)
        return D

    D = make(st)
    D.exchange_bathymetry()
    st[3] = D.download()[3]
    D.step(2)
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
