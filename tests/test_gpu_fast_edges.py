"""An edge of the fast step has one solution: what the cell below it gets and
what the cell above it gets come from one evaluation, wherever the edge lies in
a thread's pair of rows and whatever the other cells of its warp hold.  (A warp
has 64 rows.  Its lowest edge alone is solved twice, by it and by the warp
below.)  Wide domains, so that a CTA has columns inside its segment; no
tolerance."""
import numpy as np
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu

WARP_ROWS = 64


def step(swe, solver, nx, ny, fields):
    """one step of one block inside walls; interior h, hu, hv as (nx, ny)"""
    D = swe.Domain([nx], [ny], 100.0, 100.0, boundary=[1] * 4, solver=solver, arithmetic=swe.FAST)
    D.upload(*[np.ascontiguousarray(f, dtype=np.float32).ravel() for f in fields])
    D.exchange_bathymetry()
    D.step(1)
    out = [a.reshape(nx + 2, ny + 2)[1:-1, 1:-1] for a in D.download()[:3]]
    assert D.status() == 0
    D.close()
    return out


def water(nx, ny, seed):
    """shallow choppy water, wet and subcritical, that a step moves by a good part
    of its depth; one deep cell sets the time step"""
    r = np.random.default_rng(seed)
    h = r.uniform(1, 3, (nx + 2, ny + 2))
    h[3, 150] = 8.0
    return [h, h * r.uniform(-0.5, 0.5, h.shape), h * r.uniform(-0.5, 0.5, h.shape), r.uniform(-0.1, 0.1, h.shape)]


@pytest.mark.parametrize("nx,ny", [(8000, 256), (301, 300), (3000, 1024)])
def test_rows_do_not_depend_on_their_place_in_a_thread(swe, nx, ny):
    """the same rows one place further down: bits as before, except in the lowest
    row of a warp (f-wave; HLLE's bound from the cell above a pair is rounded
    once less than from a cell inside it)"""
    f = water(nx, ny + 1, nx + ny)
    low = step(swe, 1, nx, ny, [a[:, :ny + 2] for a in f])
    high = step(swe, 1, nx, ny, [a[:, 1:] for a in f])
    y = np.arange(3, ny)  # rows of the first that are not on the rim in either
    y = y[((y - 1) % WARP_ROWS != 0) & ((y - 2) % WARP_ROWS != 0)]
    for a, b, name in zip(low, high, ("h", "hu", "hv")):
        assert_bitwise(a[:, y - 1], b[:, y - 2], name)


@pytest.mark.parametrize("solver", [1, 4])
@pytest.mark.parametrize("kind", ["dry", "supercritical"])
def test_rows_do_not_depend_on_other_cells_of_their_warp(swe, solver, kind):
    """a row of cells whose edges their threads solve again leaves the other
    threads' rows as they are"""
    nx, ny, row = 8000, 200, 100
    a = water(nx, ny, 5)
    b = [f.copy() for f in a]
    if kind == "dry":
        for f in b[:3]:
            f[:, row] = 0.0
    else:
        b[0][:, row] = 0.2
        b[1][:, row] = b[2][:, row] = 0.2 * 3.0
    away = np.abs(np.arange(1, ny + 1) - row) > 3
    for f, g, name in zip(step(swe, solver, nx, ny, a), step(swe, solver, nx, ny, b), ("h", "hu", "hv")):
        assert (f != g).any()
        assert_bitwise(f[:, away], g[:, away], name)
