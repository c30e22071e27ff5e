"""The update pass in CTAs of four teams that keep pace (domains whose partition
gives every SM four 256-row runs) against the pass in CTAs of one (another
segment length), bit for bit: runs of unequal length, blocks that end inside a
run, groups that have stopped, and local time stepping's changing lists."""
import numpy as np
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu


def waves(swe, nx, ny, nb, seed):
    geo, h, hu, hv, b = swe.init_domain(swe.SCENARIO_DAM_BREAK, nx, ny, nb, [1000.0, 200.0, 12.0, 6.0, 0.0])
    r = np.random.default_rng(seed)
    h = (h + r.uniform(0, 1, h.shape)).astype(np.float32)
    return geo, (h, (h * r.uniform(-1, 1, h.shape)).astype(np.float32), (h * r.uniform(-1, 1, h.shape)).astype(np.float32),
                 r.uniform(-1, 1, b.shape).astype(np.float32))


def same(make, st, drive, rows=None):
    out = []
    for cols in (0, 128):
        D = make(cols)
        if rows and not cols:
            D.retile(rows, 0)
        D.upload(*st)
        D.exchange_bathymetry()
        drive(D)
        out.append(D.download() + D.group_state())
        assert D.status() == 0
        D.close()
    for a, r, k in zip(*out, ("h", "hu", "hv", "b", "time", "dt", "steps")):
        assert_bitwise(a, r, k)


# from just above the sizes that run several steps per launch to several segments per team
@pytest.mark.parametrize("solver", [1, 4])
@pytest.mark.parametrize("nx,ny,nb", [(2500, 256, 1), (1100, 769, 1), (1300, 1280, 4), (2048, 2048, 16), (9000, 1024, 1)])
def test_teams_equal_single(swe, solver, nx, ny, nb):
    geo, st = waves(swe, nx, ny, nb, nx)
    same(lambda c: swe.Domain(geo["nx_cols"], geo["ny_rows"], geo["dx"], geo["dy"], boundary=[0, 1, 1, 0], solver=solver,
                              tile_cols=c, tile_rows=256), st, lambda D: D.step(4))


def test_teams_with_stopped_groups(swe):
    sizes = [(700, 256), (900, 512), (650, 256), (800, 1024)]
    inst, st = [], [[], [], [], []]
    for i, (nx, ny) in enumerate(sizes):
        geo, f = waves(swe, nx, ny, 1, i)
        inst.append((nx, ny, 2.0 + 3.0 * i, 5.0, [1, 0, 0, 1]))
        for a, v in zip(st, f):
            a.append(v)
    st = [np.concatenate(a) for a in st]
    same(lambda c: swe.Ensemble(inst, solver=4, tile_cols=c, tile_rows=256), st, lambda D: D.advance(0.6), rows=256)


def test_teams_local_time_stepping(swe):
    geo, st = waves(swe, 2048, 1024, 8, 2)
    n = len(geo["nx_cols"]) * len(geo["ny_rows"])
    dx = geo["dx"] * 20

    def make(c):
        return swe.Domain(geo["nx_cols"], geo["ny_rows"], dx, dx, boundary=[1] * 4, solver=4, tile_cols=c, tile_rows=256,
                          lts_max_timestep=1.0, duration=100.0)

    out = []
    for cols in (0, 128):
        D = make(cols)
        D.upload(*st)
        D.exchange_bathymetry()
        D.lts_advance(1.5)
        out.append(D.download() + (D.lts_state()[3],))
        assert D.status() == 0 and len(out[-1][4]) == n
        D.close()
    for a, r, k in zip(*out, ("h", "hu", "hv", "b", "steps")):
        assert_bitwise(a, r, k)
