"""Several steps per launch (small domains, swe_small.cu) against the two-pass
step (a given segment length selects it), bit for bit: every solver, segments
of 1, 2 and 4 columns, partial tiles and last segments, every boundary type,
blocks and ensembles, clocks and stopping at a time."""
import numpy as np
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu

SOLVERS = [1, 2, 3, 4]


def state(swe, nx, ny, nb, seed, dry=True):
    """random water over a random bed, dry in places, with momentum"""
    geo, h, hu, hv, b = swe.init_domain(swe.SCENARIO_DAM_BREAK, nx, ny, nb, [1000.0, 200.0, 12.0, 6.0, 0.0])
    r = np.random.default_rng(seed)
    b = (r.uniform(-2, 2, b.shape)).astype(np.float32)
    h = (h + r.uniform(-1, 1, h.shape)).astype(np.float32)
    if dry:
        h[r.random(h.shape) < 0.1] = 0.0
    wet = h > 0.2
    hu, hv = [np.where(wet, h * r.uniform(-2, 2, h.shape), 0).astype(np.float32) for _ in range(2)]
    return geo, (h, hu, hv, b)


def pair(swe, make, st, drive):
    out = []
    for cols in (0, 128):
        D = make(cols)
        D.upload(*st)
        D.exchange_bathymetry()
        D.set_ghost_layer()
        got = drive(D)
        out.append(D.download() + tuple(D.group_state()) + ((np.asarray(got, np.float32),) if got is not None else ()))
        assert D.status() == 0
        out[-1] += (np.asarray(D.launch_count()),)
        D.close()
    a, r = out
    assert a[-1] < r[-1]  # (fewer launches: the path under test ran)
    for x, y, k in zip(a[:-1], r[:-1], ("h", "hu", "hv", "b", "time", "dt", "steps", "result")):
        assert_bitwise(x, y, k)


@pytest.mark.parametrize("solver", SOLVERS)
@pytest.mark.parametrize("nx,ny,nb", [(1, 1, 1), (3, 2, 1), (33, 31, 1), (130, 257, 1), (64, 128, 4), (301, 255, 1), (97, 120, 6)])
def test_small_equals_two_pass(swe, solver, nx, ny, nb):
    geo, st = state(swe, nx, ny, nb, nx + ny)
    pair(swe, lambda c: swe.Domain(geo["nx_cols"], geo["ny_rows"], geo["dx"], geo["dy"], boundary=geo["boundary"],
                                   solver=solver, tile_cols=c), st, lambda D: D.step(7))


# segments of 2 and 4 columns (with a last one that is not full); the augmented solver has 1 only
@pytest.mark.parametrize("solver", [1, 3, 4])
@pytest.mark.parametrize("nx,ny", [(609, 200), (1215, 100), (1217, 256), (1823, 200), (1821, 256)])
def test_small_segment_widths(swe, solver, nx, ny):
    geo, st = state(swe, nx, ny, 1, nx, dry=False)
    pair(swe, lambda c: swe.Domain([nx], [ny], geo["dx"], geo["dy"], boundary=[1, 0, 1, 0], solver=solver, tile_cols=c), st,
         lambda D: D.step(5))


@pytest.mark.parametrize("boundary", [[0, 1, 2, 5], [1, 2, 0, 1], [5, 0, 1, 2], [2, 5, 5, 0]])
def test_small_boundaries(swe, boundary):
    geo, st = state(swe, 70, 90, 4, 5)
    pair(swe, lambda c: swe.Domain(geo["nx_cols"], geo["ny_rows"], geo["dx"], geo["dy"], boundary=boundary, solver=4,
                                   tile_cols=c), st, lambda D: D.step(9))


@pytest.mark.parametrize("solver", [2, 4])
def test_small_ensemble_stops_each_instance_at_its_time(swe, solver):
    sizes = [(40, 33), (65, 70), (31, 129), (1, 8), (90, 64)]
    inst, st = [], [[], [], [], []]
    for i, (nx, ny) in enumerate(sizes):
        geo, f = state(swe, nx, ny, 1, i, dry=False)
        inst.append((nx, ny, 5.0 + i, 6.0, [1, 0, 0, 1]))
        for a, v in zip(st, f):
            a.append(v)
    st = [np.concatenate(a) for a in st]
    pair(swe, lambda c: swe.Ensemble(inst, solver=solver, tile_cols=c), st, lambda D: D.advance(2.5))


def test_small_long_runs_and_mixed_calls(swe):
    """more steps than one launch takes, and the block calls between"""
    geo, st = state(swe, 48, 40, 1, 3, dry=False)

    def drive(D):
        D.step(300)
        dts = []
        for _ in range(3):
            D.set_ghost_layer()
            D.compute_fluxes()
            dts.append(D.max_timestep())
            D.update_unknowns()
        D.step(2)
        return dts

    pair(swe, lambda c: swe.Domain([48], [40], geo["dx"], geo["dy"], boundary=[1] * 4, solver=4, tile_cols=c), st, drive)
