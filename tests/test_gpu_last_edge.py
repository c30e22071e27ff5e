"""The split step whose dt keeps the last edge's speed (one thread per group
instead of a pass over every edge) against the oracle, bit for bit: dt and
state, sizes around the tiles, ensembles, and a last edge that is dry (dt
infinite, as the reference computes it)."""
import numpy as np
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", [1, 2, 3, 4])
@pytest.mark.parametrize("nx,ny", [(1, 1), (31, 257), (130, 64), (700, 300)])
def test_last_edge_equals_oracle(swe, oracle_mod, solver, nx, ny):
    geo, h, hu, hv, b = swe.init_domain(swe.SCENARIO_DAM_BREAK, nx, ny, 1, [1000.0, 200.0, 12.0, 6.0, 0.0])
    kw = dict(solver=solver, semantics=swe.SPLIT, split_dt_mode=swe.SPLIT_DT_LAST_EDGE)
    D = swe.Domain([nx], [ny], geo["dx"], geo["dy"], boundary=geo["boundary"], **kw)
    R = oracle_mod.Domain([nx], [ny], geo["dx"], geo["dy"], outer=geo["boundary"], **kw)
    D.upload(h, hu, hv, b)
    R.set_state(h, hu, hv, b)
    D.exchange_bathymetry()
    R.bathymetry_ghosts()
    D.step(6)
    dts = R.step(6)
    for a, r, k in zip(D.download(), R.get_state(), ("h", "hu", "hv", "b")):
        assert_bitwise(a, r, k)
    assert np.float32(D.group_state()[1][0]) == np.float32(np.asarray(dts).ravel()[-1])
    D.close()


def test_last_edge_ensemble_and_dry_corner(swe):
    sizes = [(40, 33), (65, 300), (31, 129)]
    inst, st = [], [[], [], [], []]
    for i, (nx, ny) in enumerate(sizes):
        geo, *f = swe.init_domain(swe.SCENARIO_DAM_BREAK, nx, ny, 1, [1000.0, 150.0, 12.0, 5.0 + i, 0.0])
        if i == 2:  # dry where the last edge lies
            f[0].reshape(nx + 2, ny + 2)[-3:, -3:] = 0.0
        inst.append((nx, ny, geo["dx"], geo["dy"], geo["boundary"]))
        for a, v in zip(st, f):
            a.append(v)
    kw = dict(solver=4, semantics=swe.SPLIT, split_dt_mode=swe.SPLIT_DT_LAST_EDGE)
    E = swe.Ensemble(inst, **kw)
    E.upload(*[np.concatenate(a) for a in st])
    E.exchange_bathymetry()
    E.step(1)
    _, dt, _ = E.group_state()
    assert np.isinf(dt[2]) and np.isfinite(dt[:2]).all()
    for i, (nx, ny, dx, dy, bnd) in enumerate(inst[:2]):
        D = swe.Domain([nx], [ny], dx, dy, boundary=bnd, **kw)
        D.upload(*[a[i] for a in st])
        D.exchange_bathymetry()
        D.step(1)
        assert np.float32(D.group_state()[1][0]) == dt[i]
        for a, r in zip(E.download_block(i), D.download_block(0)):
            assert_bitwise(a, r, "instance %d" % i)
        D.close()
    E.close()
