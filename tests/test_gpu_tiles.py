"""The default partition of the step kernels (tile height and segment length by
the domain's shape): results do not
depend on them, bit for bit."""
import numpy as np
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu


def dam(swe, nx, ny, seed):
    r = np.random.default_rng(seed)
    prm = [1000.0, float(r.uniform(60, 300)), float(r.uniform(9, 15)), float(r.uniform(4, 8)), 0.0]
    return swe.init_domain(swe.SCENARIO_DAM_BREAK, nx, ny, 1, prm)


# heights around the choice of 128- or 256-row tiles (partial tiles of 1 row, full ones, one short of full)
@pytest.mark.parametrize("arithmetic", [0, 1])
@pytest.mark.parametrize("ny", [127, 128, 129, 255, 256, 257, 300, 383, 384, 385])
def test_default_tile_height(swe, ny, arithmetic):
    geo, h, hu, hv, b = swe.init_domain(swe.SCENARIO_TSUNAMI, 94, 2 * ny, 4, [94, 7])
    out = []
    for rows in (0, 256):
        D = swe.Domain(geo["nx_cols"], geo["ny_rows"], geo["dx"], geo["dy"], boundary=geo["boundary"], tile_rows=rows,
                       arithmetic=arithmetic)
        D.upload(h, hu, hv, b)
        D.exchange_bathymetry()
        D.step(5)
        out.append(D.download() + (np.float32(D.time()[0]),))
        D.close()
    for a, r, k in zip(*out, ("h", "hu", "hv", "b", "t")):
        assert_bitwise(np.asarray(a), np.asarray(r), "%s ny=%d" % (k, ny))


# runs past 64 columns per CTA with partly idle tiles: short segments
@pytest.mark.parametrize("arithmetic", [0, 1])
@pytest.mark.parametrize("nx,heights", [(2000, (90, 110, 65)), (2300, (140, 131, 33))])
def test_short_segments_of_partial_tiles(swe, nx, heights, arithmetic):
    sizes = [(nx + 3 * i, heights[i % 3]) for i in range(24)]
    inst, state = [], [[], [], [], []]
    for i, (x, y) in enumerate(sizes):
        geo, *f = dam(swe, x, y, i)
        inst.append((x, y, geo["dx"], geo["dy"], geo["boundary"]))
        for s, v in zip(state, f):
            s.append(v)
    state = [np.concatenate(s) for s in state]
    out = []
    for rows, cols in ((0, 0), (256, 128)):
        E = swe.Ensemble(inst, arithmetic=arithmetic, tile_rows=rows, tile_cols=cols)
        E.upload(*state)
        E.exchange_bathymetry()
        E.step(4)
        out.append(E.download() + E.group_state())
        E.close()
    for a, r, k in zip(*out, ("h", "hu", "hv", "b", "time", "dt", "steps")):
        assert_bitwise(a, r, k)
