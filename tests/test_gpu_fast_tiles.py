"""The fast-arithmetic step solves an edge once from each side where two lanes,
two warps or two tiles meet (packed in one, as a single edge in the other).
Both must give the same bits: the state after a few steps does not depend on
where the tiles' and warps' rows end."""
import numpy as np
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["HLLE", "FWAVE"])
@pytest.mark.parametrize("sid,nx,ny,nb,params", [
    (10, 96, 259, 1, [1000.0, 150.0, 20.0, 0.5, 0, 0, 0]),  # supercritical front: edges solved again
    (11, 130, 192, 2, [192, 7.0, 100000.0]),                 # wet everywhere, ragged columns
    (12, 96, 96, 1, [3.0, 50000.0]),                         # dry cells
])
def test_fast_step_does_not_depend_on_the_tile_rows(swe, solver, sid, nx, ny, nb, params):
    geo, h, hu, hv, b = swe.init_domain(sid, nx, ny, nb, params)
    outs = []
    for rows in (64, 256):
        D = swe.Domain(geo["nx_cols"], geo["ny_rows"], geo["dx"], geo["dy"], boundary=geo["boundary"],
                       solver=getattr(swe, solver), arithmetic=swe.FAST, tile_rows=rows)
        D.upload(h, hu, hv, b)
        D.exchange_bathymetry()
        D.step(7)
        D.set_ghost_layer()
        outs.append((D.download(), D.time()[0]))
        assert D.status() == 0
        D.close()
    (a, ta), (c, tc) = outs
    assert np.float32(ta) == np.float32(tc)
    for x, y, k in zip(a, c, "h hu hv b".split()):
        # a wave that vanishes may leave either zero
        assert_bitwise(x + np.float32(0), y + np.float32(0), k)
