"""The edge pass's tiles where a column's y-edges do not fill them (heights that
are a multiple of 128 take the lowest y-edges along the row): the augmented
solver's default step against its two-pass step, and the surrogate's counted
edges, bit for bit."""
import numpy as np
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nb", [(700, 127, 1), (700, 128, 1), (129, 1280, 1), (640, 1024, 4), (513, 1023, 1), (1100, 256, 2)])
def test_edge_tiles(swe, nx, ny, nb):
    geo, h, hu, hv, b = swe.init_domain(swe.SCENARIO_DAM_BREAK, nx, ny, nb, [1000.0, 200.0, 12.0, 6.0, 0.0])
    r = np.random.default_rng(nx)
    b = r.uniform(-1, 1, b.shape).astype(np.float32)
    out = []
    for mode in ("default", "two-pass", "surrogate call"):
        D = swe.Domain(geo["nx_cols"], geo["ny_rows"], geo["dx"], geo["dy"], boundary=geo["boundary"], solver=swe.AUGRIE,
                       speed_pass=1 if mode == "two-pass" else 0, tile_cols=128)
        D.upload(h, hu, hv, b)
        D.exchange_bathymetry()
        if mode == "surrogate call":
            D.set_ghost_layer()
            assert D.surrogate_step(None, 4) == 0
        else:
            D.step(4)
        out.append(D.download() + (np.asarray(D.time(), np.float32),))
        D.close()
    for got in (out[0], out[2]):
        for a, x, k in zip(got, out[1], ("h", "hu", "hv", "b", "time")):
            assert_bitwise(a, x, k)


def test_surrogate_counts_every_edge_once(swe):
    """all wet, still and flat: the fitted-to-zero network passes the gate on every edge"""
    nx, ny = 300, 256
    D = swe.Domain([nx], [ny], 10.0, 10.0, boundary=[0] * 4, solver=swe.HLLE)
    n = (nx + 2) * (ny + 2)
    D.upload(np.full(n, 5.0), np.zeros(n), np.zeros(n), np.zeros(n))
    D.exchange_bathymetry()
    D.set_ghost_layer()
    assert D.surrogate_step(swe.Surrogate(0), 1) == D.surrogate_edge_count()
    D.close()
