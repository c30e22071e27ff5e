"""advance() after an upload whose ghost ring holds anything: it steps on the
ring that the boundary conditions and the neighbours give, as step() does, for
few steps and many, at a handle's first call and at later ones, whether several
steps go out in one launch (small domains) or as a captured graph.  Bit for bit
against step() on a fresh handle."""
import numpy as np
import pytest

from helpers import assert_bitwise, interior_mask

pytestmark = pytest.mark.gpu

# (nx, ny, blocks, more): small and beyond, every kind of step
DOMAINS = {
    "small": (96, 80, 4, dict(solver=4)),
    "small_hybrid": (130, 70, 1, dict(solver=3)),
    "bounded": (1300, 900, 4, dict(solver=4)),
    "augmented": (700, 600, 4, dict(solver=2)),
    "two_pass": (300, 200, 1, dict(solver=1, tile_cols=32)),
    "split_last_edge": (300, 200, 1, dict(solver=1, semantics=1, split_dt_mode=1)),
    "split_max": (300, 200, 1, dict(solver=4, semantics=1, split_dt_mode=0)),
    "fast": (300, 200, 4, dict(solver=4, arithmetic=1)),
}


def state(swe, nx, ny, nb, seed):
    """uneven water over an uneven bed, ghost cells of h, hu and hv garbage"""
    geo, h, hu, hv, b = swe.init_domain(swe.SCENARIO_DAM_BREAK, nx, ny, nb, [1000.0, 200.0, 12.0, 6.0, 0.0])
    r = np.random.default_rng(seed)
    q = [h + r.uniform(0, 1, h.shape), h * r.uniform(-1, 1, h.shape), h * r.uniform(-1, 1, h.shape)]
    ghost = ~interior_mask(geo["nx_cols"], geo["ny_rows"])
    for v in q:
        v[ghost] = r.uniform(20, 30, int(ghost.sum()))
    return geo, [v.astype(np.float32) for v in q] + [r.uniform(-1, 1, b.shape).astype(np.float32)]


def fresh(swe, geo, more, st):
    D = swe.Domain(geo["nx_cols"], geo["ny_rows"], geo["dx"], geo["dy"], boundary=[1, 0, 0, 1], **more)
    upload(D, st)
    return D


def upload(D, st):
    D.upload(*st)
    D.exchange_bathymetry()


def stepped(swe, geo, more, st, n):
    D = fresh(swe, geo, more, st)
    D.step(n)
    out = D.download()
    D.close()
    return out


def same(D, ref, what):
    assert D.status() == 0
    for a, r, k in zip(D.download(), ref, ("h", "hu", "hv", "b")):
        assert_bitwise(a, r, "%s: %s" % (what, k))


@pytest.mark.parametrize("name", DOMAINS)
def test_advance_sets_the_ring_after_an_upload(swe, name):
    nx, ny, nb, more = DOMAINS[name]
    geo, first = state(swe, nx, ny, nb, 1)
    _, second = state(swe, nx, ny, nb, 2)
    D = fresh(swe, geo, more, first)
    D.advance(1e30, max_steps=0)  # (takes no step)
    assert D.advance(1e30, max_steps=5)[0] == 5
    same(D, stepped(swe, geo, more, first, 5), "first call, few steps")
    for st, n in ((second, 16), (first, 3), (second, 35)):
        upload(D, st)
        assert D.advance(1e30, max_steps=n)[0] == n
        same(D, stepped(swe, geo, more, st, n), "later upload, %d steps" % n)
    D.close()
    D = fresh(swe, geo, more, first)  # the first call on a ring that is valid already
    D.set_ghost_layer()
    D.advance(1e30, max_steps=16)
    same(D, stepped(swe, geo, more, first, 16), "after set_ghost_layer")
    upload(D, second)
    D.advance(1e30, max_steps=16)
    same(D, stepped(swe, geo, more, second, 16), "upload after a call on a valid ring")
    D.close()
