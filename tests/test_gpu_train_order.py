"""An epoch's order of the edges (shuffled on the device) against the sequential
Fisher-Yates shuffle: with batches of one edge, training on all edges gives the
same bits as training on one edge after the other in that order, epoch after
epoch."""
import numpy as np
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu

MASK = (1 << 64) - 1


def orders(n, seed, epochs):
    """the shuffle's orders from a splitmix64 stream"""
    s = seed
    for _ in range(epochs):
        p = list(range(n))
        for i in range(n - 1, 0, -1):
            s = (s + 0x9E3779B97F4A7C15) & MASK
            z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & MASK
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & MASK
            j = (z ^ (z >> 31)) % (i + 1)
            p[i], p[j] = p[j], p[i]
        yield p


@pytest.mark.parametrize("n,epochs,seed", [(1, 2, 5), (2, 3, 0), (3, 3, 9), (17, 2, 1), (255, 1, 7), (256, 1, 8), (257, 2, MASK),
                                           (1500, 1, 123456789)])
def test_order_equals_sequential_shuffle(swe, n, epochs, seed):
    r = np.random.default_rng(n)
    h = r.uniform(0.5, 5.0, (2, n))
    e = np.stack([h[0], h[1], h[0] * r.uniform(-1, 1, n), h[1] * r.uniform(-1, 1, n), r.uniform(-1, 1, n),
                  r.uniform(-1, 1, n)]).astype(np.float32)
    t = r.uniform(-1, 1, (4, n)).astype(np.float32)
    a, b = swe.Surrogate(3), swe.Surrogate(3)
    a.train(e, t, epochs=epochs, batch=1, lr=1e-2, seed=seed)
    for p in orders(n, seed, epochs):
        for k in p:
            b.train(e[:, k:k + 1], t[:, k:k + 1], epochs=1, batch=1, lr=1e-2, seed=0)
    assert_bitwise(a.params, b.params, "parameters after %d edges" % (n * epochs))
    a.close()
    b.close()
