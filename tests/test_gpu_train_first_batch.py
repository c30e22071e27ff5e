"""The first batch of an epoch takes the epoch's own order.  The kernel that
trains a batch reads its edges ahead of its wait for the launch before it, and
for an epoch's first batch that launch is the shuffle: it must be over.  So a
handle whose buffer for the order holds something else -- another seed's order
of the same edges, the order of more edges, or nothing yet -- trains to the same
bits, with the batch that is read first as large as the whole set or a tile of
it.  Where the first batch is trained on stale order, the parameters differ."""
import numpy as np
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu


def edges(n):
    r = np.random.default_rng(n)
    h = r.uniform(0.5, 5.0, (2, n))
    e = np.stack([h[0], h[1], h[0] * r.uniform(-1, 1, n), h[1] * r.uniform(-1, 1, n), r.uniform(-1, 1, n),
                  r.uniform(-1, 1, n)]).astype(np.float32)
    return e, r.uniform(-1, 1, (4, n)).astype(np.float32)


@pytest.mark.parametrize("n,batch", [(129, 128), (8192, 128), (65536, 8192), (300000, 4096), (300000, 300000)])
def test_first_batch_takes_the_new_order(swe, n, batch):
    e, t = edges(n)
    more = edges(n + 77)
    used, got = swe.Surrogate(3), []
    start = used.params
    for before in (None, (e, t, 99), more + (7,)):
        if before:  # leaves another order behind
            used.train(before[0], before[1], epochs=1, batch=batch, lr=1e-2, seed=before[2])
        used.params = start
        losses = used.train(e, t, epochs=3, batch=batch, lr=1e-2, seed=5)
        got.append((np.asarray(losses), used.params))
    fresh = swe.Surrogate(3)
    fresh.params = start
    ref = np.asarray(fresh.train(e, t, epochs=3, batch=batch, lr=1e-2, seed=5)), fresh.params
    for losses, params in got:
        assert_bitwise(losses, ref[0], "losses")
        assert_bitwise(params, ref[1], "parameters")
    used.close()
    fresh.close()
