"""The allocation-free block step in one cooperative launch (blocks whose CTAs
are all resident at once) against a domain's two-pass step, bit for bit: one,
two and four columns per CTA, blocks just within and just beyond the limit
(of resident CTAs, and of the unit table),
one-cell blocks, and a captured call replayed on a second state."""
import numpy as np
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

RIM = [1, 2, 0, 1]  # wall, inflow (kept), outflow, wall


def state(nx, ny, seed):
    r = np.random.default_rng(seed)
    q = [10.0 + r.random((nx + 2, ny + 2)), r.random((nx + 2, ny + 2)) - 0.5, r.random((nx + 2, ny + 2)) - 0.5,
         -10.0 + 0.1 * r.random((nx + 2, ny + 2))]
    q[0][: nx // 3] = 0.0  # a dry part
    q[1][: nx // 3] = q[2][: nx // 3] = 0.0
    return [a.astype(np.float32) for a in q]


def two_pass(swe, solver, nx, ny, st):
    D = swe.Domain([nx], [ny], 10.0, 12.0, boundary=RIM, solver=solver, speed_pass=1)
    D.upload(*[a.ravel() for a in st])
    D.set_ghost_layer()
    D.compute_fluxes()
    dt = D.max_timestep()
    D.update_unknowns()
    D.set_ghost_layer()
    out = D.download()[:3]
    D.close()
    return dt, out


@pytest.mark.parametrize("solver,nx,ny", [
    (4, 1, 1), (4, 33, 31), (1, 608, 256), (1, 609, 256), (4, 1217, 255), (3, 300, 300), (2, 424, 26),
    (4, 1824, 250), (4, 1900, 256), (1, 2500, 100), (4, 4096, 20), (1, 4500, 20),
])
def test_block_step_equals_two_pass_step(swe, solver, nx, ny):
    cur = [torch.empty((nx + 2) * (ny + 2), device="cuda") for _ in range(4)]
    nxt = [torch.empty_like(cur[0]) for _ in range(3)]
    graph = torch.cuda.CUDAGraph()

    def call(stream, want_dt):
        return swe.step_block_noalloc(solver, 0, nx, ny, 10.0, 12.0, RIM, ny + 2, [t.data_ptr() for t in cur],
                                      [t.data_ptr() for t in nxt], stream=stream, want_dt=want_dt)

    for k in range(2):
        st = state(nx, ny, 7 * k + nx)
        dt, ref = two_pass(swe, solver, nx, ny, st)
        for t, a in zip(cur, st):
            t.copy_(torch.from_numpy(a.ravel()))
        for t in nxt:
            t.fill_(-1.0)
        torch.cuda.synchronize()
        if k == 0:
            got = call(torch.cuda.current_stream().cuda_stream, True)
            assert np.float32(got) == np.float32(dt)
            torch.cuda.synchronize()
            with torch.cuda.graph(graph):
                call(torch.cuda.current_stream().cuda_stream, False)
        else:
            graph.replay()
            torch.cuda.synchronize()
        for t, r, name in zip(nxt, ref, ("h", "hu", "hv")):
            assert_bitwise(t.cpu().numpy(), np.asarray(r).ravel(), "state %d %s" % (k, name))
