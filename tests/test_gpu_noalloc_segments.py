"""The allocation-free step's segments: results do not depend on how a block is
cut, bit for bit."""
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# column counts around one, two and three columns per segment (4 CTAs on each of 152 SMs), one
# row, one cell, several row tiles, and a block that fills the GPU with 32-column segments
@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 33), (607, 40), (608, 40), (609, 40), (1216, 31), (1217, 32), (1825, 64),
                                   (300, 700), (32, 5000), (2600, 1900)])
@pytest.mark.parametrize("solver,semantics", [(4, 0), (3, 1)])
def test_noalloc_segments(swe, nx, ny, solver, semantics):
    geo, h, hu, hv, b = swe.init_domain(swe.SCENARIO_DAM_BREAK, nx, ny, 1, [1000.0, 200.0, 12.0, 6.0, 0.0])
    D = swe.Domain([nx], [ny], geo["dx"], geo["dy"], boundary=geo["boundary"], solver=solver, semantics=semantics)
    D.upload(h, hu, hv, b)
    D.step(1)
    D.set_ghost_layer()
    ref = D.download()[:3]
    D.close()
    ins = [torch.from_numpy(a).cuda() for a in (h, hu, hv, b)]
    outs = [torch.zeros_like(ins[0]) for _ in range(3)]
    torch.cuda.synchronize()
    swe.step_block_noalloc(solver, semantics, nx, ny, geo["dx"], geo["dy"], geo["boundary"], ny + 2,
                           [t.data_ptr() for t in ins], [t.data_ptr() for t in outs])
    torch.cuda.synchronize()
    for t, r, k in zip(outs, ref, ("h", "hu", "hv")):
        assert_bitwise(t.cpu().numpy(), r, k)
