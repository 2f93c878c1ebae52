"""KN loops that end within their first iterations (csrc/stages.cu, kn_loop)."""
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["KolmogorovNagumoIntegrator", "RowBlockKolmogorovNagumoIntegrator"])
def test_no_graph_is_captured_for_a_loop_that_ends_in_its_first_chunk(cuda, name):
    """A capture costs more than the loop itself then: the run with graph loops takes no longer than without."""
    from mcnla_b200 import _lib, isvd
    m, l, N = 1000, 20, 16
    g = torch.Generator(device=cuda)
    g.manual_seed(3)
    base = torch.linalg.qr(torch.randn(m, l, generator=g, dtype=torch.float64, device=cuda))[0]
    noise = torch.randn(N, m, l, generator=g, dtype=torch.float64, device=cuda)
    q = torch.linalg.qr(base[None] + 1e-4 * noise)[0].permute(1, 0, 2).reshape(m, -1).contiguous()
    prm = isvd.Parameters().setSize(m, m).setRank(l).setOverRank(0).setNumSketch(N).sync()
    st = getattr(isvd, name)(prm, 256, 1e-3)
    st.initialize()
    qbar = prm.createMatrixQbar()
    ctx = isvd.context()
    best = {}
    try:
        for i in range(40):
            for on in (0, 1):
                _lib.check(ctx.lib.mcnla_b200_set_graph_loop(ctx.bind(), on), "set_graph_loop")
                torch.cuda.synchronize()
                t = time.perf_counter()
                st(q, qbar)
                torch.cuda.synchronize()
                best[on] = min(best.get(on, 1e9), time.perf_counter() - t)
    finally:
        _lib.check(ctx.lib.mcnla_b200_set_graph_loop(ctx.bind(), 1), "set_graph_loop")
    assert st.iteration() <= 8
    assert best[1] < 1.15 * best[0], best
