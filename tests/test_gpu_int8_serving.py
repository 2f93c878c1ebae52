"""Problems whose products run on the int8 tensor cores, served (the same bits as alone), and their workspaces."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("integrator", ["kn", "rb_kn"])
def test_loops_with_slices_served_as_alone(cuda, integrator):
    """From 8e6 elements of Qs on the loops multiply with its int8 slices; a worker's share of the SMs must not change
    that, nor the bits."""
    from mcnla_b200 import isvd, synthetic
    m, n, k, p, N = 8200, 900, 48, 16, 16
    a = torch.as_tensor(synthetic.lowrank_np(m, n, [1.0 / j for j in range(1, 121)], seed=3, noise=1e-4), device=cuda)
    reqs = [isvd.Request(a, k, p, N, seed=5 + i, integrator=integrator, former="svd", tol=1e-6, maxit=32)
            for i in range(3)]
    with isvd.Server(workers=2) as server:
        for r in reqs:
            server.submit(r)
        for r in reqs:
            server.wait(r)
    for i, r in enumerate(reqs):
        s, u, v, it = isvd.solve(a, k, p, N, seed=5 + i, integrator=integrator, former="svd", tol=1e-6, maxit=32)
        assert it == r.result.iteration
        assert torch.equal(s, r.s) and torch.equal(u, r.u) and torch.equal(v, r.v)


@pytest.mark.parametrize("name", ["KolmogorovNagumoIntegrator", "RowBlockKolmogorovNagumoIntegrator"])
def test_initialize_allocates_what_the_loop_uses(cuda, name):
    from mcnla_b200 import isvd
    m, l, N = 60000, 64, 16 if name.startswith("K") else 20
    g = torch.Generator(device=cuda)
    g.manual_seed(2)
    q = torch.randn(m, l * N, generator=g, dtype=torch.float64, device=cuda) / m ** 0.5
    prm = isvd.Parameters().setSize(m, 1000).setRank(l).setOverRank(0).setNumSketch(N).sync()
    st = getattr(isvd, name)(prm, 16, 1e-6)
    st.initialize()
    qbar = prm.createMatrixQbar()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    st(q, qbar)
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < 64 << 20      # the code of a kernel's first launch, not 14 m L bytes


def test_mixed_request_is_admitted_without_the_int8_sketch(cuda):
    """A mixed solve sketches on BF16 parts: it is admitted with less than the upper estimate, whose largest term is the
    workspace of an FP64 sketch."""
    from mcnla_b200 import isvd, synthetic
    m, n, k, p, N = 8192, 2048, 32, 16, 8
    a = torch.as_tensor(synthetic.lowrank_np(m, n, [1.0 / j for j in range(1, 81)], seed=3, noise=1e-4), device=cuda)
    req = isvd.Request(a, k, p, N, seed=5, integrator="rb_gramian_kn", former="svd", tol=1e-5, mixed=3)
    with isvd.Server(workers=1) as server:
        server.wait(server.submit(req))
        peak = server.stats()["peak_bytes"]
    assert req.result.status == 0
    assert peak < req.bytes() - (100 << 20)
