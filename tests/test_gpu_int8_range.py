"""The loops' int8-slice products (csrc/slice_gemm.cu) on bases outside the dense, evenly scaled ones: rows of any finite
magnitude, and rows and columns in which few entries dominate."""
import pytest
import torch

from test_gpu_int8 import _kn

pytestmark = pytest.mark.gpu


def _integrate(cls, q, l, N, maxit, tol):
    from mcnla_b200 import isvd
    prm = isvd.Parameters().setSize(q.shape[0], q.shape[0]).setRank(l).setOverRank(0).setNumSketch(N).sync()
    st = getattr(isvd, cls)(prm, maxit, tol)
    st.initialize()
    qbar = prm.createMatrixQbar()
    st(q, qbar)
    return qbar, st.iteration()


def _orth(y):
    return torch.linalg.qr(y)[0].permute(1, 0, 2).reshape(y.shape[1], -1).contiguous()


@pytest.mark.parametrize("scale", [1e-121, 1e-130, 1e-250, 1e-300])
@pytest.mark.parametrize("cls", ["KolmogorovNagumoIntegrator", "RowBlockKolmogorovNagumoIntegrator"])
def test_row_of_tiny_magnitude(cuda, cls, scale):
    """A row of Qs is as small as A's row.  Its result keeps the relative accuracy of an FP64 product."""
    m, l, N = 8192, 64, 16
    g = torch.Generator(device=cuda)
    g.manual_seed(4)
    y = torch.randn(m, l, generator=g, dtype=torch.float64, device=cuda)[None]
    y = y + 0.3 * torch.randn(N, m, l, generator=g, dtype=torch.float64, device=cuda)
    y[:, 100] = 0
    q = _orth(y)
    q[100] = scale * torch.randn(l * N, generator=g, dtype=torch.float64, device=cuda)
    qbar, it = _integrate(cls, q, l, N, 12, 1e-9)
    ref, itr = _kn(q, l, N, 12, 1e-9)
    assert it == itr and float((qbar - ref).abs().max()) < 1e-12
    assert float((qbar[100] - ref[100]).abs().max()) < 1e-12 * float(ref[100].abs().max())


@pytest.mark.parametrize("integrator", ["kn", "rb_kn"])
def test_solve_with_a_tiny_row(cuda, integrator):
    from mcnla_b200 import isvd
    m, n, k, p, N = 8192, 1200, 50, 14, 16
    g = torch.Generator(device=cuda)
    g.manual_seed(6)
    a = torch.randn(m, 80, generator=g, dtype=torch.float64, device=cuda) @ torch.randn(
        80, n, generator=g, dtype=torch.float64, device=cuda)
    omega = torch.randn(n, (k + p) * N, generator=g, dtype=torch.float64, device=cuda)
    a[77] *= 1e-130
    kw = dict(integrator=integrator, former="svd", maxit=16, tol=1e-6)
    s, u, v, it = isvd.solve(a, k, p, N, omega=omega.clone(), **kw)
    a[77] = 0
    s0, u0, v0, it0 = isvd.solve(a, k, p, N, omega=omega.clone(), **kw)
    assert it == it0 and all(bool(torch.isfinite(x).all()) for x in (s, u, v))
    assert float(((s - s0) / s0).abs().max()) < 1e-12
    assert 1e-140 < float(u[77].abs().max()) < 1e-125


@pytest.mark.parametrize("rest", [1e-5, 1e-7])
@pytest.mark.parametrize("cls", ["KolmogorovNagumoIntegrator", "RowBlockKolmogorovNagumoIntegrator"])
def test_columns_of_one_dominating_entry(cuda, cls, rest):
    """Bases of a matrix with localized singular vectors.  Against the definition in FP64 the two differ by a few
    roundings of every product's result an iteration: 8 maxit 2^-53 ||Qbar||_F, ||Qbar||_F = sqrt(l)."""
    m, l, N, maxit = 16384, 48, 16, 12
    g = torch.Generator(device=cuda)
    g.manual_seed(1)
    base = rest * torch.randn(m, l, generator=g, dtype=torch.float64, device=cuda)
    base[torch.randperm(m, generator=g, device=cuda)[:l], torch.arange(l, device=cuda)] = 1.0
    q = _orth(base[None] + 0.1 * rest * torch.randn(N, m, l, generator=g, dtype=torch.float64, device=cuda))
    qbar, it = _integrate(cls, q, l, N, maxit, 0.0)
    ref, itr = _kn(q, l, N, maxit, 0.0)
    assert it == itr
    assert float((qbar - ref).norm()) < 8 * maxit * 2.0 ** -53 * l ** 0.5
