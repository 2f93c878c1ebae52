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


def _sketch_ms(a, omega, k, p, N):
    from mcnla_b200 import isvd
    m, n = a.shape
    prm = isvd.Parameters().setSize(m, n).setRank(k).setOverRank(p).setNumSketch(N).sync()
    st = isvd.GaussianProjectionSketcher(prm, 0, 0).setOmega(omega)
    st.initialize()
    q = prm.createCollectionQ()
    times = []
    for _ in range(8):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        st(a, q)
        e1.record()
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1))
    return q, min(times)


@pytest.mark.parametrize("m,n", [(16384, 4096), (16321, 4095)])
def test_spread_rows_for_the_fp64_units(cuda, m, n):
    """A sparse row in every 64 leaves no tile to the int8 units: the sketch must not take longer than that of a matrix
    of sparse rows alone, which the FP64 units compute, and gives what they give."""
    k, p, N = 64, 32, 8
    g = torch.Generator(device=cuda)
    g.manual_seed(12)
    a = torch.randn(m, n, generator=g, dtype=torch.float64, device=cuda)
    omega = torch.randn(n, (k + p) * N, generator=g, dtype=torch.float64, device=cuda)
    keep = torch.rand(n, generator=g, device=cuda) < 8.0 / n
    a[::64] *= keep
    q, some = _sketch_ms(a, omega, k, p, N)
    ref = a @ omega
    assert float(((q - ref).norm(dim=1) / (a.norm(dim=1) * omega.norm() + 1e-300)).max()) < 1e-14
    a *= keep
    _, every = _sketch_ms(a, omega, k, p, N)
    assert some < 1.12 * every


@pytest.mark.parametrize("n,layout", [(1200, "row"), (24000, "row"), (24000, "col")])
def test_flags_over_chunks(cuda, n, layout):
    """More columns of A than a chunk of K holds, with a NaN, an infinity and a sparse row whose entries lie in the last
    chunk: the FP64 units' values in those rows' tiles, in the others the bound."""
    from test_gpu_int8 import _check, _sketch
    m, k, p, N = 1500, 100, 28, 32
    g = torch.Generator(device=cuda)
    g.manual_seed(n)
    a = torch.randn(m, n, generator=g, dtype=torch.float64, device=cuda)
    omega = torch.randn(n, (k + p) * N, generator=g, dtype=torch.float64, device=cuda)
    a[300, n - 2] = float("nan")
    a[700, n - 3] = float("inf")
    a[1100] = 0
    a[1100, n - 5] = 2.0
    x = a.t().contiguous().t() if layout == "col" else a
    q, _ = _sketch(x, omega, k, p, N)
    ref = a @ omega
    assert torch.isnan(q[300]).all() and torch.equal(q[700], ref[700])
    assert torch.equal(q[1100], 2.0 * omega[n - 5])
    _check(q, a, omega, [0, 127, 128, 255, 1025, 1151, 1152, 1499], [0, 255, 256, 4095])
    ok = torch.ones(m, dtype=torch.bool, device=cuda)
    ok[[300, 700]] = False
    assert float(((q - ref)[ok].norm(dim=1) / (a[ok].norm(dim=1) * omega.norm())).max()) < 1e-14


@pytest.mark.parametrize("m,n,k,p,N", [(2048, 4096, 64, 32, 16), (2176, 4001, 64, 32, 16), (4480, 4096, 16, 8, 8)])
def test_omega_small_where_a_is_large(cuda, m, n, k, p, N):
    """Sums whose large factors do not meet: an Omega that is zero where A is large, a share of A's rows with few entries,
    and a power iteration on rows of two scales.  The error stays within what a running FP64 sum loses by
    elements, sqrt(K) 2^-53 |A| |B| (rounding errors of K terms, uncorrelated)."""
    import numpy as np
    from test_gpu_int8 import _sketch
    g = torch.Generator(device=cuda)
    g.manual_seed(n)
    a = torch.randn(m, n, generator=g, dtype=torch.float64, device=cuda)
    omega = torch.randn(n, (k + p) * N, generator=g, dtype=torch.float64, device=cuda)
    a[:, :n // 2] *= 1e10
    omega[:n // 2] = 0
    a[1000:1100] *= torch.rand(100, n, generator=g, device=cuda) < 0.01
    q, _ = _sketch(a, omega.clone(), k, p, N)
    rows = [0, 1, 127, 128, 1000, 1050, 1099, m - 1]
    cols = list(range(0, (k + p) * N, 37))
    al, bl = a[rows].cpu().numpy().astype(np.longdouble), omega[:, cols].cpu().numpy().astype(np.longdouble)
    err = np.abs(q[rows][:, cols].cpu().numpy() - al @ bl)
    assert (err <= 2.0 ** -53 * n ** 0.5 * (np.abs(al) @ np.abs(bl))).all()
    # A' Q with Q = A Omega: columns of A that live on the small rows alone
    a = torch.randn(m, n, generator=g, dtype=torch.float64, device=cuda)
    a[:m // 2, n // 2:] = 0
    a[m // 2:, :n // 2] = 0
    a[m // 2:] *= 1e-8
    omega = torch.randn(n, (k + p) * N, generator=g, dtype=torch.float64, device=cuda)
    q, _ = _sketch(a, omega.clone(), k, p, N, exponent=1)
    ref = a @ (a.T @ (a @ omega))
    low = q[m // 2:]
    assert float((low - ref[m // 2:]).norm() / ref[m // 2:].norm()) < 1e-13


def test_gramian_over_chunks(cuda):
    """Bs = Qs' Qs with more rows than a chunk of K holds: the same Qbar as the row-block form, which makes no Gramian."""
    m, l, N = 40001, 64, 16
    g = torch.Generator(device=cuda)
    g.manual_seed(21)
    base = torch.linalg.qr(torch.randn(m, l, generator=g, dtype=torch.float64, device=cuda))[0]
    q = _orth(base[None] + 0.3 / m ** 0.5 * torch.randn(N, m, l, generator=g, dtype=torch.float64, device=cuda))
    a, ita = _integrate("RowBlockGramianKolmogorovNagumoIntegrator", q, l, N, 64, 1e-6)
    b, itb = _integrate("RowBlockKolmogorovNagumoIntegrator", q, l, N, 64, 1e-6)
    assert ita == itb and float((a - b).abs().max()) < 1e-12
