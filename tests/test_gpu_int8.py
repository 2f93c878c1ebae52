"""FP64 products on the int8 tensor cores (csrc/rns_gemm.cu), through the sketcher and the whole solve.

A product takes this path by its size; the sizes here are just above the line, around the edges of its 256 x 256 x 128
tiles.  Bound: row a is scaled to a 2-norm in (2^56, 2^57] and rounded to integers, column b to (2^57, 2^58], so
the product is off by at most sqrt(K) (2^-57 + 2^-58) |a| |b| (plus the second-order term) and one rounding.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sketch(a, omega, k, p, N, exponent=0):
    from mcnla_b200 import isvd
    m, n = a.shape
    prm = isvd.Parameters().setSize(m, n).setRank(k).setOverRank(p).setNumSketch(N).sync()
    st = isvd.GaussianProjectionSketcher(prm, 0, exponent).setOmega(omega)
    st.initialize()
    q = prm.createCollectionQ()
    before = isvd.context().kernels_launched()
    st(a, q)
    return q, isvd.context().kernels_launched() - before


def _check(q, a, omega, rows, cols):
    al, bl = a[rows].cpu().numpy().astype(np.longdouble), omega[:, cols].cpu().numpy().astype(np.longdouble)
    ref = al @ bl
    na, nb = np.sqrt((al ** 2).sum(1)), np.sqrt((bl ** 2).sum(0))
    K = a.shape[1]
    bound = 1.01 * np.sqrt(K) * (2.0 ** -57 + 2.0 ** -58) * np.outer(na, nb) + 2.0 ** -52 * np.abs(ref)
    err = np.abs(q[rows][:, cols].cpu().numpy().astype(np.longdouble) - ref)
    assert (err <= bound).all(), float((err / bound).max())


@pytest.mark.parametrize("layout", ["row", "col", "pitched"])
@pytest.mark.parametrize("m,n,k,p,N", [(2048, 1024, 64, 32, 8), (2049, 1025, 64, 33, 8), (2303, 1151, 59, 10, 15),
                                       (1000, 2000, 64, 16, 32), (700, 8193, 50, 15, 13), (16385, 1024, 17, 7, 8)])
def test_sketch_tile_edges(cuda, layout, m, n, k, p, N):
    g = torch.Generator(device=cuda)
    g.manual_seed(m)
    a = torch.randn(m, n, generator=g, dtype=torch.float64, device=cuda)
    a *= torch.logspace(-60, 60, m, dtype=torch.float64, device=cuda)[:, None]      # every row its own scale
    if layout == "col":
        a = a.t().contiguous().t()
    elif layout == "pitched":
        wide = torch.zeros(m, n + 3, dtype=torch.float64, device=cuda)
        wide[:, 1:n + 1] = a
        a = wide[:, 1:n + 1]
    omega = torch.randn(n, (k + p) * N, generator=g, dtype=torch.float64, device=cuda)
    q, launches = _sketch(a, omega, k, p, N)
    assert launches > 3                       # the DMMA path is one or two launches
    rows = sorted({0, 1, 127, 128, 255, 256, m // 2, m - 2, m - 1} & set(range(m)))
    cols = sorted({0, 31, 32, 127, 128, 255, 256, (k + p) * N - 1} & set(range((k + p) * N)))
    _check(q, a, omega, rows, cols)
    assert torch.allclose(q, a @ omega, rtol=0, atol=float("inf"))                # every element finite
    assert float(((q - a @ omega).norm(dim=1) / (a.norm(dim=1) * omega.norm() + 1e-300)).max()) < 1e-14


def test_rows_and_columns_left_to_the_fp64_units(cuda):
    """NaN, infinities, extreme magnitudes, few large entries: those rows and columns have the FP64 GEMM's values;
    zero rows are zero; the others are as exact as ever."""
    m, n, k, p, N = 2100, 1100, 64, 32, 8
    g = torch.Generator(device=cuda)
    g.manual_seed(5)
    a = torch.randn(m, n, generator=g, dtype=torch.float64, device=cuda)
    omega = torch.randn(n, (k + p) * N, generator=g, dtype=torch.float64, device=cuda)
    a[3, 17] = float("nan")
    a[300, 5] = float("inf")
    a[301] = 0.0
    a[302] *= 1e-200
    a[303] *= 1e200
    a[304] = 0.0
    a[304, 9] = 2.0                            # one entry: the product is exact in FP64
    a[2099, :] = 1e-308 * torch.randn(n, generator=g, dtype=torch.float64, device=cuda)
    omega[:, 500] *= 1e-250
    omega[7, 501] = float("-inf")
    omega[:, 502] = 0.0
    omega[:, 503] = 0.0
    omega[30, 503] = 1.0
    q, _ = _sketch(a, omega, k, p, N)
    ref = a @ omega
    assert torch.equal(torch.isnan(q), torch.isnan(ref))
    fin = torch.isfinite(ref)
    inf = ~fin & ~torch.isnan(ref)
    assert torch.equal(fin, torch.isfinite(q)) and torch.equal(q[inf], ref[inf])
    assert torch.equal(q[304][fin[304]], 2.0 * omega[9][fin[304]])
    assert torch.equal(q[:, 503][fin[:, 503]], a[:, 30][fin[:, 503]])
    assert (q[301][fin[301]] == 0).all() and (q[:, 502][fin[:, 502]] == 0).all()
    for r in (302, 303, 2099):
        ok = fin[r]
        assert float((q[r][ok] - ref[r][ok]).abs().max()) <= 1e-13 * float(ref[r][ok].abs().max())
    rows = [0, 1, 2, 255, 256, 299, 305, 2098]
    cols = [0, 255, 256, 499, 504, 767]
    _check(q, a, omega, rows, cols)


def test_row_blocks_and_power_iteration(cuda):
    """A host matrix streamed in row blocks gives the device-resident solve's bits; the power iteration's transposed
    product takes the path as well."""
    from mcnla_b200 import isvd
    m, n, k, p, N = 9000, 1200, 50, 14, 16
    g = torch.Generator(device=cuda)
    g.manual_seed(8)
    a = torch.randn(m, n, generator=g, dtype=torch.float64, device=cuda)
    a[4097, 3] = 1e9                           # a row for the FP64 units inside one of the blocks
    omega = torch.randn(n, (k + p) * N, generator=g, dtype=torch.float64, device=cuda)
    s, u, v, it = isvd.solve(a, k, p, N, omega=omega, integrator="rb_gramian_kn", former="rb_gramian", maxit=8)
    sh, uh, vh, ith = isvd.solve_host(a.cpu().pin_memory(), omega.cpu().pin_memory(), k, p, N,
                                      integrator="rb_gramian_kn", former="rb_gramian", maxit=8)
    assert it == ith and torch.equal(s.cpu(), sh) and torch.equal(u.cpu(), uh) and torch.equal(v.cpu(), vh)
    q, _ = _sketch(a, omega.clone(), k, p, N, exponent=1)
    ref = a @ (a.T @ (a @ omega))
    assert float((q - ref).norm() / ref.norm()) < 1e-13


def test_gramian(cuda):
    """Bs = Qs' Qs of the Gramian integrator (one set of residues, lower triangle): the same Qbar as the row-block
    form, which makes no Gramian."""
    from mcnla_b200 import isvd
    m, k, p, N = 6001, 50, 15, 16
    g = torch.Generator(device=cuda)
    g.manual_seed(9)
    base = torch.linalg.qr(torch.randn(m, k + p, generator=g, dtype=torch.float64, device=cuda))[0]
    noise = torch.randn(N, m, k + p, generator=g, dtype=torch.float64, device=cuda) / m ** 0.5
    q = torch.linalg.qr(base[None] + 0.3 * noise)[0].permute(1, 0, 2).reshape(m, -1).contiguous()
    prm = isvd.Parameters().setSize(m, m).setRank(k).setOverRank(p).setNumSketch(N).sync()
    out = []
    for cls in (isvd.RowBlockGramianKolmogorovNagumoIntegrator, isvd.RowBlockKolmogorovNagumoIntegrator):
        st = cls(prm, 256, 1e-4)
        st.initialize()
        qbar = prm.createMatrixQbar()
        st(q, qbar)
        out.append((qbar, st.iteration()))
    assert out[0][1] == out[1][1]
    assert float((out[0][0] - out[1][0]).abs().max()) < 1e-12


def _bases(cuda, m, l, N, seed):
    g = torch.Generator(device=cuda)
    g.manual_seed(seed)
    base = torch.linalg.qr(torch.randn(m, l, generator=g, dtype=torch.float64, device=cuda))[0]
    noise = torch.randn(N, m, l, generator=g, dtype=torch.float64, device=cuda) / m ** 0.5
    return torch.linalg.qr(base[None] + 0.3 * noise)[0].permute(1, 0, 2).reshape(m, -1).contiguous()


def _kn(q, l, N, maxit, tol):
    """The Kolmogorov-Nagumo average by its definition, in FP64."""
    qc = q[:, :l].clone()
    for it in range(1, maxit + 1):
        b = q.T @ qc
        x = (q @ b - qc @ (b.T @ b)) / N
        lam, vec = torch.linalg.eigh(x.T @ x)
        e = torch.sqrt(0.5 + torch.sqrt(0.25 - lam))
        qc = qc @ ((vec * e) @ vec.T) + x @ ((vec / e) @ vec.T)
        if not float(torch.linalg.norm(e - 1)) >= tol:
            break
    return qc, it


@pytest.mark.parametrize("cls,m,k,p,N", [
    ("KolmogorovNagumoIntegrator", 8192, 20, 11, 33), ("KolmogorovNagumoIntegrator", 12001, 20, 12, 24),
    ("KolmogorovNagumoIntegrator", 20000, 20, 13, 13), ("RowBlockKolmogorovNagumoIntegrator", 8001, 50, 14, 16),
    ("RowBlockKolmogorovNagumoIntegrator", 8193, 50, 15, 16), ("RowBlockKolmogorovNagumoIntegrator", 20000, 3, 2, 129),
    ("RowBlockKolmogorovNagumoIntegrator", 6000, 128, 32, 10),
    ("RowBlockGramianKolmogorovNagumoIntegrator", 3001, 50, 14, 45),
    ("RowBlockGramianKolmogorovNagumoIntegrator", 3100, 20, 9, 99)])
def test_iteration_products(cuda, cls, m, k, p, N):
    """The loops' products with Qs, Qs' and Bs in int8 slices (csrc/slice_gemm.cu): rows, columns and K around the
    tiles (128, 32 or 64 columns a group, 128 of K, parts of K).  The products are off by about 1e-15 of the bases'
    scale an iteration, as a running FP64 sum is; 1e-12 leaves room for the iterations' growth."""
    from mcnla_b200 import isvd
    l = k + p
    q = _bases(cuda, m, l, N, m + k)
    prm = isvd.Parameters().setSize(m, m).setRank(k).setOverRank(p).setNumSketch(N).sync()
    st = getattr(isvd, cls)(prm, 64, 1e-6)
    st.initialize()
    qbar = prm.createMatrixQbar()
    st(q, qbar)
    ref, it = _kn(q, l, N, 64, 1e-6)
    assert st.iteration() == it
    assert float((qbar - ref).abs().max()) < 1e-12


def test_iteration_products_scales_and_nan(cuda):
    """Rows of very different magnitude keep their relative accuracy (the plain integrator: the row-block ones assume
    orthonormal bases, which the scaled row ends); a NaN in Qs reaches the result and the iteration ends."""
    from mcnla_b200 import isvd
    m, k, p, N = 8192, 50, 14, 16
    l = k + p
    q = _bases(cuda, m, l, N, 3)
    q[100] *= 1e-12
    prm = isvd.Parameters().setSize(m, m).setRank(k).setOverRank(p).setNumSketch(N).sync()
    st = isvd.KolmogorovNagumoIntegrator(prm, 12, 1e-9)
    st.initialize()
    qbar = prm.createMatrixQbar()
    st(q, qbar)
    ref, it = _kn(q, l, N, 12, 1e-9)
    assert st.iteration() == it and float((qbar - ref).abs().max()) < 1e-12
    assert float((qbar[100] - ref[100]).abs().max()) < 1e-12 * float(ref[100].abs().max())
    q[7, 3] = float("nan")
    st(q, qbar)
    assert st.iteration() == 1 and torch.isnan(qbar).any()
