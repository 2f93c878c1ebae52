"""CPU checks that the admission estimate covers what a problem's stages allocate (mcnla_b200_problem_bytes, host only)."""
import ctypes

from mcnla_b200 import _lib


def _bytes(m, n, k, p, N, integrator, maxit=256):
    pr = _lib.Problem()
    pr.params = _lib.Params(m, n, k, p, N)
    pr.A = ctypes.c_void_p(0x1000)                        # only its presence is read
    pr.integrator = integrator
    pr.max_iteration = maxit
    pr.precision = _lib.PRECISION_FP64
    return _lib.load().mcnla_b200_problem_bytes(ctypes.byref(pr))


def test_slices_of_the_loops_counted():
    m, n, k, p, N = 65536, 2048, 48, 16, 32
    l, L = k + p, (k + p) * N
    for integrator in (_lib.KOLMOGOROV_NAGUMO, _lib.ROW_BLOCK_KOLMOGOROV_NAGUMO):
        # Q, Qbar and Omega, the loop's state and 7 bytes an element of Qs in each layout
        need = (m * L + m * l + n * L) * 8 + 2 * m * 2 * l * 8 + 14 * m * L
        assert _bytes(m, n, k, p, N, integrator) >= need
        # a handful of iterations takes none
        assert _bytes(m, n, k, p, N, integrator, maxit=7) < need
