"""FITC's substitution with the rows of a matrix, whose products run on the tensor cores from 1024
rows and 16 M multiply-adds on: its residual, which no condition number enters, for the factor
of a smooth kernel."""
import numpy as np
import pytest

from gplite_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def sexp(a, b, lscale):
    return np.exp(-((a[:, None] - b[None]) ** 2).sum(2) / (2 * lscale**2))


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n,M", [(3, 1), (40, 8), (17, 9), (40, 16), (33, 17), (50, 32), (1100, 33), (70, 63), (40, 200),
                                 (1023, 65), (1024, 64), (1024, 65), (1500, 100), (2047, 192), (2048, 192), (2049, 257),
                                 (4500, 200)])
def test_residual_of_a_smooth_kernels_factor(n, M, mode):
    """X L^T = B (mode 1: X L = B) for the factor L of a squared exponential's K_z, singular up
    to its jitter of 1e-6, where inverses of diagonal blocks would lose digits. Substitution is
    backward stable: a row's residual is at most (M + 3) 2^-53 (|X| |L|^T), with one more
    rounding each for the reciprocal of a pivot and the sum over blocks of 64 columns; the sliced
    products add at most 9 K 2^-64 + 2^-63 of the product of their rows' powers of two
    (K = 64 in each of M / 64 of them; twice the largest entries)."""
    rng = np.random.default_rng(n + M)
    z = rng.uniform(-1, 1, (M, 2))
    x = rng.uniform(-1, 1, (n, 2))
    F = np.linalg.cholesky(sexp(z, z, 1.0) + 1e-6 * np.eye(M))
    B = np.asfortranarray(sexp(x, z, 1.0))
    X = np.empty_like(B, order="F")
    ctx = L.default_context(0)
    L.check(L.load().gpgp_tri_rows_selftest(ctx.h, n, M, L.ptr(np.asfortranarray(F)), L.ptr(B), mode, L.ptr(X)), ctx.h)
    T = F.T if mode == 0 else F
    # the residual in long double
    R = np.zeros((n, M), dtype=np.longdouble)
    Xl, Tl = X.astype(np.longdouble), T.astype(np.longdouble)
    for k in range(M):
        R += np.outer(Xl[:, k], Tl[k])
    R -= B
    bound = (M + 3 + 2 + M // 64) * 2.0**-53 * (np.abs(X) @ np.abs(T))
    bound += (M / 64 + 1) * (9 * 64 * 2.0**-64 + 2.0**-63) * 4 * np.outer(np.abs(X).max(1), np.abs(T).max(0))
    assert (np.abs(R) <= bound).all(), float((np.abs(R) / bound).max())
