"""What the eight-slice product keeps: its error against the exact product, in units of the two
rows' scales, with entries spread over 2^40 within a row and sums that cancel (elsewhere the
rounding of the result, 2^-53 of it, would hide the slices)."""
from fractions import Fraction

import numpy as np
import pytest

from gplite_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def sliced(A, B, slices=8):
    A, B = np.asfortranarray(A), np.asfortranarray(B)
    C = np.empty((A.shape[0], B.shape[0]), order="F")
    ctx = L.default_context(0)
    L.check(L.load().gpgp_sliced_product_selftest(ctx.h, A.shape[0], B.shape[0], A.shape[1], slices, L.ptr(A), L.ptr(B),
                                                  L.ptr(C)), ctx.h)
    return C


UNIT = 260  # fixed point of the exact sums: 2^-260 a unit, which every double here is a multiple of


def as_ints(A):
    """Doubles as integers in units of 2^-UNIT."""
    m, e = np.frexp(A)
    k = (m * 2.0**53).astype(np.int64)
    return np.array([[int(a) << int(s) if s >= 0 else int(a) >> -int(s) for a, s in zip(ra, rs)]
                     for ra, rs in zip(k, e - 53 + UNIT)], dtype=object)


def error(A, B, C):
    """(C - A B^T) / (2^e_i 2^f_j) for rows of largest entry 0.5 .. 1 times those powers, and the same of
    A B^T, from exact integer sums."""
    P = as_ints(A).dot(as_ints(B).T)  # units of 2^-2 UNIT
    D = np.array([[int(c) for c in r] for r in as_ints(C)], dtype=object) * (1 << UNIT) - P
    ea, eb = (np.frexp(np.abs(x).max(1))[1] for x in (A, B))
    scale = np.ldexp(1.0, -(ea[:, None] + eb[None, :]))
    f = lambda X: np.array([[float(Fraction(v, 1 << 2 * UNIT)) for v in r] for r in X]) * scale  # noqa: E731
    return f(D), f(P)


@pytest.mark.parametrize("spread", [0, 12, 40])
@pytest.mark.parametrize("K", [2, 16, 130, 256, 514, 1026])
def test_error_of_the_kept_levels(K, spread):
    """An entry is held to 2^-64 of its row's power of two and the products of levels 8 and on are
    dropped: seven pairs of digits of at most 128 at 2^-78, of random sign. Both together
    have a standard deviation below 2^-63.5 a term; each exactly summed group of 256 K adds at most
    2^-63 (its deepest level, rounded to a unit of the level before). Eight standard deviations, and
    the result's own rounding."""
    rng = np.random.default_rng(1000 * K + spread)
    M, N, h = 21, 19, K // 2

    def entries(r):
        return rng.uniform(0.5, 1, (r, h)) * np.ldexp(1.0, -rng.integers(0, spread + 1, (r, h))) * rng.choice(
            [-1.0, 1.0], (r, h))
    a, b = entries(M), entries(N)
    A = np.concatenate([a, a], 1)
    B = np.concatenate([b, -b * (1 + 2.0**-42 * rng.uniform(-1, 1, (N, h)))], 1)
    err, P = error(A, B, sliced(A, B))
    bound = (8 * np.sqrt(K) + -(-K // 256)) * 2.0**-63 + 2.0**-53 * np.abs(P)
    assert (np.abs(err) <= bound).all(), float((np.abs(err) / bound).max())
