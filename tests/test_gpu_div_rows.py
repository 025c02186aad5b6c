"""FITC's row scaling X / v by reciprocals with a residual correction against the division."""
import numpy as np
import pytest

from gplite_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def div_rows(X, v):
    X, v = np.asfortranarray(X, dtype=np.float64), np.ascontiguousarray(v, dtype=np.float64)
    out = np.empty_like(X, order="F")
    ctx = L.default_context(0)
    L.check(L.load().gpgp_div_rows_selftest(ctx.h, X.shape[0], X.shape[1], L.ptr(X), L.ptr(v), L.ptr(out)), ctx.h)
    return out


@pytest.mark.parametrize("spread", [1, 30, 300, 1000])
def test_quotients_are_the_division(spread):
    """The corrected quotient is x / d (1 + 2^-104), rounded once: it can differ from the
    division only where x / d lies within 2^-50 ulp of a midpoint of two doubles, which no one
    of 10^6 random quotients does (probability 10^-9). Mantissas at the ends of the binade and
    exponents up to +-`spread`, so that both paths and their border are taken."""
    rng = np.random.default_rng(spread)
    n, M = 4000, 256
    man = lambda *s: np.where(rng.uniform(size=s) < 0.2, 2.0 - rng.integers(1, 9, s) * 2.0**-52,  # noqa: E731
                              rng.uniform(1, 2, s))
    X = np.ldexp(man(n, M), rng.integers(-spread, spread + 1, (n, M))) * rng.choice([-1.0, 1.0], (n, M))
    v = np.ldexp(man(n), rng.integers(-spread, spread + 1, n)) * rng.choice([-1.0, 1.0], n)
    with np.errstate(all="ignore"):
        want = X / v[:, None]
    np.testing.assert_array_equal(div_rows(X, v), want)


def test_special_values_are_the_division():
    """Zeros of either sign, infinities, NaN, subnormal and extreme operands."""
    s = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -2e-310, 2.0**-1022, 2.0**1023 * 1.9, 1.0, -3.0, 2.0**-900,
                  2.0**900, 2.0**-958, 2.0**960, 2.0**-895, 2.0**961])
    X = np.tile(s, (len(s), 1))
    with np.errstate(all="ignore"):
        want = X / s[:, None]
    got = div_rows(X, s)
    np.testing.assert_array_equal(got, want)
    z = want == 0
    np.testing.assert_array_equal(np.signbit(got[z]), np.signbit(want[z]))
