"""The FP64-accurate sliced product (8 slices of 8 bits on the tensor cores) and the
FP64 path of large n that is built on it."""
import ctypes as C

import numpy as np
import pytest

import gplite_gb300 as G
from gplite_gb300 import _lib as L
from oracle import gplite_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(33, 1, 1), (64, 64, 16), (127, 65, 15), (128, 64, 256), (129, 191, 257),
                                   (300, 200, 272), (1000, 700, 130), (640, 640, 2049)])
def test_sliced_product_is_as_accurate_as_fp64(M, N, K):
    """-A B^T + C against the FP64 GEMM. The self-test's entries are at most 8 in
    magnitude (|u| <= 1/2 times 2^(-4..4)): the slices drop at most 2^-63 of a row's
    power of two (at most 8) per entry and the levels beyond the kept ones 2^-59 of the
    product of both; the FP64 sums round at K 2^-53 of theirs, and the largest |C| is
    at least 1/4 (C starts uniform in [-1/2, 1/2], here of an M, N where that holds)."""
    err = C.c_double(-1.0)
    ctx = L.default_context(0)
    L.check(L.load().gpgp_mixed_selftest(ctx.h, M, N, K, 8, C.byref(err)), ctx.h)
    assert 0.0 <= err.value <= 64.0 * K * (2.0 ** -58 + 2.0 ** -53) / 0.25


@pytest.mark.parametrize("n", [895, 896, 897, 959, 960, 961, 1024, 1153, 1600])
def test_fp64_fit_either_side_of_the_sliced_sizes(n):
    """Evidence, gradient and predictions around the size where the factorisation's
    products move to the tensor cores, at the FP64 path's tolerance."""
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, 3))
    y = np.sin(3 * x[:, 0]) + x[:, 1] + 0.1 * rng.standard_normal(n)
    xt = rng.uniform(-1, 1, (65, 3))
    g = G.gp_fit(G.gp_init([G.cf_matern52(lscale=0.6), G.cf_const(1.0)], G.lik_gaussian(sigma=0.1)), x, y, grad=True)
    o = R.gp_fit(R.gp_init([R.cf("matern52", lscale=0.6, magn=1.0), R.cf("const", magn=1.0)],
                           R.lik("gaussian", sigma=0.1)), x, y)
    assert abs(g.fit["log_evidence"] - o.fit["log_evidence"]) <= 1e-10 * abs(o.fit["log_evidence"])
    ref = R.gp_energy_grad(o)
    assert np.allclose(G.gp_energy_grad(g), ref, rtol=1e-10, atol=1e-10 * np.abs(ref).max())
    p, q = G.gp_pred(g, xt, var=True), R.gp_pred(o, xt, var=True)
    assert np.allclose(p["mean"], q["mean"], rtol=1e-10, atol=1e-10)
    assert np.allclose(p["var"], q["var"], rtol=1e-9, atol=1e-11)


@pytest.mark.parametrize("n", [700, 1100])
def test_a_nan_entry_of_the_matrix_is_refused(n):
    """Inputs so far apart that a squared distance overflows make the Matern kernel NaN
    off the diagonal: the factorisation refuses the matrix on either path."""
    rng = np.random.default_rng(3)
    x = rng.uniform(-1, 1, (n, 1))
    x[n // 2] = 1e200
    with pytest.raises((L.GpgpError, np.linalg.LinAlgError)):
        G.gp_fit(G.gp_init(G.cf_matern52(lscale=0.5), G.lik_gaussian(sigma=0.1)), x, rng.standard_normal(n))


@pytest.mark.parametrize("n,M", [(1023, 65), (1024, 64), (4095, 33), (4096, 128), (4353, 63), (9001, 129), (8500, 1)])
def test_fitc_either_side_of_the_sliced_sizes(n, M):
    """FITC fits and predictions around the row counts where the Gram products and the
    substitution's products move to the tensor cores, at inducing counts around the
    block sizes. The Matern 3/2 kernel at scattered inducing inputs keeps K_z's condition
    number below ~1e4, so 64-bit sums of up to 1e4 terms agree to ~1e-10; 1e-9 here."""
    rng = np.random.default_rng(n + M)
    x = rng.uniform(-2, 2, (n, 2))
    y = np.sin(2 * x[:, 0]) * np.cos(x[:, 1]) + 0.1 * rng.standard_normal(n)
    z = x[rng.choice(n, M, replace=False)]
    xt = rng.uniform(-2, 2, (70, 2))
    g = G.gp_fit(G.gp_init(G.cf_matern32(lscale=0.3), G.lik_gaussian(sigma=0.2), G.method_fitc(inducing=z)), x, y)
    o = R.gp_fit(R.gp_init([R.cf("matern32", lscale=0.3, magn=1.0)], R.lik("gaussian", sigma=0.2),
                           R.method_fitc(z)), x, y)
    assert abs(g.fit["log_evidence"] - o.fit["log_evidence"]) <= 1e-9 * abs(o.fit["log_evidence"])
    p, q = G.gp_pred(g, xt, var=True), R.gp_pred(o, xt, var=True)
    assert np.allclose(p["mean"], q["mean"], rtol=1e-9, atol=1e-9)
    assert np.allclose(p["var"], q["var"], rtol=1e-8, atol=1e-9)
    if n < 5000:
        assert np.allclose(G.gp_loo(g, x, y)["loos"], R.gp_loo(o, x, y)["loos"], rtol=1e-8, atol=1e-8)


@pytest.mark.parametrize("n,m", [(900, 704), (900, 769), (1500, 448), (1500, 449), (4600, 129)])
def test_variance_either_side_of_the_sliced_solve(n, m):
    """The variance's solve moves to the tensor cores at 180 tiles of 64 x 64 (condition number of
    B below 1e4: 1e-10)."""
    rng = np.random.default_rng(n + m)
    x = rng.uniform(-1, 1, (n, 3))
    y = np.sin(3 * x[:, 0]) + 0.2 * rng.standard_normal(n)
    xt = rng.uniform(-1, 1, (m, 3))
    g = G.gp_fit(G.gp_init(G.cf_matern32(lscale=0.5), G.lik_gaussian(sigma=0.2)), x, y)
    o = R.gp_fit(R.gp_init([R.cf("matern32", lscale=0.5, magn=1.0)], R.lik("gaussian", sigma=0.2)), x, y)
    p, q = G.gp_pred(g, xt, var=True), R.gp_pred(o, xt, var=True)
    assert np.abs(p["mean"] - q["mean"]).max() <= 1e-10
    assert np.abs(p["var"] - q["var"]).max() <= 1e-10


def test_few_predictions_take_few_launches():
    """The sliced solve takes at least five launches for each 64 rows, which few right-hand sides
    do not repay; the FP64 pipe's two."""
    rng = np.random.default_rng(2)
    x = rng.uniform(-1, 1, (1500, 2))
    g = G.gp_fit(G.gp_init(G.cf_sexp(lscale=0.5), G.lik_gaussian(sigma=0.2)), x, np.sin(3 * x[:, 0]))
    for m in (1, 300):
        before = L.launch_count()
        G.gp_pred(g, x[:m], var=True)
        assert L.launch_count() - before <= 3 * 24
