"""The outer panels of the sliced Cholesky: the kernel of a panel's rows below it, and the
chain of its diagonal blocks, at ragged last panels, last blocks and last row tiles."""
import numpy as np
import pytest

import gplite_gb300 as G
from oracle import gplite_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,rtol", [("fp64", 1e-10), ("mixed", 1e-6)])
@pytest.mark.parametrize("n", [385, 448, 768, 769, 833, 1025, 1151, 1152, 1153, 1217, 1281, 1409])
def test_panel_edges(n, precision, rtol):
    """Outer panels are 384 columns of 64-wide blocks, row tiles 128: sizes at and beside
    their multiples. B = I + K / 0.04 has a condition number of about n / 0.04 / 10 < 1e4:
    64-bit results agree to 1e4 2^-53 n^(1/2) < 1e-10; four slices (32 bits below a row's
    largest entry, sums of up to n terms of random sign) to 1e4 2^-32 < 1e-5 of the
    smallest eigenvalue's share and 1e-6 of the largest entries, as compared here."""
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, 3))
    y = np.sin(3 * x[:, 0]) + x[:, 1] + 0.2 * rng.standard_normal(n)
    xt = rng.uniform(-1, 1, (33, 3))
    g = G.gp_fit(G.gp_init(G.cf_matern32(lscale=0.5), G.lik_gaussian(sigma=0.2)), x, y, precision=precision)
    o = R.gp_fit(R.gp_init([R.cf("matern32", lscale=0.5, magn=1.0)], R.lik("gaussian", sigma=0.2)), x, y)
    assert abs(g.fit["log_evidence"] - o.fit["log_evidence"]) <= rtol * n
    a, b = G.model_field(g, "alpha"), o.fit["alpha"]
    assert np.abs(a - b).max() <= rtol * np.abs(b).max()
    p, q = G.gp_pred(g, xt, var=True), R.gp_pred(o, xt, var=True)
    assert np.abs(p["mean"] - q["mean"]).max() <= rtol
    assert np.abs(p["var"] - q["var"]).max() <= rtol


@pytest.mark.parametrize("n,m", [(31, 1), (33, 5), (65, 64), (97, 3), (130, 63), (193, 65), (257, 129), (320, 7)])
def test_small_product_edges(n, m):
    """Products of few elements with K up to 256 (32 x 4 elements to a CTA, K in chunks of
    64): the trailing updates of a fit, FITC's and the predictions' products at sizes around
    those. Condition number below 1e4 as above: 1e-10."""
    rng = np.random.default_rng(n + m)
    x = rng.uniform(-1, 1, (n, 2))
    y = np.sin(3 * x[:, 0]) + 0.2 * rng.standard_normal(n)
    xt = rng.uniform(-1, 1, (m, 2))
    z = x[rng.choice(n, min(n - 1, m + 8), replace=False)]
    for gm, om in ((None, None), (G.method_fitc(inducing=z), R.method_fitc(z))):
        g = G.gp_fit(G.gp_init(G.cf_matern32(lscale=0.3), G.lik_gaussian(sigma=0.2), *([gm] if gm else [])), x, y)
        o = R.gp_fit(R.gp_init([R.cf("matern32", lscale=0.3, magn=1.0)], R.lik("gaussian", sigma=0.2),
                               *([om] if om else [])), x, y)
        assert abs(g.fit["log_evidence"] - o.fit["log_evidence"]) <= 1e-10 * n
        p, q = G.gp_pred(g, xt, var=True), R.gp_pred(o, xt, var=True)
        assert np.abs(p["mean"] - q["mean"]).max() <= 1e-10
        assert np.abs(p["var"] - q["var"]).max() <= 1e-10
