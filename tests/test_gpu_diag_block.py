"""The diagonal-block kernel (factor and inverse of up to 64 x 64, in segments of 4
columns, 16 to a CTA)."""
import numpy as np
import pytest

import gplite_gb300 as G
from oracle import gplite_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 79, 81])
def test_partial_blocks_and_panel_edges(n):
    """One block (and its neighbour) at every panel edge, on a smooth kernel with little
    noise: B's condition number is about n / sigma^2 = 64e4, so 64-bit results agree to
    ~1e-16 x 1e6 = 1e-10 of their largest entry; the evidence (a sum of logarithms and a
    quadratic form that the same factor decides) to 1e-10."""
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, 2))
    y = np.sin(3 * x[:, 0]) + 0.01 * rng.standard_normal(n)
    xt = rng.uniform(-1, 1, (9, 2))
    g = G.gp_fit(G.gp_init(G.cf_sexp(lscale=0.8), G.lik_gaussian(sigma=0.01)), x, y)
    o = R.gp_fit(R.gp_init([R.cf("sexp", lscale=0.8, magn=1.0)], R.lik("gaussian", sigma=0.01)), x, y)
    assert abs(g.fit["log_evidence"] - o.fit["log_evidence"]) <= 1e-10 * max(abs(o.fit["log_evidence"]), n)
    a, b = G.model_field(g, "alpha"), o.fit["alpha"]
    assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max()
    p, q = G.gp_pred(g, xt, var=True), R.gp_pred(o, xt, var=True)
    assert np.allclose(p["mean"], q["mean"], rtol=0, atol=1e-10)
    assert np.allclose(p["var"], q["var"], rtol=0, atol=1e-10)
