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
