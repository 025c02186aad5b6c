"""FP64 calls whose sliced operands do not fit the device: they take the FP64 pipe, which
needs none of that scratch, and give the same results to FP64 accuracy."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# a process of its own, whose device memory is filled up to `room` bytes by a tensor
CHILD = """
import sys
import numpy as np, torch
import gplite_gb300 as G
what, n, m, room = sys.argv[1], int(sys.argv[2]), int(sys.argv[3]), int(sys.argv[4])
rng = np.random.default_rng(5)
x = rng.uniform(-1, 1, (n, 3))
y = np.sin(3 * x[:, 0]) + 0.2 * rng.standard_normal(n)
xt = rng.uniform(-1, 1, (m, 3))
def call():
    g = G.gp_fit(G.gp_init(G.cf_matern32(lscale=0.5), G.lik_gaussian(sigma=0.2)), x, y)
    if what == "grad": return np.asarray(G.gp_energy_grad(g))
    if what == "loo": return G.gp_loo(g, x, y)["loos"]
    return G.gp_pred(g, xt, var=True)["var"]
if room:
    G.gp_fit(G.gp_init(), x[:20], y[:20])
    free = torch.cuda.mem_get_info()[0]
    ballast = torch.empty(free - room, dtype=torch.uint8, device="cuda")
np.save(sys.argv[5], call())
"""


@pytest.mark.parametrize("what,n,m,room", [
    # K and L (16 n^2 bytes) for the fit; then L, L^-1 and B^-1 (24 n^2), and 16 n^2 for the
    # split L^-1
    ("grad", 6000, 1, 33 * 6000**2),
    # L and L^-1 (16 n^2), and 10 n^2 for the operands of the inverse
    ("loo", 6000, 1, 21 * 6000**2),
    # the n x m cross covariance (8 n m) and the FP64 pipe's 64 x m, and 8192 m for the split one
    ("var", 1000, 200000, 8 * 1000 * 200000 + 4500 * 200000),
])
def test_scratch_that_does_not_fit(tmp_path, what, n, m, room):
    """Condition number of B below 1e5: 64-bit results agree to 1e-10 of their largest."""
    import numpy as np
    res = []
    for r in (0, room):
        out = str(tmp_path / ("%d.npy" % r))
        p = subprocess.run([sys.executable, "-c", CHILD, what, str(n), str(m), str(r), out], cwd=ROOT,
                           capture_output=True, text=True, timeout=240)
        assert p.returncode == 0, p.stderr[-2000:]
        res.append(np.load(out))
    a, b = res
    assert not np.array_equal(a, b)  # (the other path was taken)
    assert np.abs(a - b).max() <= 1e-10 * np.abs(a).max()
