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


# the default memory pool's high-water mark after a fit with random features
CHILD_HIGH = """
import ctypes as C, sys
import numpy as np
import gplite_gb300 as G
n, D = int(sys.argv[1]), int(sys.argv[2])
rng = np.random.default_rng(5)
x = rng.uniform(-1, 1, (n, 2))
y = np.sin(3 * x[:, 0]) + 0.2 * rng.standard_normal(n)
G.gp_fit(G.gp_init(G.cf_sexp(lscale=0.5), G.lik_gaussian(sigma=0.2), G.method_rf(num_basis=D)), x, y)
cu, pool, high = C.CDLL("libcuda.so.1"), C.c_void_p(), C.c_uint64()
assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
assert cu.cuMemPoolGetAttribute(pool, 8, C.byref(high)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_HIGH
print(high.value)
"""


def test_gram_partials_do_not_grow_with_n():
    """A Gram product of n rows and D columns cuts n into ranges, 19 here. Their D x D partials
    are added as they fill their slots (128 MB, one partial here), not kept: beside two n x D
    matrices, eight D x D ones and the split operands (2 x 128 MB, and a margin) nothing grows."""
    n, D = 32768, 4096
    p = subprocess.run([sys.executable, "-c", CHILD_HIGH, str(n), str(D)], cwd=ROOT, capture_output=True, text=True,
                       timeout=240)
    assert p.returncode == 0, p.stderr[-2000:]
    assert int(p.stdout) <= 8 * (2 * n * D + 8 * D * D) + (3 << 27)


@pytest.mark.parametrize("n,D", [(16384, 2048), (20000, 2048), (23041, 2000)])
def test_gram_of_more_ranges_than_slots(n, D):
    """Five ranges and more of 3840 rows, four or five slots: the sums go on over the flushes. The
    evidence's terms are sums of n, as in the random features' tests."""
    import numpy as np

    import gplite_gb300 as G
    from helpers import oracle_gp
    from oracle import gplite_ref as R
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, 2))
    y = np.sin(3 * x[:, 0]) + 0.3 * rng.standard_normal(n)
    g = G.gp_init(G.cf_sexp(lscale=0.5), G.lik_gaussian(sigma=0.3), G.method_rf(num_basis=D))
    o = R.gp_fit(oracle_gp(g), x, y)
    g = G.gp_fit(g, x, y)
    assert abs(g.fit["log_evidence"] - o.fit["log_evidence"]) <= 1e-10 * max(abs(o.fit["log_evidence"]), n)
    a, b = G.model_field(g, "fmean"), o.fit["fmean"]
    assert np.abs(a - b).max() <= 1e-9 * np.abs(b).max()
