"""Waits that run out inside the kernels: every kernel that waits for another part of
itself gives up after a bounded number of polls, lets what it has issued land, frees its
tensor memory and reports; the call returns GPGP_ETIMEOUT and the context stays usable."""
import contextlib
import ctypes as C

import numpy as np
import pytest

import gplite_gb300 as G
from gplite_gb300 import _lib as L
from gplite_gb300.batch import gp_fit_batched

pytestmark = pytest.mark.gpu

GEMM, DIAG, PANEL, FLOW = 0, 1, 2, 3


@contextlib.contextmanager
def bound(kernel, polls, chunks=-1):
    """Shorter waits for the launches of this thread (gpgp_wait_bound)."""
    lib = L.load()
    assert lib.gpgp_wait_bound(kernel, polls, chunks) == 0
    try:
        yield
    finally:
        assert lib.gpgp_wait_bound(kernel, -1, -1) == 0


def product(M, N, K, slices):
    ctx = L.default_context(0)
    err = C.c_double(-1.0)
    return L.load().gpgp_mixed_selftest(ctx.h, M, N, K, slices, C.byref(err)), err.value


@pytest.mark.parametrize("slices", [4, 5, 8])
@pytest.mark.parametrize("polls,chunks", [(0, -1), (64, 0), (1, 1), (64, 1), (2000, 3), (64, 5), (3, 17)])
def test_gemm_gives_up_and_recovers(slices, polls, chunks):
    """The producer falls silent after some K chunks of each tile (19 or 38 here), with
    products already issued, or no wait may poll at all."""
    with bound(GEMM, polls, chunks):
        status, _ = product(300, 200, 600, slices)
    assert status == L.ETIMEOUT
    status, err = product(300, 200, 600, slices)
    assert status == 0 and err < 2e-9


def fit(n, precision, kind="full"):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, 2))
    y = np.sin(3 * x[:, 0]) + 0.1 * rng.standard_normal(n)
    if kind == "ep":
        gp = G.gp_init(G.cf_sexp(lscale=0.5), G.lik_bernoulli(), approx=G.approx_ep())
        return G.gp_fit(gp, x, (y > 0).astype(float), precision=precision)
    method = [G.method_fitc(inducing=x[:20])] if kind == "fitc" else []
    return G.gp_fit(G.gp_init(G.cf_matern32(lscale=0.5), G.lik_gaussian(sigma=0.1), *method), x, y,
                    precision=precision)


def gives_up_and_recovers(kernel, n, precision, kind="full"):
    """No wait may poll at all: the call reports the wait, not what it left behind."""
    ref = fit(n, precision, kind).fit["log_evidence"]
    with bound(kernel, 0):
        with pytest.raises(L.GpgpError) as e:
            fit(n, precision, kind)
    assert e.value.status == L.ETIMEOUT
    assert fit(n, precision, kind).fit["log_evidence"] == ref


@pytest.mark.parametrize("n,precision,kind", [(17, "fp64", "full"), (64, "mixed", "full"), (200, "fp64", "full"),
                                              (1000, "fp64", "full"), (900, "mixed", "full"), (90, "fp64", "ep"),
                                              (120, "fp64", "fitc")])
def test_diagonal_block_gives_up_and_recovers(n, precision, kind):
    """A wait of the diagonal block's cluster that runs out is no verdict on the matrix: not
    'not positive definite', and no fit in the other precision."""
    gives_up_and_recovers(DIAG, n, precision, kind)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batched_diagonal_block_gives_up_and_recovers(precision):
    rng = np.random.default_rng(1)
    probs = [dict(x=x, y=np.sin(x[:, 0]), xt=x[:2], lscale=0.5, sigma=0.1)
             for x in (rng.uniform(-1, 1, (n, 2)) for n in (30, 70, 150))]
    with bound(DIAG, 0):
        with pytest.raises(L.GpgpError) as e:
            gp_fit_batched(probs, precision=precision)
    assert e.value.status == L.ETIMEOUT
    assert all(np.isfinite(r["log_evidence"]) for r in gp_fit_batched(probs, precision=precision))


@pytest.mark.parametrize("n,precision", [(500, "mixed"), (1000, "fp64"), (1700, "mixed"), (1700, "fp64")])
def test_panel_gives_up_and_recovers(n, precision):
    """The rows below a panel stop waiting for their products while these still run (one CTA
    and a cluster of CTAs to a row tile): the products land before their memory is freed."""
    gives_up_and_recovers(PANEL, n, precision)


@pytest.mark.parametrize("n", [577, 850, 3000])
def test_triangular_solve_gives_up_and_recovers(n):
    """Blocks of the solution that are not there at the first look (n > 512: many CTAs)."""
    gives_up_and_recovers(FLOW, n, "fp64")
