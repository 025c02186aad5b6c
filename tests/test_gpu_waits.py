"""Waits that run out inside the kernels: every kernel that waits for another part of
itself gives up after a bounded number of polls, lets what it has issued land, frees its
tensor memory and reports; the call returns GPGP_ETIMEOUT and the context stays usable."""
import contextlib
import ctypes as C

import pytest

from gplite_gb300 import _lib as L

pytestmark = pytest.mark.gpu

GEMM = 0


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
