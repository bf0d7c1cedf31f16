"""A panel whose CTAs wait in vain for one of them (the failure hook keeps its
last CTA silent): the call returns TMVG_TIMEOUT, the interchanges it leaves are
valid row numbers (the kernels that follow use them as such), and the same handle
then factors correctly.  No kernel traps or spins without a limit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TIMEOUT = 5


@pytest.mark.parametrize("reg2", [False, True])
@pytest.mark.parametrize("n", [200, 1100, 1500])
def test_silent_cta_of_the_real_panel(dev, n, reg2, monkeypatch):
    import torch
    from helpers import to_dev

    from tmv_gb300 import _lib

    if reg2:
        if n <= 512:
            pytest.skip("one CTA")
        monkeypatch.setenv("TMVG_PANEL_REG2", "1")
    h = _lib.Handle(dev.index or 0)
    h.set_stream(torch.cuda.current_stream().cuda_stream)
    a = np.random.default_rng(n).standard_normal((n, n))

    def factor(A, P):
        return h.call("tmvg_lu_decompose_f64", n, C.c_void_p(A.data_ptr()), n, C.c_void_p(P.data_ptr()))

    A = to_dev(a, dev, "F")
    P = torch.full((n,), -(2 ** 40), dtype=torch.int64, device=dev)
    h.check(h.call("tmvg_test_set_silent", 1), "test_set_silent")
    st = factor(A, P)
    msg = h.lib.tmvg_last_error(h.h)
    assert st == TIMEOUT and b"timed out" in msg
    p = P.cpu().numpy()
    assert ((p >= np.arange(n)) & (p < n)).all()
    A = to_dev(a, dev, "F")
    assert factor(A, P) == 0
    lu = A.cpu().numpy()
    for i, q in enumerate(P.cpu().numpy()):
        a[[i, q]] = a[[q, i]]
    low, up = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    assert np.abs(low).max() <= 1.0
    assert (np.abs(low @ up - a) <= 2 * n * 2.0 ** -53 * (np.abs(low) @ np.abs(up))).all()


def test_silent_cta_of_the_mixed_solve(dev):
    from helpers import to_dev, to_host

    from tmv_gb300 import TmvgError, linalg

    rng = np.random.default_rng(3)
    n = 1024
    a, b = rng.standard_normal((n, n)) + 4.0 * np.sqrt(n) * np.eye(n), rng.standard_normal((n, 1))
    A, B = to_dev(a, dev, "F"), to_dev(b, dev, "F")
    h = linalg.handle(dev.index or 0)
    h.check(h.call("tmvg_test_set_silent", 1), "test_set_silent")
    try:
        with pytest.raises(TmvgError) as ei:
            linalg.solve_mixed(A, B)
    finally:
        h.check(h.call("tmvg_test_set_silent", 0), "test_set_silent")
    assert ei.value.status == TIMEOUT
    X, info = linalg.solve_mixed(A, B)
    assert info.converged == 1
    x = to_host(X)
    assert np.abs(a @ x - b).max() <= 1e-12 * (np.abs(a).sum(axis=1).max() * np.abs(x).max())


def test_hook_rejects_unknown_parts(dev):
    from tmv_gb300 import linalg

    assert linalg.handle(dev.index or 0).call("tmvg_test_set_silent", -1) == 3
