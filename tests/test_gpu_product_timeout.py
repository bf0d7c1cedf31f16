"""Products whose waits run out (the failure hook keeps one CTA's loader silent):
every entry point that synchronises returns TMVG_TIMEOUT and not a result, an
asynchronous product leaves it to the next such call, and the same handle then
works.  No kernel traps or spins without a limit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TIMEOUT = 5
PRODUCT = 2


@pytest.fixture
def silent(dev):
    from tmv_gb300 import linalg

    h = linalg.handle(dev.index or 0)
    yield lambda: h.check(h.call("tmvg_test_set_silent", PRODUCT), "test_set_silent")
    h.check(h.call("tmvg_test_set_silent", 0), "test_set_silent")


@pytest.mark.parametrize("m,n,k", [(300, 300, 300), (1000, 900, 64)])  # 64- and 32-column tiles
def test_asynchronous_product(dev, silent, m, n, k):
    from helpers import to_dev, to_host

    from tmv_gb300 import linalg

    rng = np.random.default_rng(m)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    A, B, X = to_dev(a, dev), to_dev(b, dev), to_dev(np.zeros((m, n)), dev)
    h = linalg.handle(dev.index or 0)
    silent()
    linalg.multmm(False, 1.0, A, B, X)
    assert h.call("tmvg_synchronize") == TIMEOUT
    assert h.call("tmvg_synchronize") == 0
    linalg.multmm(False, 1.0, A, B, X)
    assert h.call("tmvg_synchronize") == 0
    assert (np.abs(to_host(X) - a @ b) <= 2 * k * 2.0 ** -53 * (np.abs(a) @ np.abs(b))).all()


def test_host_product(dev, silent):
    from tmv_gb300 import linalg

    rng = np.random.default_rng(1)
    n = 300
    a, b = (np.asfortranarray(rng.standard_normal((n, n))) for _ in range(2))
    x = np.zeros((n, n), order="F")
    h = linalg.handle(dev.index or 0)

    def product():
        p = [C.c_void_p(v.ctypes.data) for v in (a, b, x)]
        return h.call("tmvg_multmm_f64_host", 0, 1.0, n, n, n, p[0], 1, n, p[1], 1, n, p[2], 1, n)

    silent()
    assert product() == TIMEOUT
    assert product() == 0
    assert (np.abs(x - a @ b) <= 2 * n * 2.0 ** -53 * (np.abs(a) @ np.abs(b))).all()


@pytest.mark.parametrize("what", ["factor", "mixed", "backward", "complex host"])
def test_factorisations(dev, silent, what):
    import torch
    from helpers import to_dev

    from tmv_gb300 import TmvgError, linalg

    rng = np.random.default_rng(2)
    n = 1100
    a = rng.standard_normal((n, n)) + 4.0 * np.sqrt(n) * np.eye(n)
    A, B = to_dev(a, dev), to_dev(rng.standard_normal((n, 64)), dev)
    h = linalg.handle(dev.index or 0)
    if what == "factor":
        run = lambda: linalg.lu_decompose(A.t().clone().t())  # noqa: E731
    elif what == "mixed":  # the FP32 factorisation's streamed update
        run = lambda: linalg.solve_mixed(A, B[:, :1].t().clone().t())  # noqa: E731
    elif what == "backward":  # gA = -gB X^T after the solve
        X, LU, P = linalg.divide(A, B)
        G, gA = B.t().clone().t(), torch.empty_like(A)
        p = [C.c_void_p(t.data_ptr()) for t in (LU, P, X, G, gA)]
        run = lambda: h.check(h.call("tmvg_lu_solve_bwd_f64", n, p[0], n, p[1], 64, p[2], n, p[3], n,  # noqa: E731
                                     None, n, p[4], n))
    else:
        z = np.asfortranarray(a + 1j * rng.standard_normal((n, n)))
        piv = np.zeros(n, np.int64)

        def run():
            w = z.copy("F")
            h.check(h.call("tmvg_lu_decompose_z64_host", n, C.c_void_p(w.ctypes.data), 1, n,
                           C.c_void_p(piv.ctypes.data)))

    silent()
    with pytest.raises(TmvgError) as ei:
        run()
    assert ei.value.status == TIMEOUT
    run()
    assert h.call("tmvg_synchronize") == 0
