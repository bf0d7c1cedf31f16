"""Calls whose faster form needs buffers of its own, on a handle that cannot grow
them (tmvg_test_refuse_memory): they run in the form that needs none.

Bounds are those of the elimination and substitution themselves, n 2^-53 times
the moduli's products (4 times that for complex entries), doubled for the
reference."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WORK, PANEL, INV, WORDS, POOL = 1, 2, 4, 8, 16
U = 2.0 ** -53


class _Handle:
    """A new handle without the buffers named, and its calls by device pointers."""

    def __init__(self, dev, refuse):
        import torch

        from tmv_gb300 import _lib

        self.h = _lib.Handle(dev.index or 0)
        self.h.set_stream(torch.cuda.current_stream().cuda_stream)
        self.h.check(self.h.call("tmvg_test_refuse_memory", refuse), "refuse")

    def __call__(self, name, *args):
        ptr = [C.c_void_p(a.data_ptr()) if hasattr(a, "data_ptr") else a for a in args]
        self.h.check(self.h.call(name, *ptr), name)


def _dev(a, dev):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a.T)).to(dev).t()


def _factors(rng, n, z=False):
    """Unit lower and upper triangles as partial pivoting leaves them, packed."""
    lu = rng.uniform(-0.5, 0.5, (n, n)) + (1j * rng.uniform(-0.5, 0.5, (n, n)) if z else 0) + 4.0 * np.eye(n)
    return lu, np.tril(lu, -1) + np.eye(n), np.triu(lu)


@pytest.mark.parametrize("n", [40, 700, 1500])
def test_factorisation_without_scratch_panels(dev, n):
    import torch

    a = np.random.default_rng(n).standard_normal((n, n))
    A, P = _dev(a, dev), torch.empty(n, dtype=torch.int64, device=dev)
    _Handle(dev, PANEL)("tmvg_lu_decompose_f64", n, A, n, P)
    lu = A.cpu().numpy()
    for i, q in enumerate(P.cpu().numpy()):
        a[[i, q]] = a[[q, i]]
    low, up = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    assert np.abs(low).max() <= 1.0
    assert (np.abs(low @ up - a) <= 2 * n * U * (np.abs(low) @ np.abs(up))).all()


@pytest.mark.parametrize("refuse", [INV, WORDS])
@pytest.mark.parametrize("upper", [0, 1])
@pytest.mark.parametrize("nrhs", [1, 3, 20, 200])
def test_triangular_solve(dev, refuse, upper, nrhs):
    n = 300
    rng = np.random.default_rng(nrhs)
    t = rng.uniform(-0.5, 0.5, (n, n))
    t = (np.triu(t, 1) if upper else np.tril(t, -1)) + np.diag(3.0 + rng.random(n))
    b = rng.standard_normal((n, nrhs))
    T, B = _dev(t, dev), _dev(b, dev)
    _Handle(dev, refuse)("tmvg_tri_ldiveq_f64", upper, 0, n, T, 1, n, nrhs, B, 1, n)
    x = B.cpu().numpy()
    assert (np.abs(t @ x - b) <= 2 * n * U * (np.abs(t) @ np.abs(x))).all()


@pytest.mark.parametrize("n", [64, 300, 700])
def test_inverse(dev, n):
    import torch

    lu, low, up = _factors(np.random.default_rng(n), n)
    Y = torch.empty(n, n, dtype=torch.float64, device=dev).t()
    _Handle(dev, INV)("tmvg_lu_inverse_f64", n, _dev(lu, dev), n, torch.arange(n, device=dev), Y, n)
    y = Y.cpu().numpy()
    # by rows of y: y (L U) = I up to the two triangles' and the products' rounding
    size = np.abs(y) @ np.abs(low) @ np.abs(up)
    inv = np.abs(np.linalg.inv(up)) @ np.abs(np.linalg.inv(low))
    assert (np.abs(y @ low @ up - np.eye(n)) <= 6 * n * U * (size + inv @ np.abs(low) @ np.abs(up))).all()


@pytest.mark.parametrize("n,refuse", [(40, WORK | INV | WORDS), (127, WORK | INV | WORDS), (200, INV), (200, WORDS)])
@pytest.mark.parametrize("nrhs", [2, 70])
def test_complex_left_solve(dev, n, refuse, nrhs):
    import torch

    rng = np.random.default_rng(n + nrhs)
    lu, low, up = _factors(rng, n, True)
    b = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    B = _dev(b, dev)
    _Handle(dev, refuse)("tmvg_lu_ldiveq_z64", n, _dev(lu, dev), n, torch.arange(n, device=dev), nrhs, B, n)
    x = B.cpu().numpy()
    assert (np.abs(low @ (up @ x) - b) <= 16 * n * U * (np.abs(low) @ (np.abs(up) @ np.abs(x)))).all()


@pytest.mark.parametrize("refuse", [WORK, INV, WORDS])
def test_complex_right_solve(dev, refuse):
    import torch

    n, rows = 200, 70
    rng = np.random.default_rng(refuse)
    lu, low, up = _factors(rng, n, True)
    b = rng.standard_normal((rows, n)) + 1j * rng.standard_normal((rows, n))
    B = _dev(b, dev)
    _Handle(dev, refuse)("tmvg_lu_rdiveq_z64", n, _dev(lu, dev), n, torch.arange(n, device=dev), rows, B, rows)
    x = B.cpu().numpy()
    assert (np.abs((x @ low) @ up - b) <= 16 * n * U * (np.abs(x) @ np.abs(low) @ np.abs(up))).all()


def test_product(dev):
    rng = np.random.default_rng(0)
    m, n, k = 300, 310, 320
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    X = _dev(np.zeros((m, n)), dev)
    _Handle(dev, POOL)("tmvg_multmm_f64", 0, 1.0, m, n, k, _dev(a, dev), 1, m, _dev(b, dev), 1, k, X, 1, m)
    assert (np.abs(X.cpu().numpy() - a @ b) <= 2 * k * U * (np.abs(a) @ np.abs(b))).all()
