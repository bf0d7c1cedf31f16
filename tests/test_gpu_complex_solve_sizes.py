"""The complex left solve and inverse on both sides of every line of their dispatch
(31/32, 47/48, 64/65, 127/128 unknowns; 64/65 columns): backward error entry by
entry, 4 operations per complex one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 32, 40, 47, 48, 64, 65, 100, 127, 128])
@pytest.mark.parametrize("nrhs", [1, 64, 65, 130])
def test_left_solve(dev, n, nrhs):
    import torch

    from tmv_gb300 import linalg

    rng = np.random.default_rng(1000 * n + nrhs)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    b = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    LU, X = (linalg.colmajor(torch.from_numpy(v).to(dev)) for v in (a, b))
    P = linalg.lu_decompose_z(LU)
    linalg.lu_ldiveq_z(LU, P, X)
    lu, x = LU.cpu().numpy(), X.cpu().numpy()
    for i, q in enumerate(P.cpu().numpy()):
        b[[i, q]] = b[[q, i]]
    low, up = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    assert (np.abs(low @ (up @ x) - b) <= 16 * n * 2.0 ** -53 * (np.abs(low) @ (np.abs(up) @ np.abs(x)))).all()


@pytest.mark.parametrize("n", [31, 32, 33, 47, 48, 65, 127])
def test_inverse(dev, n):
    import torch

    from tmv_gb300 import linalg

    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 3 * n ** 0.5 * np.eye(n)
    LU = linalg.colmajor(torch.from_numpy(a).to(dev))
    P = linalg.lu_decompose_z(LU)
    y = linalg.lu_inverse_z(LU, P).cpu().numpy()
    assert np.abs(a @ y - np.eye(n)).max() <= 16 * n * 2.0 ** -53 * np.abs(a).sum(1).max() * np.abs(y).max()
