"""Real solves and inverses of one and two 64-row blocks with any number of columns,
entry by entry: n 2^-53 |L||U||x| for the two triangles' substitutions, doubled for
the FP64 reference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _factor(dev, n, seed):
    import torch

    from tmv_gb300 import linalg

    a = np.random.default_rng(seed).standard_normal((n, n))
    LU = linalg.colmajor(torch.from_numpy(a).to(dev))
    P = linalg.lu_decompose(LU)
    lu = LU.cpu().numpy()
    return a, LU, P, np.tril(lu, -1) + np.eye(n), np.triu(lu)


@pytest.mark.parametrize("n", [1, 2, 16, 63, 64, 65])
@pytest.mark.parametrize("nrhs", [1, 8, 9, 17, 100, 256])
def test_left_and_right_solve(dev, n, nrhs):
    import torch

    from tmv_gb300 import linalg

    a, LU, P, low, up = _factor(dev, n, n)
    b = np.random.default_rng(nrhs).standard_normal((n, nrhs))
    X, Y = linalg.colmajor(torch.from_numpy(b).to(dev)), linalg.colmajor(torch.from_numpy(b.T.copy()).to(dev))
    linalg.lu_ldiveq(LU, P, X)
    linalg.lu_rdiveq(LU, P, Y)
    x, y = X.cpu().numpy(), Y.cpu().numpy()
    pa = np.arange(n)
    for i, q in enumerate(P.cpu().numpy()):
        pa[[i, q]] = pa[[q, i]]
    lim = 4 * (n + 1) * 2.0 ** -53
    assert (np.abs(low @ (up @ x) - b[pa]) <= lim * (np.abs(low) @ (np.abs(up) @ np.abs(x)))).all()
    z = y[:, pa]  # y P^-1 ... (y P) L U = b^T
    assert (np.abs((z @ low) @ up - b.T) <= lim * (np.abs(z) @ np.abs(low) @ np.abs(up))).all()


@pytest.mark.parametrize("n", [1, 2, 8, 33, 43, 44, 45, 64])
def test_inverse(dev, n):
    """Both sides of the inverse's line (44)."""
    from tmv_gb300 import linalg

    a, LU, P, low, up = _factor(dev, n, 70 + n)
    y = linalg.lu_inverse(LU, P).cpu().numpy()
    pa = np.arange(n)
    for i, q in enumerate(P.cpu().numpy()):
        pa[[i, q]] = pa[[q, i]]
    z = y[:, pa]  # (P A)^-1: columns of U^-1 L^-1, each by two substitutions
    size = np.abs(low) @ (np.abs(up) @ np.abs(z))
    assert (np.abs(low @ (up @ z) - np.eye(n)) <= 4 * (n + 1) * 2.0 ** -53 * size).all()
