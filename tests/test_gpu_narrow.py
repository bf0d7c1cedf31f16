"""The update of the next panel's columns at the edges of its rows per CTA (4, 8
or 16 by the rows left): |PA - LU| <= n 2^-53 |L||U| entry by entry (gamma_n of the
elimination, an operation per term), and every multiplier at most 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 36, 37, 64, 609, 639, 640, 641, 673, 1217, 1248, 1249, 1281])
def test_factors_reproduce_the_matrix(dev, n):
    import torch

    from tmv_gb300 import linalg

    a = np.random.default_rng(n).standard_normal((n, n))
    LU = torch.from_numpy(np.ascontiguousarray(a.T)).to(dev).t()
    P = linalg.lu_decompose(LU).cpu().numpy()
    lu = LU.cpu().numpy()
    for i, q in enumerate(P):
        a[[i, q]] = a[[q, i]]
    low, up = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    assert np.abs(low).max() <= 1.0
    ext = np.longdouble if n < 700 else np.float64  # (FP64: its own n 2^-53 |L||U| allowed for)
    r = np.abs((low.astype(ext) @ up.astype(ext) - a).astype(float))
    assert (r <= (1 if n < 700 else 2) * n * 2.0 ** -53 * (np.abs(low) @ np.abs(up))).all()
