"""The inverse from its factors where the 64-row diagonal blocks are hard: unit
lower blocks with large multipliers."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inverse(dev, lu):
    import torch
    from helpers import to_dev, to_host

    from tmv_gb300 import linalg

    n = lu.shape[0]
    LU, P = to_dev(lu, dev), torch.arange(n, device=dev)
    Y = torch.empty(n, n, dtype=torch.float64, device=dev).t()
    h = linalg.handle(dev.index or 0)
    h.check(h.call("tmvg_lu_inverse_f64", n, C.c_void_p(LU.data_ptr()), n, C.c_void_p(P.data_ptr()),
                   C.c_void_p(Y.data_ptr()), n))
    return to_host(Y)


def _substitute(low, cols):
    """Columns `cols` of low^-1 in FP64, a column of low at a time."""
    n = low.shape[0]
    y = np.eye(n)[:, cols]
    for k in range(n):
        y[k + 1:] -= low[k + 1:, k:k + 1] * y[k]
    return y


@pytest.mark.parametrize("n", [64, 130, 448, 512, 513, 700, 1000])
def test_lower_blocks_with_large_multipliers(dev, n):
    """U = I, multipliers uniform in (-1, 1): the factors of a legal partial
    pivoting whose 64-row blocks are far from orthogonal.  The componentwise
    residual |L Y - I| / |L||Y| may be three times that of the plain substitution
    (about 2e-16); blocks multiplied by their inverse without a correction leave
    1e-15 and more."""
    rng = np.random.default_rng(n)
    low = np.tril(rng.uniform(-1.0, 1.0, (n, n)), -1) + np.eye(n)
    cols = np.unique(np.concatenate([np.arange(0, n, max(1, n // 24)), [n - 1]]))

    def residual(y):
        ext = low.astype(np.longdouble)
        r = np.abs(ext @ y.astype(np.longdouble) - np.eye(n)[:, cols])
        size = np.abs(low) @ np.abs(y)
        return float((r / np.where(size > 0, size, 1.0)).max())

    assert residual(_inverse(dev, low)[:, cols]) <= 3 * residual(_substitute(low, cols))
