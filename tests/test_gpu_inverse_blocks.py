"""The inverse from its factors where the 64-row diagonal blocks are hard: unit
lower blocks with large multipliers, and blocks whose own inverse is not finite."""
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


# (rows and columns of a 64-row block, and of two blocks)
@pytest.mark.parametrize("n,i,j", [(40, 3, 9), (64, 0, 63), (150, 70, 100), (150, 130, 149), (700, 600, 630)])
@pytest.mark.parametrize("size", [1e200, np.inf])
def test_block_whose_inverse_overflows(dev, n, i, j, size):
    """U = I but for two diagonal entries 1e-200 and U(i, j): x(i, j) overflows, all
    other entries are finite (or, under an infinite U(i, j), what 0 times it
    leaves), as the substitution finds them."""
    up = np.eye(n)
    up[i, i] = up[j, j] = 1e-200
    up[i, j] = size
    want = np.eye(n)
    b0 = j // 64 * 64
    with np.errstate(all="ignore"):
        for k in reversed(range(n)):
            want[k] = want[k] * (1.0 / up[k, k])
            want[:k] -= up[:k, k:k + 1] * want[k]
    got = _inverse(dev, up)
    assert b0 <= i, "both in one block"
    assert np.array_equal(np.isnan(got), np.isnan(want))
    fin = np.isfinite(want)
    assert np.array_equal(got[~fin & ~np.isnan(want)], want[~fin & ~np.isnan(want)])
    assert (np.abs(got - want)[fin] <= 2.0 ** -50 * np.abs(want)[fin]).all()


def test_lower_block_whose_inverse_overflows(dev):
    """Multipliers of 1e160 twice in a row: one entry of L^-1 overflows, and 0 times
    it fills its column, below by L and above by U = I; every other column is as the
    substitution has it."""
    n = 100
    low = np.eye(n)
    low[71, 70] = low[72, 71] = 1e160
    with np.errstate(all="ignore"):
        want = _substitute(low, np.arange(n))
        assert np.isinf(want).sum() == 1
        for k in reversed(range(n)):
            want[:k] -= 0.0 * want[k]
    assert np.array_equal(_inverse(dev, low), want, equal_nan=True)
