"""Small complex left solves whose factors are not finite, against TMV's rule (the
oracle): a column of zeros is skipped and stays zero, every other column carries
the NaN to where the substitution takes it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 48, 65, 100, 127])
@pytest.mark.parametrize("what", [np.nan, np.inf])
@pytest.mark.parametrize("at", ["lower", "upper"])
def test_zero_columns_under_factors_not_finite(dev, orc, n, what, at):
    import torch

    from tmv_gb300 import linalg

    rng = np.random.default_rng(n)
    lu = rng.uniform(-0.5, 0.5, (n, n)) + 1j * rng.uniform(-0.5, 0.5, (n, n)) + 4 * np.eye(n)
    i, j = (n - 3, 1) if at == "lower" else (1, n - 3)
    lu[i, j] = what
    b = rng.standard_normal((n, 5)) + 1j * rng.standard_normal((n, 5))
    b[:, 1] = 0
    b[:, 3] = 0
    p = np.arange(n)
    X = linalg.colmajor(torch.from_numpy(b).to(dev))
    linalg.lu_ldiveq_z(linalg.colmajor(torch.from_numpy(lu).to(dev)), torch.from_numpy(p).to(dev), X)
    x = X.cpu().numpy()
    ref = np.asfortranarray(b.copy())
    orc.ldiveq_z(np.asfortranarray(lu), p, ref)
    assert (x[:, [1, 3]] == 0).all() and (ref[:, [1, 3]] == 0).all()
    # (which of NaN and infinity a complex product with an infinite part gives is
    # the order of its real operations', which nothing here promises)
    fin = np.isfinite(ref)
    assert np.array_equal(np.isfinite(x), fin)
    assert np.abs(x - ref)[fin].max() <= 16 * n * 2.0 ** -53 * np.abs(ref[fin]).max()
