"""alpha on products whose K is taken in blocks: alpha times the whole sum, also
where alpha times a part of it leaves the range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha", [np.inf, -np.inf, np.nan, 1e300, -1e-300, 0.5, 2.0 ** 60, 2.0 ** 61])
@pytest.mark.parametrize("add", [False, True])
def test_alpha_with_long_k(dev, alpha, add):
    import torch
    from helpers import to_dev, to_host

    from tmv_gb300 import linalg

    rng = np.random.default_rng(3)
    m, n, k = 70, 60, 20000
    a, b = rng.integers(-8, 9, (m, k)).astype(float), rng.integers(-8, 9, (k, n)).astype(float)
    b[:k // 2] += 4e6  # parts of the sum near 1e11 ...
    a[:, :k // 2] = np.abs(a[:, :k // 2])
    a[:, k // 2:2 * (k // 2)] = -a[:, :k // 2]  # ... that cancel
    b[k // 2:2 * (k // 2)] = b[:k // 2] + rng.integers(-8, 9, (k // 2, n))
    c = rng.standard_normal((m, n))
    want = a.astype(np.longdouble) @ b.astype(np.longdouble)  # exact: integers below 2^63
    X = to_dev(c, dev)
    linalg.multmm(add, float(alpha), to_dev(a, dev), to_dev(b, dev), X)
    torch.cuda.synchronize()
    got = to_host(X)
    with np.errstate(all="ignore"):
        ref = (float(alpha) * want.astype(float)) + (c if add else 0.0)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    inf = np.isinf(ref)
    assert np.array_equal(got[inf], ref[inf])
    fin = np.isfinite(ref)
    # the sums are exact in FP64 (below 2^53); alpha and the sum with C round
    part = np.abs(a[:, :k // 2]) @ np.abs(b[:k // 2])
    lim = 2.0 ** -52 * np.abs(ref) + (2.0 ** -52 * abs(alpha) * part if abs(alpha) <= 2.0 ** 60 else 0.0) + 5e-324
    assert (np.abs(got - ref)[fin] <= lim[fin]).all()
