"""The 64-row diagonal blocks of the sync-free triangular solve: by their
inverse with one correction (up to 8 columns), by the inverse (more), by
substitution (a zero diagonal, n <= 64, or a result that is not finite).

Tolerance: componentwise backward error |b - T x| <= c (|T| |x|).  A
substitution of n rows has c = n 2^-53 (Higham, Accuracy and Stability of
Numerical Algorithms, theorem 8.5); the corrected product of a 64-row block
satisfies the same order of bound, so 2 n 2^-53 is asked of both.  The plain
inverse's bound carries the block's condition: 64 2^-53 cond(block).  Asked
only where the solution is within the range of FP64 (a long triangle with a
small diagonal overflows), which extended precision decides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _triangle(n, bad, seed):
    rng = np.random.default_rng(seed)
    t = rng.standard_normal((n, n)) / np.sqrt(n)
    t[np.diag_indices(n)] = 10.0 ** rng.uniform(-5, 0, n) if bad else 1.0 + rng.random(n)
    return t


def _solve(dev, t, b, upper, unit):
    import torch
    from helpers import to_dev, to_host

    from tmv_gb300 import linalg

    B = to_dev(b, dev, "F")
    linalg.tri_ldiveq(to_dev(t, dev, "F"), upper, unit, B)
    torch.cuda.synchronize()
    return to_host(B)


def _in_range(m, b, upper):
    x = b.astype(np.longdouble)
    m = m.astype(np.longdouble)
    order = range(len(m))[::-1] if upper else range(len(m))
    for j in order:
        x[j] /= m[j, j]
        rest = slice(0, j) if upper else slice(j + 1, None)
        x[rest] -= np.outer(m[rest, j], x[j])
    return float(np.abs(x).max()) < 1e290


@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 128, 129, 320, 1000])
@pytest.mark.parametrize("nrhs", [1, 2, 8, 9, 33])
@pytest.mark.parametrize("bad", [False, True])
def test_backward_error(dev, n, nrhs, bad):
    t = _triangle(n, bad, n + nrhs)
    b = np.random.default_rng(n * nrhs).standard_normal((n, nrhs))
    for upper, unit in [(True, False), (False, False), (False, True), (True, True)]:
        m = np.triu(t) if upper else np.tril(t)
        if unit:
            m[np.diag_indices(n)] = 1.0
        x = _solve(dev, t, b, upper, unit)
        if not _in_range(m, b, upper):
            assert bad
            continue
        r = np.abs((m.astype(np.longdouble) @ x.astype(np.longdouble) - b).astype(float))
        c = 2 * n * 2.0 ** -53
        if nrhs > 8:
            c += 64 * 2.0 ** -53 * max(np.linalg.cond(m[i:i + 64, i:i + 64]) for i in range(0, n, 64))
        assert (r <= c * (np.abs(m) @ np.abs(x))).all(), (upper, unit)


@pytest.mark.parametrize("nrhs", [1, 3])
def test_not_finite_stays_where_substitution_puts_it(dev, nrhs):
    """A NaN or an infinity in b or in T reaches the entries it reaches in a
    column-by-column substitution, and no other."""
    n = 200
    t = _triangle(n, False, 5)
    b = np.random.default_rng(6).standard_normal((n, nrhs))
    for at, value in [(70, np.nan), (130, np.inf)]:
        c = b.copy()
        c[at, 0] = value
        for upper in (False, True):
            x = _solve(dev, t, c, upper, False)
            reached = np.arange(n) >= at if not upper else np.arange(n) <= at
            assert not np.isfinite(x[reached, 0]).any() and np.isfinite(x[~reached, 0]).all()
            assert np.isfinite(x[:, 1:]).all()
    s = t.copy()
    s[100, 97] = np.inf  # strictly lower: rows 100.. of the lower solve only
    x = _solve(dev, s, b, False, False)
    assert np.isfinite(x[:100]).all() and not np.isfinite(x[100:]).any()
    assert np.isfinite(_solve(dev, s, b, True, False)).all()
