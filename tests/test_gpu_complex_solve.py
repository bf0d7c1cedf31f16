"""The complex left and right solves as real ones (zlu.cu, trsv.cu), against the
backward error of a substitution: |b - A x| <= c n 2^-53 (|L||U||x|), with c = 8
for complex arithmetic (four real products and two sums per complex one, both
triangles), at the edges of its 32-row blocks; a singular factor is reported
and leaves nothing behind on the handle; a column with a NaN reaches no other
column."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(n, nrhs, seed):
    rng = np.random.default_rng(seed)
    z = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    return z(n, n), z(n, nrhs)


def _dev(a, dev):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a.T)).to(dev).t()


@pytest.mark.parametrize("n", [32, 33, 63, 64, 128, 129, 159, 160, 161, 192, 500])
@pytest.mark.parametrize("nrhs", [1, 3, 8, 9, 64])
def test_backward_error(dev, n, nrhs):
    from tmv_gb300 import linalg

    a, b = _problem(n, nrhs, n + nrhs)
    LU, X = _dev(a, dev), _dev(b, dev)
    P = linalg.lu_decompose_z(LU)
    linalg.lu_ldiveq_z(LU, P, X)
    lu, x, p = LU.cpu().numpy(), X.cpu().numpy(), P.cpu().numpy()
    pb = b.copy()
    for i, q in enumerate(p):
        pb[[i, q]] = pb[[q, i]]
    low, up = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    ext = np.clongdouble
    r = np.abs((low.astype(ext) @ (up.astype(ext) @ x.astype(ext)) - pb).astype(complex))
    assert (r <= 8 * n * 2.0 ** -53 * (np.abs(low) @ (np.abs(up) @ np.abs(x)))).all()


def test_singular_then_regular_and_nan(dev):
    from tmv_gb300 import _lib, linalg

    n = 200
    a, b = _problem(n, 4, 1)
    good, x0 = _dev(a, dev), _dev(b, dev)
    P = linalg.lu_decompose_z(good)
    bad = _dev(good.cpu().numpy(), dev)
    bad[150, 150] = 0.0
    x = _dev(b, dev)
    with pytest.raises(_lib.SingularError):
        linalg.lu_ldiveq_z(bad, P, x)
    linalg.lu_ldiveq_z(good, P, x0)
    want = np.linalg.solve(a, b)
    assert np.linalg.norm(x0.cpu().numpy() - want) <= 1e-10 * np.linalg.norm(want)
    c = b.copy()
    c[70, 2] = np.nan
    x = _dev(c, dev)
    linalg.lu_ldiveq_z(good, P, x)
    got = x.cpu().numpy()
    assert np.isnan(got[:, 2]).any()
    rest = [0, 1, 3]
    assert np.linalg.norm(got[:, rest] - want[:, rest]) <= 1e-10 * np.linalg.norm(want)


# (one more row than a launch takes, and more than two launches of rows)
@pytest.mark.parametrize("n", [131, 159, 160, 161, 500])
@pytest.mark.parametrize("rows", [1, 3, 64, 65, 130])
def test_right_backward_error(dev, n, rows):
    from tmv_gb300 import linalg

    a, b = _problem(n, rows, n + rows)
    b = np.ascontiguousarray(b.T)
    LU, X = _dev(a, dev), _dev(b, dev)
    P = linalg.lu_decompose_z(LU)
    linalg.lu_rdiveq_z(LU, P, X)
    lu, x, p = LU.cpu().numpy(), X.cpu().numpy(), P.cpu().numpy()
    for i, q in enumerate(p):
        x[:, [i, q]] = x[:, [q, i]]
    low, up = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    ext = np.clongdouble
    r = np.abs(((x.astype(ext) @ low.astype(ext)) @ up.astype(ext) - b).astype(complex))
    assert (r <= 8 * n * 2.0 ** -53 * ((np.abs(x) @ np.abs(low)) @ np.abs(up))).all()


def test_right_singular_then_regular_and_nan(dev):
    from tmv_gb300 import _lib, linalg

    n = 200
    a, b = _problem(n, 70, 2)
    b = np.ascontiguousarray(b.T)
    good = _dev(a, dev)
    P = linalg.lu_decompose_z(good)
    bad = _dev(good.cpu().numpy(), dev)
    bad[150, 150] = 0.0
    with pytest.raises(_lib.SingularError):
        linalg.lu_rdiveq_z(bad, P, _dev(b, dev))
    want = np.linalg.solve(a.T, b.T).T
    c = b.copy()
    c[2, 70] = np.nan
    x = _dev(c, dev)
    linalg.lu_rdiveq_z(good, P, x)
    got = x.cpu().numpy()
    rest = np.arange(70) != 2
    assert np.linalg.norm(got[rest] - want[rest]) <= 1e-10 * np.linalg.norm(want[rest])
    assert np.isnan(got[2]).any()


def _right_serial(lu, p, b):
    """TMV's order, one operation at a time (numpy would fuse nothing, but
    reorders nothing either: scalar products and sums)."""
    n = lu.shape[0]
    mul = lambda x, y: complex(x.real * y.real - x.imag * y.imag, x.real * y.imag + x.imag * y.real)  # noqa: E731

    def inv(d):
        r, i = d.real, d.imag
        if abs(r) > abs(i):
            i = i / r
            t = r * (1.0 + i * i)
            return complex(1.0 / t, -i / t)
        r = r / i
        t = i * (1.0 + r * r)
        return complex(r / t, -1.0 / t)

    x = [complex(v) for v in b]
    i1 = next((i for i in range(n) if x[i] != 0), n)
    for i in range(i1, n):
        v = x[i]
        for j in range(i1, i):
            v = v - mul(x[j], complex(lu[j, i]))
        x[i] = mul(v, inv(complex(lu[i, i])))
    i2 = max((i + 1 for i in range(n) if x[i] != 0), default=0)
    for i in range(i2 - 1, -1, -1):
        v = x[i]
        for j in range(i + 1, i2):
            v = v - mul(x[j], complex(lu[j, i]))
        x[i] = v
    for i in range(n - 1, -1, -1):
        x[i], x[p[i]] = x[p[i]], x[i]
    return np.array(x)


# edges of the warps and of the range, rows that start or end with zeros
@pytest.mark.parametrize("n", [1, 2, 31, 33, 64, 97, 129, 130])
def test_right_small_keeps_the_order(dev, n):
    from tmv_gb300 import linalg

    a, b = _problem(n, 5, 31 * n)
    b = np.ascontiguousarray(b.T)
    b[1, : n // 2] = 0
    b[2, n // 2:] = 0
    b[3] = 0
    LU, X = _dev(a, dev), _dev(b, dev)
    P = linalg.lu_decompose_z(LU)
    linalg.lu_rdiveq_z(LU, P, X)
    lu, p, x = LU.cpu().numpy(), P.cpu().numpy(), X.cpu().numpy()
    for r in range(5):
        np.testing.assert_array_equal(x[r], _right_serial(lu, p, b[r]))
