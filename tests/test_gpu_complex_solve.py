"""The complex left solve as a real one (zlu.cu, trsv.cu), against the
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


@pytest.mark.parametrize("n", [128, 129, 159, 160, 161, 192, 500])
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
