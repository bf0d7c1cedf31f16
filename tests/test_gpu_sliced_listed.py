"""Products some of whose tiles cannot be sliced: those run on the FP64 pipe in a
launch of their own, spread over the device in 8 x 8 blocks, while the rest of the
product stays on the tensor cores.

Bound per element: a chain of K FMAs, K 2^-53 |A||B| (sliced tiles are below it),
one rounding for alpha and one for the sum with C; a factor 2 for the reference,
which is computed in extended precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _operand(rng, what, m, k):
    a = rng.standard_normal((m, k))
    if what == "lower":
        a = np.tril(a)
    elif what == "upper":
        a = np.triu(a)
    elif what == "band":
        a = np.triu(np.tril(a, 2), -2)
    elif what == "alternate":  # every other 128 rows sparse: both kinds of tile in one CTA
        sparse = (np.arange(m) // 128 % 2 == 0)[:, None]
        a = np.where(sparse, a * (rng.random((m, k)) < 0.02), a)
    elif what == "graded":
        a = a * 2.0 ** -np.linspace(0, 60, k)
    return a


def _check(dev, a, b, c0, add, alpha, la, lb, lc, rows):
    import torch
    from helpers import to_dev, to_host

    from tmv_gb300 import linalg

    A, B, C = to_dev(a, dev, la), to_dev(b, dev, lb), to_dev(c0, dev, lc)
    linalg.multmm(add, alpha, A, B, C)
    torch.cuda.synchronize()
    got = to_host(C)[rows]
    k = a.shape[1]
    want = alpha * (a[rows].astype(np.longdouble) @ b.astype(np.longdouble)) + (c0[rows] if add else 0.0)
    size = abs(alpha) * (np.abs(a[rows]) @ np.abs(b))
    lim = 2 * (k * 2.0 ** -53 * size + 2.0 ** -52 * np.abs(want).astype(float) + (2.0 ** -53 * size))
    assert (np.abs((got - want).astype(float)) <= lim).all()


# edges of the 128 x 64 (short K: 128 x 32) tiles, of the 8 x 8 blocks and of K = 32
@pytest.mark.parametrize("m,n,k", [(300, 300, 300), (257, 130, 700), (129, 1000, 97), (1030, 400, 33), (500, 777, 32),
                                   (64, 48, 4001)])
@pytest.mark.parametrize("what", ["lower", "upper", "band", "alternate", "graded"])
@pytest.mark.parametrize("la,lb,lc", [("F", "F", "F"), ("C", "C", "F"), ("F", "F", "C")])
def test_unsliceable_operands(dev, m, n, k, what, la, lb, lc):
    rng = np.random.default_rng(m + n + k)
    a, b, c0 = _operand(rng, what, m, k), rng.standard_normal((k, n)), rng.standard_normal((m, n))
    if what == "graded":
        b = b * 2.0 ** np.linspace(0, 60, k)[:, None]
    rows = np.unique(np.concatenate([[0, m - 1], rng.integers(0, m, 40)]))
    for add, alpha in [(False, 1.0), (True, -1.0), (True, 0.37)]:
        _check(dev, a, b, c0, add, alpha, la, lb, lc, rows)


def test_many_unsliceable_tiles_between_sliced_ones(dev):
    """Some thousand tiles, more than ten per CTA, every other row of tiles on
    the FP64 pipe."""
    rng = np.random.default_rng(8)
    m, n, k = 4100, 3000, 160
    a, b, c0 = _operand(rng, "alternate", m, k), rng.standard_normal((k, n)), rng.standard_normal((m, n))
    _check(dev, a, b, c0, True, -1.0, "F", "F", "F", np.unique(rng.integers(0, m, 60)))


def test_not_finite_entry(dev):
    """A NaN reaches its row of the product only; the other rows of tiles keep
    their bits."""
    import torch

    from tmv_gb300 import linalg

    g = torch.Generator(device=dev).manual_seed(2)
    A, B = (linalg.colmajor(torch.randn(700, 700, dtype=torch.float64, device=dev, generator=g)) for _ in range(2))
    C, D = torch.empty_like(A), torch.empty_like(A)
    linalg.multmm(False, 1.0, A, B, C)
    A[300, 5] = float("nan")
    linalg.multmm(False, 1.0, A, B, D)
    assert torch.isnan(D[300]).all()
    other = torch.arange(700, device=dev) // 128 != 300 // 128
    assert torch.equal(C[other], D[other])
    near = ~other
    near[300] = False
    size = A[near].abs().sum(1).max().item() * B.abs().max().item()
    assert (C[near] - D[near]).abs().max().item() <= 700 * 2.0 ** -52 * size


def test_complex_factors_of_a_sparse_matrix(dev):
    """The complex factorisation's wide update takes the same route (its left
    operand in real form): |PA - LU| <= 8 n 2^-53 |L||U| entry by entry."""
    import torch

    from tmv_gb300 import linalg

    rng = np.random.default_rng(4)
    n = 900
    keep = rng.random((n, n)) < 0.01
    a = np.where(keep, rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)), 0) + 0.1 * np.eye(n)
    LU = linalg.colmajor(torch.from_numpy(a).to(dev))
    P = linalg.lu_decompose_z(LU).cpu().numpy()
    lu = LU.cpu().numpy()
    for i, q in enumerate(P):
        a[[i, q]] = a[[q, i]]
    low, up = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    assert np.abs(low).max() <= 1.0 + 1e-14
    assert (np.abs(low @ up - a) <= 8 * n * 2.0 ** -53 * (np.abs(low) @ np.abs(up))).all()


def test_one_row_of_tiles_does_not_wait_for_one_sm(dev):
    """A NaN puts one row of tiles on the FP64 pipe: a fifth of a 600 x 600 x 600
    product, 93 us of a whole device's FP64 pipe (2 FMAs per SM and clock) and 1.2 ms
    where each of its ten tiles is one SM's; allowed for: five times the product
    without it (about 70 us)."""
    import torch

    from tmv_gb300 import linalg

    g = torch.Generator(device=dev).manual_seed(6)
    A, B = (linalg.colmajor(torch.randn(600, 600, dtype=torch.float64, device=dev, generator=g)) for _ in range(2))
    C, N = torch.empty_like(A), A.t().clone().t()
    N[300, 5] = float("nan")
    torch.cuda.synchronize()

    def us(X):
        out = []
        for _ in range(9):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            for _ in range(10):
                linalg.multmm(False, 1.0, X, B, C)
            e[1].record()
            torch.cuda.synchronize()
            out.append(e[0].elapsed_time(e[1]) * 100)
        return sorted(out)[4]

    us(A)
    assert us(N) <= 5 * us(A)
