"""FP64 products from exact slices on the tensor cores, against exact integer
arithmetic.

Operands are integers of up to 53 bits times a power of two, so the exact
product is a Python integer.  Tolerance, per element, of a sliced tile: the
digit pairs left out and the digits' last rounding are below K (7 + 2) 2^-64 of
the product of the row's and the column's scale (powers of two above their
largest entries), i.e. K 2^-60, and the result is rounded once (2^-53 of it),
with a rounding for alpha and one for the sum with C.  A tile (128 x 64) whose
rows and columns do not overlap in their large entries runs as a chain of FMAs:
K 2^-53 |A||B|; the tiles that certainly do overlap are worked out here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _operands(rng, m, n, k, spread):
    a = rng.integers(-2**52, 2**52, (m, k)) >> rng.integers(0, spread + 1, (m, k))
    b = rng.integers(-2**52, 2**52, (k, n)) >> rng.integers(0, spread + 1, (k, n))
    return a, b


def _run(dev, a, b, c0, add, alpha, la, lb, lc):
    import torch
    from helpers import to_dev, to_host

    from tmv_gb300 import linalg

    A, B, C = to_dev(a, dev, la), to_dev(b, dev, lb), to_dev(c0, dev, lc)
    linalg.multmm(add, alpha, A, B, C)
    torch.cuda.synchronize()
    return to_host(C)


def _sliced(a, b):
    """Per element: whether its tile's vectors have enough entries within 2^-4
    of their largest for any two to meet in 1.75 sqrt(K) places (and the
    product is large enough to be sliced at all)."""
    k = a.shape[1]
    if a.shape[0] < 64 or b.shape[1] < 48 or k < 24 or a.size * b.shape[1] < 1.2e7:
        return np.zeros((a.shape[0], b.shape[1]), bool)
    ea, eb = np.frexp(np.abs(a).astype(float))[1], np.frexp(np.abs(b).astype(float))[1]
    fa = ((ea >= ea.max(1, keepdims=True) - 4) & (a != 0)).sum(1)
    fb = ((eb >= eb.max(0, keepdims=True) - 4) & (b != 0)).sum(0)
    ta = np.repeat([fa[i:i + 128].min() for i in range(0, len(fa), 128)], 128)[:len(fa)]
    tb = np.repeat([fb[i:i + 64].min() for i in range(0, len(fb), 64)], 64)[:len(fb)]
    return ta[:, None] + tb[None, :] - k >= np.ceil(1.75 * np.sqrt(k))


# tiles are 128 x 64 (128 x 32 for short K), stages 32 and accumulation chunks 128 in K
SIZES = [(128, 64, 1500), (127, 64, 1600), (129, 65, 1537), (300, 200, 255), (640, 257, 129), (257, 700, 97),
         (1000, 500, 32), (70, 2800, 64), (64, 3000, 160), (2500, 50, 128), (600, 289, 96), (1300, 97, 127)]


@pytest.mark.parametrize("m,n,k", SIZES)
@pytest.mark.parametrize("la,lb,lc", [("F", "F", "F"), ("C", "F", "F"), ("F", "C", "C"), ("C", "C", "F")])
@pytest.mark.parametrize("spread", [1, 6])
def test_exact_integers(dev, m, n, k, la, lb, lc, spread):
    rng = np.random.default_rng(m * 7 + n * 3 + k)
    a, b = _operands(rng, m, n, k, spread)
    pick_r, pick_c = rng.integers(0, m, 24), rng.integers(0, n, 24)
    pick_r[:2], pick_c[:2] = (0, m - 1), (0, n - 1)
    exact = a[pick_r].astype(object) @ b[:, pick_c].astype(object)
    scale = np.outer(2.0 ** np.ceil(np.log2(np.abs(a[pick_r]).max(1) + 1.0)),
                     2.0 ** np.ceil(np.log2(np.abs(b[:, pick_c]).max(0) + 1.0)))
    # a row-major C is the product of the transposes: its tiles are C's
    # transposed
    tile = _sliced(a, b) if lc == "F" else _sliced(b.T, a.T).T
    tile = tile[np.ix_(pick_r, pick_c)]
    assert tile.all() or spread > 1 or min(m, n) < 64 or m * n * k < 1.2e7
    chain = k * 2.0 ** -53 * (np.abs(a[pick_r]).astype(float) @ np.abs(b[:, pick_c]).astype(float))
    for add, alpha in [(False, 1.0), (True, -1.0), (True, 0.375)]:
        c0 = rng.standard_normal((m, n)) * 2.0 ** 100
        got = _run(dev, a.astype(float), b.astype(float), c0, add, alpha, la, lb, lc)[np.ix_(pick_r, pick_c)]
        want = exact.astype(float) * alpha + (c0[np.ix_(pick_r, pick_c)] if add else 0.0)
        size = np.abs(exact.astype(float)) + (np.abs(c0[np.ix_(pick_r, pick_c)]) if add else 0.0)
        tol = np.where(tile, k * 2.0 ** -60 * scale, np.maximum(chain, k * 2.0 ** -60 * scale)) + 2.0 ** -51 * size
        assert (np.abs(got - want) <= tol).all()


@pytest.mark.parametrize("k", [32, 200, 700])
def test_special_operands(dev, k):
    """Vectors that cannot be sliced take the FP64 pipe with the FMA chain of
    the plain kernel: not finite, opposite grading, sparse, extreme scales."""
    rng = np.random.default_rng(k)
    m, n = 400, 390
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    a[5, 3], a[140, k - 1], b[2, 200] = np.nan, np.inf, -np.inf
    got = _run(dev, a, b, np.zeros((m, n)), False, 1.0, "F", "F", "F")
    with np.errstate(invalid="ignore"):
        want = a @ b
    assert np.array_equal(np.isnan(got), np.isnan(want))
    fin = np.isfinite(want)
    assert np.array_equal(got[~fin & ~np.isnan(want)], want[~fin & ~np.isnan(want)])
    lim = k * 2.0 ** -52 * (np.abs(np.nan_to_num(a, posinf=0, neginf=0)) @ np.abs(np.nan_to_num(b, posinf=0, neginf=0)))
    assert (np.abs(got - want)[fin] <= lim[fin]).all()
    # zero rows and columns among ordinary ones are exactly zero
    x, y = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    x[130:135], y[:, 70] = 0.0, 0.0
    got = _run(dev, x, y, np.zeros((m, n)), False, 1.0, "F", "F", "F")
    assert (got[130:135] == 0).all() and (got[:, 70] == 0).all()
    assert (np.abs(got - x @ y) <= k * 2.0 ** -52 * (np.abs(x) @ np.abs(y))).all()
    # graded against each other: every product is about 1, each entry's own
    # size from 1 to 2^40 of its vector's largest; and a sparse pair; both to
    # the componentwise bound of an FMA chain, K 2^-53 |A||B|
    grade = 2.0 ** np.linspace(0, 40, k)
    sparse = rng.standard_normal((m, k)) * (rng.random((m, k)) < 0.03)
    for x, y in [(rng.standard_normal((m, k)) * grade, (rng.standard_normal((n, k)) / grade).T), (sparse, np.ones((k, n))),
                 (rng.standard_normal((m, k)) * 2.0 ** 700, rng.standard_normal((k, n)) * 2.0 ** -700),
                 (rng.standard_normal((m, k)) * 2.0 ** -1060, rng.standard_normal((k, n)) * 2.0 ** 900)]:
        got = _run(dev, x, y, np.zeros((m, n)), False, 1.0, "C", "F", "F")
        ref = x.astype(np.longdouble) @ y.astype(np.longdouble)
        err = np.abs((got - ref).astype(float))
        assert (err <= k * 2.0 ** -52 * (np.abs(x) @ np.abs(y))).all()


def test_streams_do_not_share_scratch(dev):
    """Two streams' products in flight together on one handle."""
    import torch

    from tmv_gb300 import linalg

    g = torch.Generator(device=dev).manual_seed(3)
    ops = [[linalg.colmajor(torch.randn(700, 700, dtype=torch.float64, device=dev, generator=g)) for _ in range(3)]
           for _ in range(2)]
    want = []
    for A, B, C in ops:
        linalg.multmm(False, 1.0, A, B, C)
        want.append(C.clone())
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(20):
        for s, (A, B, C) in zip(streams, ops):
            with torch.cuda.stream(s):
                C.zero_()
                linalg.multmm(False, 1.0, A, B, C)
    torch.cuda.synchronize()
    for w, (_, _, C) in zip(want, ops):
        assert torch.equal(w, C)
