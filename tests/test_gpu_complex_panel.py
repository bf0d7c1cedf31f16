"""The complex panel's shared state: repeated factorisations of one matrix.

Threads of a CTA meet between one column's update and the next column's pivot
search only if each keeps its rows.  A thread that reads a row another one is
still writing picks pivots and multipliers that differ from run to run, so the
interchanges and every bit of the factors have to be the same each time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 69 to 384 rows per CTA: one thread per row, fewer than one warp's worth of
# idle threads, and (n = 8000: 16-column panels) more than one row per thread
@pytest.mark.parametrize("n,runs", [(1100, 60), (2048, 40), (4001, 10), (6144, 6), (8000, 4)])
def test_repeated_factorisation_is_bitwise(dev, n, runs):
    import torch

    from tmv_gb300 import linalg

    g = torch.Generator(device=dev).manual_seed(n)
    A = linalg.colmajor(torch.complex(*(torch.randn(n, n, dtype=torch.float64, device=dev, generator=g)
                                        for _ in range(2))))
    first = None
    for _ in range(runs):
        LU = A.t().clone().t()
        P = linalg.lu_decompose_z(LU)
        if first is None:
            first = (LU, P)
            # partial pivoting: no multiplier above 1 (to the rounding of a
            # complex quotient)
            assert torch.tril(LU, -1).abs().max().item() <= 1.0 + 1e-14
            continue
        assert torch.equal(P, first[1])
        assert torch.equal(torch.view_as_real(LU), torch.view_as_real(first[0]))


@pytest.mark.parametrize("n", [40, 300, 1100])
def test_columns_of_ties(dev, n):
    """Entries 1, i, -1, -i: every row of the first column ties, and again in the
    first column of each decoupled block, so the second exchange decides."""
    import torch

    from tmv_gb300 import linalg

    rng = np.random.default_rng(n)
    a = np.zeros((n, n), complex)
    for k in range(0, n, 20):  # blocks of 20, each with ties of its own
        w = min(20, n - k)
        a[k:k + w, k:k + w] = 1j ** rng.integers(0, 4, (w, w))
    a[:, -1] = 1j ** rng.integers(0, 4, n)
    A = linalg.colmajor(torch.from_numpy(a).to(dev))
    got = []
    for _ in range(5):
        LU = A.t().clone().t()
        got.append((linalg.lu_decompose_z(LU), LU))
    P, LU = got[0]
    for p, lu in got[1:]:
        assert torch.equal(p, P)
        assert torch.equal(torch.view_as_real(lu), torch.view_as_real(LU))
    pa, lu = a.copy(), LU.cpu().numpy()
    for i, q in enumerate(P.cpu().numpy()):
        pa[[i, q]] = pa[[q, i]]
    low, up = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    assert np.abs(low).max() <= 1.0 + 1e-14
    # gamma of a complex elimination: at most n steps, 4 operations each, and the
    # product below likewise
    assert (np.abs(low @ up - pa) <= 8 * n * 2.0 ** -53 * (np.abs(low) @ np.abs(up))).all()


def test_silent_peer_times_out_and_handle_recovers(dev):
    """One CTA of the first panel sends no candidate: the others give up after
    about a second, the solve that follows reports TMVG_TIMEOUT, the interchanges
    written are valid row numbers, and the next factorisation is right."""
    import torch

    from tmv_gb300 import TmvgError, linalg

    rng = np.random.default_rng(5)
    n = 200
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    b = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    A, B = linalg.colmajor(torch.from_numpy(a).to(dev)), linalg.colmajor(torch.from_numpy(b).to(dev))
    h = linalg.handle(dev.index or 0)
    h.check(h.call("tmvg_test_set_silent", 1), "test_set_silent")
    try:
        P = linalg.lu_decompose_z(A.t().clone().t())
        p = P.cpu().numpy()
        with pytest.raises(TmvgError) as ei:
            linalg.lu_ldiveq_z(A, torch.arange(n, device=dev), B.t().clone().t())
    finally:
        h.check(h.call("tmvg_test_set_silent", 0), "test_set_silent")
    assert ei.value.status == 5  # TMVG_TIMEOUT
    assert ((p >= np.arange(n)) & (p < n)).all()
    LU, X = A.t().clone().t(), B.t().clone().t()
    P = linalg.lu_decompose_z(LU)
    linalg.lu_ldiveq_z(LU, P, X)
    x = X.cpu().numpy()
    assert np.abs(a @ x - b).max() <= 1e-13 * np.abs(a).sum(axis=1).max() * np.abs(x).max()
