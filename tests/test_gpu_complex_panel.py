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
