"""The packed tridiagonal kernel (32-byte groups, entries four at a time where
aligned) bit for bit against the oracle: lengths around its blocks of four,
strides that are and are not multiples of four, leading and trailing zeros of
b, zero and underflowing columns, singular systems, in place (band_lu_solve)
and into another buffer (band_divide)."""
import numpy as np
import pytest

from test_gpu_band import compare, make_batch, oracle_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 5, 6, 7, 8, 9, 63, 64, 257])
@pytest.mark.parametrize("kind", ["normal", "int", "tiny"])
@pytest.mark.parametrize("shift", [0, 1])
def test_bitwise(dev, orc, n, kind, shift):
    import torch

    from tmv_gb300.band import band_divide, band_lu_solve

    rng = np.random.default_rng(n + shift)
    count = 130
    lay, ab, B = make_batch(rng, count, n, 1, 1, kind, 1)
    for s in range(0, count, 7):  # zeros at b's ends; a zero column
        B[s * n + rng.integers(1, n):(s + 1) * n] = 0.0
        if s % 14 == 0:
            B[s * n:(s + 1) * n] *= np.arange(n) >= rng.integers(0, n + 1)
            j = int(rng.integers(0, n))
            for i in range(max(0, j - 1), min(n, j + 2)):
                ab[s * lay.stride_ab + i + j * lay.ldab] = 0.0
    ref = oracle_batch(orc, lay, ab, B, count, 1, "tridiag")
    assert ref[2].any()
    dab = torch.from_numpy(ab).to(dev)
    raw = torch.from_numpy(np.concatenate([np.zeros(shift), B])).to(dev)  # shift: b is not 32-byte aligned
    dB = raw[shift:]
    P, st = band_lu_solve(dab, count, lay, dB, 1, algo="tridiag")
    torch.cuda.synchronize()
    host = lambda t: t.cpu().numpy()  # noqa: E731
    compare(lay, count, 1, (host(dab), host(P).reshape(count, -1)[:, :n], host(st), host(dB)), ref, ab)
    # into a buffer of its own: A stays, only the factors' slots are written
    dab, lu = torch.from_numpy(ab).to(dev), torch.full((count * lay.stride_ab,), 7.0, dtype=torch.float64, device=dev)
    dB = torch.from_numpy(B).to(dev)
    _, _, P, st, _ = band_divide(dab, count, lay, dB, 1, lu=lu)
    torch.cuda.synchronize()
    assert np.array_equal(host(dab).view(np.int64), ab.view(np.int64))
    compare(lay, count, 1, (host(lu), host(P).reshape(count, -1)[:, :n], host(st), host(dB)), ref,
            np.full(count * lay.stride_ab, 7.0))
