"""The quotients and reciprocals of the batched band kernels where their
short form ends: operands, results and significands at the edges, bit for bit
against the oracle (IEEE division on the host).

Diagonal-dominant systems of two unknowns make x = b / a one quotient per
entry; the factorisation adds l = a10 / a00 (tridiagonal algorithm) and
1 / a00 (general algorithm)."""
import numpy as np
import pytest

from test_gpu_band import compare, gpu_batch, oracle_batch

pytestmark = pytest.mark.gpu


def _values(rng, count):
    """Significands random, all ones, one, next to one; exponents over the
    whole range and at the ends of the short form's (biased 100 and 1945)."""
    m = rng.integers(0, 2**52, count)
    edge = rng.random(count)
    m[edge < 0.1] = 2**52 - 1
    m[(edge >= 0.1) & (edge < 0.2)] = 0
    m[(edge >= 0.2) & (edge < 0.3)] = 1
    e = rng.integers(1, 2046, count)
    near = rng.random(count)
    e[near < 0.5] = rng.integers(900, 1150, (near < 0.5).sum())
    e[(near >= 0.5) & (near < 0.6)] = rng.choice([99, 100, 101, 1944, 1945, 1946], ((near >= 0.5) & (near < 0.6)).sum())
    e[near >= 0.97] = 0
    s = rng.integers(0, 2, count)
    return ((s.astype(np.uint64) << np.uint64(63)) | (e.astype(np.uint64) << np.uint64(52)) | m.astype(np.uint64)).view(np.float64)


@pytest.mark.parametrize("algo", ["tridiag", "general"])
@pytest.mark.parametrize("nrhs", [1, 2])
def test_edges_bitwise(dev, orc, algo, nrhs):
    from tmv_gb300.band import band_layout

    rng = np.random.default_rng(17 + nrhs)
    count, n = 4000, 2
    lay = band_layout(n, 1, 1)
    ab = np.zeros(count * lay.stride_ab)
    d, low = _values(rng, 2 * count).reshape(count, 2), _values(rng, count)
    with np.errstate(all="ignore"):
        low = np.where(np.abs(low) > np.abs(d[:, 0]), low * 2.0 ** -rng.integers(0, 60, count), low)
    at = np.arange(count) * lay.stride_ab
    ab[at], ab[at + 1] = d[:, 0], low
    ab[at + lay.ldab], ab[at + lay.ldab + 1] = rng.standard_normal(count) * (rng.random(count) < 0.5), d[:, 1]
    B = _values(rng, count * n * nrhs)
    ref = oracle_batch(orc, lay, ab, B, count, nrhs, algo)
    compare(lay, count, nrhs, gpu_batch(dev, lay, ab, B, count, nrhs, algo), ref, ab)
