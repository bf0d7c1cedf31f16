"""Quotients next to a midpoint of two doubles through the batched band kernels, bit
for bit against the division on the host.

For a divisor with the odd significand B the numerator with a / b = midpoint +-
1 / (2 B) ulps (the nearest a quotient can lie) is found from the inverse of B
modulo 2^53 or 2^54; divisors are random, just below the bound at which the kernels
divide (b = 2 - 2^-13), around it, and such that 1 / b itself lies next to a
midpoint."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _divisors(rng, count):
    """Odd significands in [2^52, 2^53), as integers."""
    out = []
    for _ in range(count // 4):
        out.append(int(rng.integers(1 << 52, 1 << 53)))
        out.append((1 << 53) - int(rng.integers(1 << 39, 1 << 41)))  # 2 - 2^-13 and its surroundings
        out.append((1 << 53) - int(2 ** rng.uniform(1, 45)))
        while True:  # 2^105 / B within 2^-10 of a midpoint
            b = int(rng.integers(1 << 52, 1 << 53)) | 1
            r = (1 << 105) % b
            if abs(2 * r - b) * 1024 < b:
                break
        out.append(b)
    return [b | 1 for b in out]


def _hard_numerators(b):
    for t in (53, 54):
        inv = pow(b, -1, 1 << t)
        for k in (1, -1):
            n = (-k * inv) % (1 << t) + ((1 << 53) if t == 53 else 0)
            if (1 << 53) <= n < (1 << 54):
                a = (n * b + k) >> t
                if (1 << 52) <= a < (1 << 53):
                    yield a


@pytest.mark.parametrize("algo", ["tridiag", "general"])
def test_quotients_next_to_midpoints(dev, orc, algo):
    from test_gpu_band import compare, gpu_batch, oracle_batch
    from tmv_gb300.band import band_layout

    rng = np.random.default_rng(3)
    pairs = [(a, b) for b in _divisors(rng, 4000) for a in _hard_numerators(b)]
    count, n = len(pairs), 2
    lay = band_layout(n, 1, 1)
    a, b = (np.array([p[q] for p in pairs], float) * 2.0 ** rng.integers(-200, 200, count) for q in (0, 1))
    ab = np.zeros(count * lay.stride_ab)
    at = np.arange(count) * lay.stride_ab
    # x0 = a / b, and l = 2^e / b: a quotient of its own (tridiagonal algorithm) or
    # the rounded reciprocal's bits (general algorithm)
    ab[at], ab[at + 1] = b, 2.0 ** (np.frexp(b)[1] - 1)
    ab[at + lay.ldab + 1] = 1.0
    rhs = np.zeros(count * n)
    rhs[::2] = a
    compare(lay, count, 1, gpu_batch(dev, lay, ab, rhs, count, 1, algo), oracle_batch(orc, lay, ab, rhs, count, 1, algo),
            ab)
    assert count > 3000
