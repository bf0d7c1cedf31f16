"""The clustered update of the next panel's columns while other work holds SMs.

Its CTAs write to one another's shared memory, which they may do once all of a
cluster have started; other streams' work makes them start at different times.
The factors have to be those of an idle device, bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [200, 700, 1500])
def test_factors_do_not_depend_on_other_streams(dev, n):
    import torch

    from tmv_gb300 import linalg

    g = torch.Generator(device=dev).manual_seed(n)
    A = linalg.colmajor(torch.randn(n, n, dtype=torch.float64, device=dev, generator=g))
    LU0 = A.t().clone().t()
    P0 = linalg.lu_decompose(LU0)
    busy = [torch.cuda.Stream() for _ in range(3)]
    x = torch.randn(1 << 22, dtype=torch.float64, device=dev, generator=g)
    out = []
    for _ in range(15):
        LU = A.t().clone().t()
        for q, s in enumerate(busy):
            with torch.cuda.stream(s):
                for _ in range(4 + 3 * q):
                    torch.sin(x[: 1 << (16 + 3 * q)])
        out.append((LU, linalg.lu_decompose(LU)))
    torch.cuda.synchronize()
    for LU, P in out:
        assert torch.equal(P, P0) and torch.equal(LU, LU0)
