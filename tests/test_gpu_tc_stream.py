"""The streamed 3xTF32 update (C by TMA) against the direct one.

The two issue the same products in the same order and subtract once, so they
agree to the bit; a C whose column stride is not a multiple of 16 bytes takes
the direct kernel.
"""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _update(h, a, b, c):
    h.check(h.call("tmvg_gemm_f32_tf32x3", c.shape[0], c.shape[1], a.shape[1], C.c_void_p(a.data_ptr()),
                   a.stride(1), C.c_void_p(b.data_ptr()), b.stride(1), C.c_void_p(c.data_ptr()), c.stride(1)),
            "tf32x3")


# one tile; ragged rows and columns; a second half of no columns; runs of tiles
# that cross columns of tiles; more than two tiles a CTA; K of one chunk
@pytest.mark.parametrize("m,n,k", [(128, 128, 64), (127, 129, 64), (260, 190, 32), (1000, 777, 64),
                                   (300, 20000, 64), (20000, 300, 32), (4100, 4097, 64)])
def test_streamed_update_matches_direct(dev, m, n, k):
    import torch

    from tmv_gb300 import linalg

    g = torch.Generator(device=dev).manual_seed(m + 3 * n + k)
    col = lambda r, c, ld: torch.randn(c, ld, device=dev, generator=g).t()[:r]  # noqa: E731
    a, b = col(m, k, m), col(k, n, k)
    ld = (m + 3) // 4 * 4
    c1 = col(m, n, ld + 4)
    c2 = torch.empty(n, ld + 1, device=dev).t()[:m]
    c2.copy_(c1)
    pad = c1.t().as_strided((n, 4), (ld + 4, 1), ld).clone()
    h = linalg.handle(dev.index)
    _update(h, a, b, c1)
    _update(h, a, b, c2)
    torch.cuda.synchronize()
    assert torch.equal(c1, c2)
    assert torch.equal(c1.t().as_strided((n, 4), (ld + 4, 1), ld), pad)  # below the matrix untouched
