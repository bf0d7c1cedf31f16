"""The published entries of the sync-free solves, FP64 and FP32 on one handle: what
an FP64 solve leaves in the words must never read as an FP32 entry of a later
launch, whatever its value.  The FP64 solution here has the later launches' numbers
in its upper halves (subnormals), and 1e30 as an FP32 number in its lower ones."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("launch", [2, 3])  # the solve with L is the handle's second launch, with U the third
def test_fp64_entries_are_no_fp32_entries(dev, launch):
    import torch
    from helpers import to_dev

    from tmv_gb300 import _lib

    h = _lib.Handle(dev.index or 0)
    h.set_stream(torch.cuda.current_stream().cuda_stream)
    n = 192
    bits = (np.int64(launch) << 32) | np.int64(np.float32(1e30).view(np.int32))
    b = np.full((n, 1), bits).view(np.float64)
    T, B = to_dev(np.eye(n), dev), to_dev(b, dev)
    h.check(h.call("tmvg_tri_ldiveq_f64", 0, 1, n, C.c_void_p(T.data_ptr()), 1, n, 1, C.c_void_p(B.data_ptr()), 1, n))
    assert (B.cpu().numpy().view(np.int64) == bits).all()
    rng = np.random.default_rng(0)
    lu = np.asfortranarray(rng.uniform(-0.05, 0.05, (n, n)) + 2.0 * np.eye(n), dtype=np.float32)
    piv = np.arange(n)
    x = np.asfortranarray(rng.standard_normal((n, 1)), dtype=np.float32)
    rhs = x.astype(np.float64)
    h.check(h.call("tmvg_lu_ldiveq_f32_host", n, C.c_void_p(lu.ctypes.data), n, C.c_void_p(piv.ctypes.data), 1,
                   C.c_void_p(x.ctypes.data), 1, n))
    low, up = np.tril(lu, -1).astype(np.float64) + np.eye(n), np.triu(lu).astype(np.float64)
    # two triangles, n steps each, in FP32
    size = np.abs(low) @ (np.abs(up) @ np.abs(x))
    assert (np.abs(low @ (up @ x.astype(np.float64)) - rhs) <= 3 * n * 2.0 ** -24 * size).all()
