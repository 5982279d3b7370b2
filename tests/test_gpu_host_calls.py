"""cq_qlinear_host: pageable and page-locked buffers, with and without a bias, around the sizes where its ways part (one, eight
and nine rows, 256 KiB and a megabyte of input or result): the bits of the same call on device buffers."""
import ctypes as C

import numpy as np
import pytest

from candy_b200 import abi
from candy_b200.backend import QLinear, QStorage

pytestmark = pytest.mark.gpu


def pinned(device, shape):
    p = C.c_void_p()
    abi.check(device.ctx, device._lib.cq_malloc_host(device.ctx, 4 * int(np.prod(shape)), C.byref(p)), "pinned")
    return p, np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_float)), shape=shape)


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("qt", [abi.Q4_0, abi.Q8_0])
@pytest.mark.parametrize("m,n,k", [(1, 64, 32), (1, 4096, 256), (8, 8192, 256), (8, 8193, 256), (9, 300, 512), (64, 4096, 256), (65, 4096, 256),
                                   (1024, 40, 256), (1025, 40, 256)])
def test_same_bits_as_on_the_device(device, qt, m, n, k, bias):
    rng = np.random.default_rng(m + n)
    w = QStorage.quantize(device, qt, 0, (rng.standard_normal((n, k)) * 0.02).astype(np.float32))
    x, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    lib, ctx = device._lib, device.ctx
    xd, bd, yd = device.storage_from_slice(x), device.storage_from_slice(b) if bias else None, device.zeros(m * n)
    abi.check(ctx, lib.cq_qlinear(ctx, qt, 0, 0, xd.ptr, m, k, k, w.buf.ptr, n, bd.ptr if bias else None, yd.ptr, n), "linear")
    want = yd.data().reshape(m, n)
    (px, vx), (py, vy) = pinned(device, (m, k)), pinned(device, (m, n))
    vx[:] = x
    try:
        for src in (x.ctypes.data, px):
            y = np.full((m, n), np.nan, dtype=np.float32)
            vy[:] = np.nan
            for dst, got in ((y.ctypes.data, y), (py, vy)):
                abi.check(ctx, lib.cq_qlinear_host(ctx, qt, 0, 0, src, m, k, w.buf.ptr, n, bd.ptr if bias else None, dst), "host")
                assert np.array_equal(got, want)
    finally:
        lib.cq_free_host(ctx, px)
        lib.cq_free_host(ctx, py)
    lin = QLinear(w, b if bias else None)
    for _ in range(2):
        assert np.array_equal(lin.forward(x), want)
    assert np.array_equal(lin.forward(x[:, None]).reshape(m, n), want)
    with pytest.raises(abi.CandyqError):  # bad arguments are refused before anything is copied
        abi.check(ctx, lib.cq_qlinear_host(ctx, qt, 0, 0, x.ctypes.data, 0, k, w.buf.ptr, n, None, y.ctypes.data), "host")
