"""cq_quantize_rows at the edges of a CTA's 128 blocks, from and to addresses without 16-byte alignment: bytes equal the oracle's."""
import ctypes as C

import numpy as np
import pytest

from candy_b200 import abi
from oracle import oracle_c as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qt,order", [(oc.Q4_0, 0), (oc.Q4_0, 1), (oc.Q8_0, 0)])
@pytest.mark.parametrize("src_off,dst_off", [(0, 0), (4, 0), (0, 2), (4, 6)])
@pytest.mark.parametrize("nblocks", [1, 7, 127, 128, 129, 1000])
def test_quantize_edges(device, qt, order, src_off, dst_off, nblocks):
    rng = np.random.default_rng(nblocks)
    w = rng.standard_normal((1, nblocks * 32)).astype(np.float32)
    w[0, :32] = 0.0  # a block of zeros, and one with a tie of magnitudes
    if nblocks > 1:
        w[0, 40], w[0, 50] = -9.0, 9.0
    nbytes = nblocks * abi.BLOCK_BYTES[qt]
    src, dst = device.malloc(w.nbytes + src_off), device.malloc(nbytes + dst_off + 16)
    at = lambda p, off: C.c_void_p(p.value + off)  # noqa: E731
    lib, ctx = device._lib, device.ctx
    abi.check(ctx, lib.cq_memset(ctx, dst, 0xAB, nbytes + dst_off + 16), "fill")
    abi.check(ctx, lib.cq_memcpy_h2d(ctx, at(src, src_off), w.ctypes.data_as(C.c_void_p), w.nbytes), "in")
    abi.check(ctx, lib.cq_quantize_rows(ctx, qt, order, at(src, src_off), 1, nblocks * 32, at(dst, dst_off)), "quantize")
    out = np.empty(nbytes + dst_off + 16, dtype=np.uint8)
    abi.check(ctx, lib.cq_memcpy_d2h(ctx, out.ctypes.data_as(C.c_void_p), dst, out.nbytes), "out")
    device.free(src)
    device.free(dst)
    assert (out[dst_off:dst_off + nbytes] == oc.quantize(qt, order, w).reshape(-1)).all()
    assert (out[:dst_off] == 0xAB).all() and (out[dst_off + nbytes:] == 0xAB).all()
