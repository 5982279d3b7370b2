"""CQ_ACT_Q8_1 batches of 33 rows and more (f16 products per weight block, scaled in f32): the edges of its tiles (128 weight
rows, 64 / 128 batch rows, chunks of 256 k, shares that cut a tile) against the oracle of the reference's CUDA arithmetic, and
operands that the tensor core does not take against the integer dots of smaller batches."""
import ctypes as C

import numpy as np
import pytest

from candy_b200 import abi
from candy_b200.backend import ACT_Q8_1, CudaDevice, QStorage
from oracle import oracle_c as oc

pytestmark = pytest.mark.gpu
QT_ORDERS = [(oc.Q4_0, 0), (oc.Q4_0, 1), (oc.Q8_0, 0)]


def call(device, qt, order, x, blocks, n, bias=None, ldy=None, integer=False):
    m, k = x.shape
    ldy = ldy or n
    qs = QStorage.from_blocks(device, qt, order, n, k, blocks)
    xd, yd = device.storage_from_slice(x), device.storage_from_slice(np.full((m, ldy), -77.0, dtype=np.float32))
    bd = device.storage_from_slice(bias) if bias is not None else None
    device.set_option("split_min_rows_q8_1", 0 if integer else 33)
    try:
        st = device._lib.cq_qlinear(device.ctx, qt, order, ACT_Q8_1, xd.ptr, m, k, k, qs.buf.ptr, n, bd.ptr if bd else None, yd.ptr, ldy)
    finally:
        device.set_option("split_min_rows_q8_1", 33)
    abi.check(device.ctx, st, "linear")
    device.synchronize()
    y = yd.data().reshape(m, ldy)
    assert (y[:, n:] == -77.0).all()
    return y[:, :n]


def terms(qt, order, x, blocks, n):
    """sum over blocks of |term| per result, by which f32 additions round: at most (blocks + 4) 2^-24 of it."""
    k = x.shape[1]
    w = np.abs(oc.dequantize(qt, order, blocks.reshape(-1)).reshape(n, k).astype(np.float64))
    return np.abs(x).astype(np.float64) @ w.T


@pytest.mark.parametrize("qt,order", QT_ORDERS)
@pytest.mark.parametrize("m,n,k", [(33, 1, 256), (64, 127, 512), (65, 128, 768), (128, 129, 256), (129, 700, 2304), (300, 2000, 512), (70, 9000, 1024),
                                   (40, 300, 8192)])
def test_edges(device, qt, order, m, n, k):
    rng = np.random.default_rng(m + n + k + order)
    blocks = oc.quantize(qt, order, (rng.standard_normal((n, k)) * 0.02).astype(np.float32))
    x = (rng.standard_normal((m, k)) * 10.0 ** rng.uniform(-3, 3, (m, 1))).astype(np.float32)  # rows of very different size
    x[m // 2], x[0, :32] = 0.0, 0.0
    bias = rng.standard_normal(n).astype(np.float32) if n > 200 else None
    y = call(device, qt, order, x, blocks, n, bias, n + 3)
    want = oc.qmatmul(qt, order, x, blocks, n, nthreads=8, q8_1=True).astype(np.float64) + (bias if bias is not None else 0.0)
    bound = (k // 32 + 4) * 2.0 ** -23 * terms(qt, order, x, blocks, n) + 2.0 ** -23 * np.abs(want)  # both sides round
    assert (np.abs(y - want) <= bound).all()
    assert (y == call(device, qt, order, x, blocks, n, bias, n + 3)).all()


@pytest.mark.parametrize("qt,order", QT_ORDERS)
def test_operands_outside_f16(device, qt, order):
    """Blocks far below their row's largest value, rows at f16's limits, infinities and NaNs, and such weight scales: what the
    integer dots give, in every other row and column the same bits as without them."""
    m, n, k = 70, 300, 512
    rng = np.random.default_rng(order + qt)
    blocks = oc.quantize(qt, order, (rng.standard_normal((n, k)) * 0.02).astype(np.float32)).reshape(n, k // 32, -1)
    x = rng.standard_normal((m, k)).astype(np.float32)
    clean = call(device, qt, order, x, blocks.reshape(-1), n)
    x[1, 64:96] *= 2.0 ** -18
    x[2, 64:96] *= 2.0 ** -24
    x[3, 7], x[4] = 1e9, x[4] * 1e-6
    x[5], x[6] = x[5] * 1e-9, np.abs(x[6]) * 3e-6
    x[7, 9], x[8, 9], x[9, 9] = np.inf, np.nan, 9e6
    x[10, 32:64] = np.abs(x[10, 32:64]) * 4e3
    hurt = blocks.copy()
    hurt[17, 3, :2] = np.array([0x7C00], dtype=np.uint16).view(np.uint8)
    hurt[130, 0, :2] = np.array([0x7E01], dtype=np.uint16).view(np.uint8)
    hurt[299, 5, :2] = np.array([0x7BFF], dtype=np.uint16).view(np.uint8)
    y = call(device, qt, order, x, hurt.reshape(-1), n)
    want = call(device, qt, order, x, hurt.reshape(-1), n, integer=True)
    rows, cols = np.arange(11, m), np.setdiff1d(np.arange(n), [17, 130, 299])
    assert (y[np.ix_(rows, cols)] == clean[np.ix_(rows, cols)]).all()
    assert (np.isfinite(y) == np.isfinite(want)).all()
    f = np.isfinite(want)
    assert (np.isnan(y) == np.isnan(want)).all() and (y[np.isinf(want)] == want[np.isinf(want)]).all()
    t = terms(qt, order, np.nan_to_num(x, posinf=0.0), blocks.reshape(-1), n)
    t[:, 299] = terms(qt, order, np.nan_to_num(x, posinf=0.0), hurt[299:].reshape(-1), 1)[:, 0]
    bound = (k // 32 + 4) * 2.0 ** -23 * t + 2.0 ** -23 * np.abs(want)
    assert (np.abs(y - want)[f] <= bound[f]).all()


@pytest.mark.parametrize("qt,order", QT_ORDERS)
@pytest.mark.parametrize("m,k", [(40, 512), (128, 28672)])
def test_small_blocks_beside_large_ones(device, qt, order, m, k):
    """Blocks of 2^0 .. 2^-12 in rows whose others reach 2^12 (Q4_0, whose blocks' sums f16 has to hold) or 2^20, through weights
    that see nothing else: a block's own product is exact, so d8 and two roundings in f32 are all that there is.  And with all
    weights, every row of the batch like that, 28672 values long."""
    n = 260
    rng = np.random.default_rng(k + qt + order)
    blocks = oc.quantize(qt, order, (rng.standard_normal((n, k)) * 0.02).astype(np.float32)).reshape(n, k // 32, -1)
    x = (rng.standard_normal((m, k)) * (2.0 ** 10 if qt == oc.Q4_0 else 2.0 ** 20)).astype(np.float32)
    x[:, 64:96] = rng.standard_normal((m, 32)) * 2.0 ** -(np.arange(m) % 13)[:, None]
    only = np.zeros_like(blocks)
    only[:, 2] = blocks[:, 2]
    y, want = (call(device, qt, order, x, only.reshape(-1), n, integer=i) for i in (False, True))
    assert (np.abs(want).max(1) > 0.0).all()
    assert (np.linalg.norm(y - want, axis=1) <= 2.0 ** -21 * np.linalg.norm(want, axis=1)).all()
    y, want = (call(device, qt, order, x, blocks.reshape(-1), n, integer=i) for i in (False, True))
    assert (np.abs(y - want) <= (k // 32 + 4) * 2.0 ** -23 * terms(qt, order, x, blocks, n) + 2.0 ** -23 * np.abs(want)).all()


@pytest.mark.parametrize("qt,order", QT_ORDERS)
def test_every_row_outside_f16(device, qt, order):
    """A d8 or s8 in every row of a full tile that f16 does not hold, in several pieces of k: the infinities of
    the integer dots, and nothing that any wait in the kernel runs out over."""
    m, n, k = 128, 300, 40960
    rng = np.random.default_rng(order)
    blocks = oc.quantize(qt, order, (rng.standard_normal((n, k)) * 0.02).astype(np.float32))
    x = rng.standard_normal((m, k)).astype(np.float32)
    x[np.arange(m), rng.integers(0, k, m)] = np.where(np.arange(m) % 2, 9e6, -9e6)
    y, want = (call(device, qt, order, x, blocks, n, integer=i) for i in (False, True))
    assert np.array_equal(np.isnan(y), np.isnan(want)) and np.array_equal(y[np.isinf(want)], want[np.isinf(want)])
    assert not np.isfinite(y).any() and not np.isfinite(want).any()


@pytest.mark.parametrize("qt", [oc.Q4_0, oc.Q8_0])
@pytest.mark.parametrize("m,n,k,room", [
    (1000, 300, 8192, lambda m, k: 5 * m * k // 4 + (20 << 20)),                      # what the integer dots need: they serve it
    (100, 2000, 4096, lambda m, k: 4 * m * k + m * k // 4 + 4 * m + (4 << 10)),       # the operands, no partial tiles: whole tiles
])
def test_captured_with_little_scratch(qt, m, n, k, room):
    dev = CudaDevice(0)
    rng = np.random.default_rng(m)
    blocks = oc.quantize(qt, 0, (rng.standard_normal((n, k)) * 0.02).astype(np.float32))
    x = rng.standard_normal((m, k)).astype(np.float32)
    qs, xd, yd = QStorage.from_blocks(dev, qt, 0, n, k, blocks), dev.storage_from_slice(x), dev.zeros(m * n)
    lib, ctx = dev._lib, dev.ctx
    call_it = lambda: abi.check(ctx, lib.cq_qmatmul(ctx, qt, 0, ACT_Q8_1, xd.ptr, m, k, k, qs.buf.ptr, n, yd.ptr, n), "matmul")  # noqa: E731
    abi.check(ctx, lib.cq_reserve(ctx, room(m, k)), "reserve")
    g = C.c_void_p()
    abi.check(ctx, lib.cq_capture_begin(ctx), "begin")
    try:
        call_it()
    finally:
        abi.check(ctx, lib.cq_capture_end(ctx, C.byref(g)), "end")
    abi.check(ctx, lib.cq_memset(ctx, yd.ptr, 0, 4 * m * n), "clear")
    abi.check(ctx, lib.cq_graph_launch(ctx, g), "launch")
    got = yd.data().reshape(m, n)
    lib.cq_graph_destroy(ctx, g)
    rows = np.unique(np.linspace(0, m - 1, 40).astype(int))
    want = oc.qmatmul(qt, 0, x[rows], blocks, n, nthreads=8, q8_1=True).astype(np.float64)
    assert (np.abs(got[rows] - want) <= (k // 32 + 4) * 2.0 ** -23 * terms(qt, 0, x[rows], blocks, n)).all()
    dev.set_option("split_min_rows_q8_1", 0)
    call_it()
    integer = yd.data().reshape(m, n)
    assert np.array_equal(got, integer) == (m == 1000)
    del qs, xd, yd
    dev.close()
