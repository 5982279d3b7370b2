"""The small kernels around a layer's linears at the edges of their vector forms: odd sizes, strides and addresses that take the
element-by-element ways, and rows too long for a thread block to keep.  Moves are exact; sums and SiLU against f64."""
import numpy as np
import pytest

from candy_b200 import abi
from candy_b200.backend import RawBuffer
from oracle import attention_np as an

pytestmark = pytest.mark.gpu


def at(storage, floats):
    """A device address `floats` 4-byte words into a buffer."""
    return storage.ptr.value + 4 * floats


@pytest.mark.parametrize("rows,n,ld,shift", [(1, 1, 1, 0), (3, 7, 7, 0), (5, 512, 513, 0), (4, 514, 514, 2), (2, 1030, 1032, 0), (3, 1028, 1028, 1), (70000, 6, 8, 0)])
def test_silu_mul_pairs(device, rows, n, ld, shift):
    """`shift`: the pairs 8 bytes off a 16-byte boundary (2), the outputs 4 bytes off an 8-byte one (1)."""
    rng = np.random.default_rng(rows + n)
    gu = (4 * rng.standard_normal((rows, n, 2))).astype(np.float32)
    src = device.storage_from_slice(np.concatenate([np.zeros(2, np.float32), gu.ravel()]) if shift == 2 else gu.ravel())
    out = device.storage_from_slice(np.full(rows * ld + 1, -7.0, dtype=np.float32))
    abi.check(device.ctx, device._lib.cq_silu_mul_pairs(device.ctx, at(src, 2 if shift == 2 else 0), rows, n, at(out, int(shift == 1)), ld), "silu")
    got = out.data()[int(shift == 1):][:rows * ld].reshape(rows, ld)
    g = gu[..., 0].astype(np.float64)
    want = (g / (1.0 + np.exp(-g))).astype(np.float32) * gu[..., 1]
    assert np.abs(got[:, :n] - want).max() <= 2.0 ** -22 * np.abs(want).max()  # two roundings, and numpy's exp beside the device's
    assert (got[:, n:] == -7.0).all()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("count,src_off,dst_off", [(1, 0, 0), (3, 0, 0), (4, 0, 0), (4099, 0, 0), (4096, 1, 0), (4098, 0, 1), (300001, 8, 4)])
def test_cast16_to_f32(device, count, src_off, dst_off, bf16):
    bits = np.random.default_rng(count).standard_normal(count + src_off).astype(np.float32)
    bits = an.to_bf16_bits(bits) if bf16 else bits.astype(np.float16).view(np.uint16)
    src, dst = device.upload_bytes(bits), device.storage_from_slice(np.full(count + dst_off + 1, -7.0, dtype=np.float32))
    abi.check(device.ctx, device._lib.cq_cast16_to_f32(device.ctx, src.ptr.value + 2 * src_off, count, int(bf16), at(dst, dst_off)), "cast")
    want = an.from_bf16_bits(bits) if bf16 else bits.view(np.float16).astype(np.float32)
    got = dst.data()
    assert np.array_equal(got[dst_off:dst_off + count], want[src_off:]) and (got[:dst_off] == -7.0).all() and got[-1] == -7.0


@pytest.mark.parametrize("dim,table_off,out_off", [(4096, 0, 0), (12, 0, 0), (10, 0, 0), (257, 0, 0), (64, 1, 0), (64, 0, 2)])
def test_embedding(device, dim, table_off, out_off):
    table = np.random.default_rng(dim).standard_normal(50 * dim + table_off).astype(np.float32)
    ids = np.array([0, 49, 7, 7, 1000], dtype=np.uint32)  # the last one is beyond the table: its last row
    d_table, d_ids, out = device.storage_from_slice(table), device.upload_bytes(ids), device.zeros(ids.size * dim + out_off)
    abi.check(device.ctx, device._lib.cq_embedding(device.ctx, at(d_table, table_off), 50, dim, d_ids.ptr, ids.size, at(out, out_off)), "embedding")
    assert np.array_equal(out.data()[out_off:].reshape(ids.size, dim), table[table_off:].reshape(50, dim)[np.minimum(ids, 49)])


@pytest.mark.parametrize("add", [False, True])
@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 33), (2, 1000), (2, 4096), (5, 8192), (3, 8193), (2, 20000)])
def test_rmsnorm(device, rows, cols, add):
    rng = np.random.default_rng(cols)
    x, delta, alpha = rng.standard_normal((rows, cols)).astype(np.float32), rng.standard_normal((rows, cols)).astype(np.float32), rng.standard_normal(cols).astype(np.float32)
    for weights in (alpha, None):
        dx, dd, da, y = device.storage_from_slice(x), device.storage_from_slice(delta), device.storage_from_slice(alpha), device.zeros(rows * cols)
        a = da.ptr if weights is not None else None
        if add:
            st = device._lib.cq_add_rmsnorm(device.ctx, dx.ptr, dd.ptr, a, rows, cols, 1e-5, y.ptr)
        else:
            st = device._lib.cq_rmsnorm(device.ctx, dx.ptr, a, rows, cols, 1e-5, y.ptr)
        abi.check(device.ctx, st, "rmsnorm")
        got, after = y.data().reshape(rows, cols), dx.data().reshape(rows, cols)
        v = x + delta if add else x
        assert np.array_equal(after, v)
        want = v / np.sqrt((v.astype(np.float64) ** 2).mean(1, keepdims=True) + 1e-5) * (1.0 if weights is None else weights)
        assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()  # the sum is added up in a tree: a few roundings of f32


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("hd,shift", [(128, 0), (64, 1), (12, 0), (20, 0), (6, 0), (2, 0), (8, 0)])
def test_rope_prefill(device, hd, shift, bf16):
    """Head dimensions that are not multiples of eight, and a qkv 4 bytes off a 16-byte boundary (`shift`)."""
    lib, ctx, T, nq, nkv, max_ctx, pos0 = device._lib, device.ctx, 5, 3, 1, 9, 2
    rng = np.random.default_rng(hd)
    ang = rng.uniform(0, 6.28, size=(max_ctx, hd // 2))
    cos, sin = np.cos(ang).astype(np.float32), np.sin(ang).astype(np.float32)
    qkv = rng.standard_normal((T, nq + 2 * nkv, hd)).astype(np.float32)
    d_qkv = device.storage_from_slice(np.concatenate([np.zeros(shift, np.float32), qkv.ravel()]))
    d_cos, d_sin = device.storage_from_slice(cos), device.storage_from_slice(sin)
    kc, vc = (device.storage_from_slice(np.full(max_ctx * nkv * hd, -7.0, dtype=np.float32)) for _ in range(2))
    q16, k16, v16 = (RawBuffer(device, 2 * T * heads * hd) for heads in (nq, nkv, nkv))
    st = lib.cq_rope_prefill(ctx, at(d_qkv, shift), T, nq, nkv, hd, d_cos.ptr, d_sin.ptr, pos0, kc.ptr, vc.ptr, max_ctx, q16.ptr, k16.ptr, v16.ptr, int(bf16))
    abi.check(ctx, st, "rope prefill")
    x = qkv[:, :nq + nkv].astype(np.float64)
    c, s = cos[pos0:pos0 + T, None].astype(np.float64), sin[pos0:pos0 + T, None].astype(np.float64)
    lo, hi = x[..., :hd // 2], x[..., hd // 2:]
    want = np.concatenate([lo * c - hi * s, lo * s + hi * c], -1)
    got_k, got_v = (a.data().reshape(max_ctx, nkv, hd) for a in (kc, vc))
    inside = slice(pos0, pos0 + T)
    assert np.abs(got_k[inside] - want[:, nq:]).max() <= 2.0 ** -22 * np.abs(want).max() and np.array_equal(got_v[inside], qkv[:, nq + nkv:])
    for a in (got_k, got_v):
        assert (a[:pos0] == -7.0).all() and (a[pos0 + T:] == -7.0).all()
    bits = lambda a: an.to_bf16_bits(a) if bf16 else a.astype(np.float16).view(np.uint16)  # noqa: E731
    assert np.array_equal(k16.data().view(np.uint16).reshape(T, nkv, hd), bits(got_k[inside]))
    assert np.array_equal(v16.data().view(np.uint16).reshape(T, nkv, hd), bits(qkv[:, nq + nkv:]))
    q = q16.data().view(np.uint16).reshape(T, nq, hd)
    q = an.from_bf16_bits(q) if bf16 else q.view(np.float16).astype(np.float32)
    assert np.abs(q - want[:, :nq]).max() <= 2.0 ** (-8 if bf16 else -11) * np.abs(want).max()
