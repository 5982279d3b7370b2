"""Grouped-query decode attention at the edges of its rounds (8 keys a warp, 32 a CTA) and splits, every group size, with rows
past the position that must not be read into the result; f64 oracle, 2e-6 of the largest output for 32-bit sums of a few hundred
terms."""
import numpy as np
import pytest

from candy_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rope", [False, True])
@pytest.mark.parametrize("batch,nkv,G,max_ctx,positions", [
    (1, 1, 2, 40, (0, 6, 7, 8, 9)), (2, 2, 3, 200, (30, 31, 32, 33, 199)), (1, 4, 8, 520, (63, 64, 255, 519)), (3, 2, 5, 70, (1, 69)), (40, 8, 4, 100, (99,)),
    (1, 2, 2, 4100, (0, 40, 1500, 4099)), (20, 8, 2, 150, (0, 149)),
])
def test_rounds_and_splits(device, batch, nkv, G, max_ctx, positions, rope):
    lib, ctx, hd = device._lib, device.ctx, 128
    nq = nkv * G
    rng = np.random.default_rng(max_ctx)
    ang = rng.uniform(0, 6.28, size=(max_ctx, hd // 2))
    cos, sin = np.cos(ang).astype(np.float32), np.sin(ang).astype(np.float32)
    d_cos, d_sin = device.storage_from_slice(cos), device.storage_from_slice(sin)
    scratch, out = device.alloc(lib.cq_decode_attention_scratch_floats(batch, nq, hd, max_ctx)), device.alloc(batch * nq * hd)
    for pos in positions:
        qkv = rng.standard_normal((batch, nq + 2 * nkv, hd)).astype(np.float32)
        kc, vc = (rng.standard_normal((batch, max_ctx, nkv, hd)).astype(np.float32) for _ in range(2))
        kc[:, pos + 1:], vc[:, pos + 1:] = np.nan, np.inf
        q, k, v = qkv[:, :nq].astype(np.float64), kc.astype(np.float64), vc.astype(np.float64)
        if rope:
            def turn(a):
                lo, hi = a[..., :hd // 2], a[..., hd // 2:]
                return np.concatenate([lo * cos[pos] - hi * sin[pos], lo * sin[pos] + hi * cos[pos]], -1)
            kc[:, pos], vc[:, pos] = np.nan, np.nan  # not there yet
            q, k[:, pos], v[:, pos] = turn(q), turn(qkv[:, nq:nq + nkv].astype(np.float64)), qkv[:, nq + nkv:]
        s = np.einsum("bhgd,bthd->bhgt", q.reshape(batch, nkv, G, hd), k[:, :pos + 1]) / np.sqrt(hd)
        p = np.exp(s - s.max(-1, keepdims=True))
        want = np.einsum("bhgt,bthd->bhgd", p / p.sum(-1, keepdims=True), v[:, :pos + 1]).reshape(batch, nq, hd)
        d_qkv, d_k, d_v = device.storage_from_slice(qkv), device.storage_from_slice(kc), device.storage_from_slice(vc)
        d_pos = device.upload_bytes(np.array([pos], dtype=np.int32))
        if rope:
            st = lib.cq_decode_attention_rope(ctx, d_qkv.ptr, batch, nq, nkv, hd, d_cos.ptr, d_sin.ptr, d_pos.ptr, d_k.ptr, d_v.ptr, max_ctx, scratch.ptr, out.ptr)
        else:
            st = lib.cq_decode_attention(ctx, d_qkv.ptr, batch, nq, nkv, hd, d_pos.ptr, d_k.ptr, d_v.ptr, max_ctx, scratch.ptr, out.ptr)
        abi.check(ctx, st, "attention")
        got = out.data().reshape(batch, nq, hd)
        assert np.abs(got - want).max() <= 2e-6 * np.abs(want).max()
        if rope:
            assert np.abs(d_k.data().reshape(kc.shape)[:, pos] - k[:, pos]).max() <= 1e-6 * np.abs(k[:, pos]).max()
            assert (d_v.data().reshape(vc.shape)[:, pos] == v[:, pos]).all()
