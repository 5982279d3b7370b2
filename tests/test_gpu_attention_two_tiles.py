"""Prefill attention with two query tiles per CTA (cq_flash_attention, option fa_two_tiles = 2) against the CPU oracle, at the
edges of its tiles (256 query rows, 128 keys), where later key tiles raise a maximum, and on non-finite inputs against the kernel
with one tile.  Bars as for that kernel: the rounding of p to 16 bits (2^-9 in bf16, 2^-12 in f16) sets them."""
import ctypes as C

import numpy as np
import pytest

from candy_b200.backend import RawBuffer
from oracle import attention_np as an
from test_gpu_flash_attention import from16, run_case, to16

pytestmark = pytest.mark.gpu


@pytest.fixture
def two_tiles(device):
    device.set_option("fa_two_tiles", 2)
    yield device
    device.set_option("fa_two_tiles", 1)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("b,h,hk,sq,sk,d,bf16", [
    (1, 2, 2, 1, 1, 128, False), (1, 2, 1, 128, 127, 64, True), (1, 4, 2, 129, 128, 128, False), (2, 2, 2, 256, 129, 64, False),
    (1, 2, 1, 257, 300, 128, True), (1, 3, 3, 300, 70, 128, False), (1, 2, 2, 513, 700, 64, True), (1, 40, 8, 700, 700, 128, True),
    (2, 24, 24, 600, 200, 128, False), (1, 10, 2, 2048, 2048, 128, False),
])
def test_edges(two_tiles, b, h, hk, sq, sk, d, causal, bf16):
    err, lse_err = run_case(two_tiles, b, h, hk, sq, sk, d, causal, bf16)
    assert err <= (1.5e-2 if bf16 else 2e-3), err
    assert lse_err <= 2e-3, lse_err


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("d", [64, 128])
def test_several_items_per_cta(two_tiles, d, causal):
    """Two to three items for each CTA (2 x 64 heads x three pairs of query tiles on at most 148): the words through which the
    halves of a row exchange maxima and sums pass from item to item."""
    for _ in range(3):
        err, lse_err = run_case(two_tiles, 2, 64, 8, 600, 300, d, causal, True)
        assert err <= 1.5e-2 and lse_err <= 2e-3, (err, lse_err)


def test_packed_strides(two_tiles):
    err, lse_err = run_case(two_tiles, 2, 4, 2, 384, 384, 128, True, False, packed=True)
    assert err <= 2e-3 and lse_err <= 2e-3


def attend(device, q, k, v, scale, causal, bf16, option):
    b, sq, h, d = q.shape
    sk, hk = k.shape[1:3]
    dq, dk, dv = (device.upload_bytes(to16(a, bf16)) for a in (q, k, v))
    out, lse = RawBuffer(device, b * sq * h * d * 2), device.zeros(b * h * sq)
    device.set_option("fa_two_tiles", option)
    st = device._lib.cq_flash_attention(
        device.ctx, *(C.c_void_p(a.ptr.value) for a in (dq, dk, dv)), out.ptr, lse.ptr, None, None, None, sq * h * d, sk * hk * d, sk * hk * d, sq * h * d, 0,
        h * d, hk * d, hk * d, h * d, d, d, d, d, b, h, hk, d, d, scale, sq, sk, -(-sq // 128) * 128, -(-sk // 128) * 128, int(bf16), int(causal), 0, -1, -1, 0.0)
    device.set_option("fa_two_tiles", 1)
    assert st == 0, device._lib.cq_last_error(device.ctx)
    device.synchronize()
    return from16(out.data().view(np.uint16).reshape(b, sq, h, d), bf16), lse.data().reshape(b, h, sq)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("growth", [3.0, 30.0, 300.0])
def test_scores_that_grow_from_tile_to_tile(device, growth, causal, bf16):
    """Every key tile's scores lie about `growth` above the last one's, in some rows only: new maxima and rescaled sums."""
    rng = np.random.default_rng(int(growth))
    sq, sk, d = 300, 600, 128
    q, k, v = (rng.standard_normal((1, s, h, d)).astype(np.float32) for s, h in ((sq, 4), (sk, 2), (sk, 2)))
    q[:, ::3, :, 0], k[..., 0] = 8.0, (np.arange(sk) // 128 * growth / 8.0 * np.sqrt(d))[None, :, None]
    q, k, v = (from16(to16(a, bf16), bf16) for a in (q, k, v))
    want, want_lse = an.mha_forward(q, k, v, 1.0 / np.sqrt(d), causal)
    got, lse = attend(device, q, k, v, 1.0 / np.sqrt(d), causal, bf16, 2)
    assert np.abs(got - want).max() <= (1.5e-2 if bf16 else 2e-3) * np.abs(want).max()
    fin = np.isfinite(want_lse)
    assert np.abs(lse[fin] - want_lse[fin]).max() <= 2e-3 + 2.0 ** -22 * np.abs(want_lse[fin]).max() and np.isinf(lse[~fin]).all()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("raised", [60, 80, 95, 150, 200, 300, 400])
def test_one_key_far_above_the_first_tile(device, raised, causal, bf16):
    """In head h the key at column h of a half key tile, in a later tile, lies `raised` above everything before it: from there on
    a row's softmax is that key (times 1 / (1 + about 500 e^-raised)), whichever unit evaluates its column."""
    rng = np.random.default_rng(raised)
    sq, sk, h, d = 260, 640, 64, 64
    q, k, v = (rng.standard_normal((1, s, h, d)).astype(np.float32) for s in (sq, sk, sk))
    q[..., 0], k[..., 0] = 8.0, 0.0
    for i in range(h):
        k[0, 128 * (2 + i % 3) + 64 * (i & 1) + i, i, 0] = raised
    q, k, v = (from16(to16(a, bf16), bf16) for a in (q, k, v))
    want, want_lse = an.mha_forward(q, k, v, 1.0 / np.sqrt(d), causal)
    got, lse = attend(device, q, k, v, 1.0 / np.sqrt(d), causal, bf16, 2)
    assert np.abs(got - want).max() <= (1.5e-2 if bf16 else 2e-3) * np.abs(want).max()
    assert np.abs(lse - want_lse).max() <= 2e-3 + 2.0 ** -22 * np.abs(want_lse).max()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("sq,sk,causal", [(512, 512, False), (700, 2000, True)])
def test_as_near_to_the_oracle_as_one_tile(device, sq, sk, causal, bf16):
    """The same roundings of p, the row's largest exactly 1, and of the result: the errors' 2-norms differ by 1e-4 at most (1e-3
    where the tensor core's truncation has one sign).  With references below the maximum they were 2 to 4 % apart."""
    rng = np.random.default_rng(sk)
    q, k, v = (rng.standard_normal((1, s, h, 128)).astype(np.float32) for s, h in ((sq, 4), (sk, 2), (sk, 2)))
    q, k, v = (from16(to16(a, bf16), bf16) for a in (q, k, v))
    for values, more in ((v, 3e-4), (np.abs(v), 2e-3)):
        want, _ = an.mha_forward(q, k, values, 128 ** -0.5, causal)
        one, two = (np.linalg.norm(attend(device, q, k, values, 128 ** -0.5, causal, bf16, option)[0] - want) for option in (0, 2))
        assert two <= (1 + more) * one, (one, two)


@pytest.mark.parametrize("option", [0, 2])
def test_first_tile_at_minus_infinity(device, option):
    """Scores that overflow to -inf in the first key tile, finite ones far below zero after it."""
    rng = np.random.default_rng(3)
    q, k, v = (rng.standard_normal((1, 300, 2, 64)).astype(np.float32) for _ in range(3))
    q[..., 0] = 3e19
    k[:, :128, :, 0], k[:, 128:, :, 0] = -3e19, -1e-15
    q, k, v = (from16(to16(a, True), True) for a in (q, k, v))
    want, want_lse = an.mha_forward(q, k, v, 0.125, False)
    got, lse = attend(device, q, k, v, 0.125, False, True, option)
    assert np.abs(got - want).max() <= 1.5e-2 * np.abs(want).max()
    assert np.abs(lse - want_lse).max() <= 2e-3 + 2.0 ** -22 * np.abs(want_lse).max()


@pytest.mark.parametrize("scale", [0.09, 0.0, -0.09])
def test_not_finite_as_with_one_tile(device, scale):
    """Infinities and NaNs in q, k or v, and scales that are not positive (which keep one tile per CTA)."""
    rng = np.random.default_rng(11)
    q, k, v = (rng.standard_normal((1, 300, 2, 64)).astype(np.float32) for _ in range(3))
    q[0, 5, 0, 3], q[0, 140, 1, 0], q[0, 290, 0, 7] = np.nan, np.inf, -np.inf
    k[0, 200, 1, 1], v[0, 130, 0, 2] = np.nan, np.inf
    one, lse1 = attend(device, q, k, v, scale, True, False, 0)
    two, lse2 = attend(device, q, k, v, scale, True, False, 2)
    if scale <= 0.0:
        assert np.array_equal(one, two, equal_nan=True) and np.array_equal(lse1, lse2, equal_nan=True)
        return
    assert (np.isfinite(one) == np.isfinite(two)).all() and (np.isfinite(lse1) == np.isfinite(lse2)).all()
    f = np.isfinite(one)
    assert np.abs(one[f] - two[f]).max() <= 4e-3 * np.abs(one[f]).max()
