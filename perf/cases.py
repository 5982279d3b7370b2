"""Performance cases of the library: what a user of it has it do, through the entry points that a host program calls.

``listed()`` names twelve such jobs, ``draw(rng)`` makes one more of the same ranges, ``prepare`` builds what the
program has in hand before the call (weights, inputs, buffers, a model and its captured graph), ``run`` is one pass.
``work`` counts what a pass cannot do without, ``tolerance`` what another correct implementation may differ by, and
``exact`` evaluates a case in 64 bits with plain torch.

Kinds of case:
  linear     cq_qmatmul / cq_qlinear on device tensors: y = x W^T (+ b) with block-quantized W, one row (decode),
             a few rows (small batches) or many (prompts), in each activation mode
  forward    QLinear.forward on host arrays: the call of candy's nn.Linear.Forward
  attention  cq_flash_attention: the prompt's attention, and its log-sum-exp
  codec      cq_quantize_rows, then cq_dequantize of the blocks just made
  decode     greedy decode steps of a decoder, one captured step replayed per token
  prompt     QuantDecoder.prefill: a prompt in one pass, logits of its last position
  layers     a decode step of bare decoder layers for a batch of sequences at a given context
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from candy_b200 import abi
from candy_b200.backend import ACT_F16, ACT_F32, ACT_Q8_1, CudaDevice, QLinear, QStorage, RawBuffer
from candy_b200.decoder import DecoderConfig, QuantDecoder

QTYPES = {"q4_0": abi.Q4_0, "q8_0": abi.Q8_0, "q4_1": abi.Q4_1, "q5_0": abi.Q5_0, "q4_k": abi.Q4_K, "q6_k": abi.Q6_K}
ACTS = {"f32": ACT_F32, "q8_1": ACT_Q8_1, "f16": ACT_F16}


def listed():
    return [
        # One token through an attention projection of the 7B shape: the smallest call, latency counts.
        {"name": "gemv_4096", "kind": "linear", "qtype": "q4_0", "order": 0, "act": "f32", "m": 1, "n": 4096, "k": 4096, "bias": False},
        # One token through its output layer, blocks as GGUF files order them: the longest single GEMV of a token.
        {"name": "gemv_32000", "kind": "linear", "qtype": "q4_0", "order": 1, "act": "f32", "m": 1, "n": 32000, "k": 4096, "bias": False},
        # candy's nn.Linear.Forward on host data, 8-bit weights, one row in and one row out.
        {"name": "forward_q8_0", "kind": "forward", "qtype": "q8_0", "act": "f32", "m": 1, "n": 4096, "k": 4096},
        # Eight sequences decoded together, feed-forward projection of the 7B shape.
        {"name": "batch8", "kind": "linear", "qtype": "q4_0", "order": 0, "act": "f32", "m": 8, "n": 11008, "k": 4096, "bias": False},
        # A ragged batch in the numerics of the reference's CUDA kernels (Q8_1 activations, integer dots).
        {"name": "batch100_q8_1", "kind": "linear", "qtype": "q8_0", "order": 0, "act": "q8_1", "m": 100, "n": 11008, "k": 4096, "bias": False},
        # A prompt of 512 tokens through a linear layer with bias in the default activation mode.
        {"name": "linear512_f32", "kind": "linear", "qtype": "q4_0", "order": 0, "act": "f32", "m": 512, "n": 11008, "k": 4096, "bias": True},
        # A long prompt through a feed-forward projection in the mode meant for prompts.
        {"name": "linear2048_f16", "kind": "linear", "qtype": "q8_0", "order": 0, "act": "f16", "m": 2048, "n": 11008, "k": 4096, "bias": False},
        # Attention of two 4096-token prompts with the grouped heads of the 70B shape, bf16.
        {"name": "attention_4096", "kind": "attention", "b": 2, "h": 64, "hk": 8, "sq": 4096, "sk": 4096, "d": 128, "causal": True, "bf16": True},
        # Weights quantized on the device when a model is made, and read back as f32 (a checkpoint conversion).
        {"name": "codec", "kind": "codec", "qtype": "q4_0", "order": 0, "n": 11008, "k": 4096},
        # Four greedy tokens of a decoder with the 7B layer shape and vocabulary, half its depth, one sequence.
        {"name": "decode_7b", "kind": "decode", "layers": 16, "dim": 4096, "heads": 32, "kv_heads": 32, "ffn": 11008, "vocab": 32000,
         "pos": 128, "tokens": 4},
        # The 128-token prompt of the same model in one pass.
        {"name": "prompt_7b", "kind": "prompt", "layers": 16, "dim": 4096, "heads": 32, "kv_heads": 32, "ffn": 11008, "vocab": 32000,
         "tokens": 128},
        # 32 sequences through two layers of the 70B shape at 2048 positions of context.
        {"name": "layers_70b_batch32", "kind": "layers", "layers": 2, "dim": 8192, "heads": 64, "kv_heads": 8, "ffn": 28672, "batch": 32,
         "ctx": 2048},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear"] * 10 + ["forward"] * 2 + ["attention"] * 3 + ["codec", "decode", "prompt", "layers"])
    if kind in ("linear", "forward"):
        qtype = rng.choice(["q4_0"] * 5 + ["q8_0"] * 4 + (["q4_1", "q5_0", "q4_k", "q6_k"] if kind == "linear" else []))
        # rows of a Llama-like layer are multiples of 256 values; every fourth matrix has just whole blocks
        n, k = _log_int(rng, 700, 32000), 256 * _log_int(rng, 4, 56)
        if qtype in ("q4_0", "q8_0") and rng.random() < 0.25:
            k += 32 * rng.randrange(1, 8)
        whole = k % 256 == 0
        m = 1 if rng.random() < 0.3 else _log_int(rng, 1, 2048 if kind == "linear" else 64)
        act = rng.choice(["f32", "f32", "q8_1", "f16"])
        if qtype not in ("q4_0", "q8_0"):  # formats with a decode GEMV and an f16 GEMM
            act = "f32" if m <= 8 else "f16"
        elif not whole and m > 64:  # rows that are not multiples of 256 values serve batches in the f16 mode
            act = "f16"
        n = max(700, min(n, 2048 * 11008 * 4096 // (m * k)))
        case = {"kind": kind, "qtype": qtype, "act": act, "m": m, "n": n, "k": k}
        if kind == "linear":
            case.update(order=1 if qtype not in ("q4_0", "q8_0") else rng.randrange(2), bias=rng.random() < 0.25)
        return case
    if kind == "attention":
        sk = _log_int(rng, 64, 4096)
        sq = sk if rng.random() < 0.7 else _log_int(rng, 64, sk)
        hk = rng.choice([1, 2, 4, 8, 16, 32])
        h = hk * rng.choice([1, 2, 4, 8]) if hk <= 8 else hk
        return {"kind": kind, "b": rng.randrange(1, 3), "h": h, "hk": hk, "sq": sq, "sk": sk, "d": rng.choice([64, 128, 128]),
                "causal": rng.random() < 0.75, "bf16": rng.random() < 0.5}
    if kind == "codec":
        return {"kind": kind, "qtype": rng.choice(["q4_0", "q8_0"]), "order": rng.randrange(2), "n": _log_int(rng, 256, 11008),
                "k": 32 * _log_int(rng, 32, 128)}
    kv = rng.choice([4, 8])
    heads = kv * rng.choice([1, 2, 4])
    shape = {"kind": kind, "layers": rng.randrange(2, 9), "dim": 256 * rng.randrange(4, 17), "heads": heads, "kv_heads": kv,
             "ffn": 64 * rng.randrange(32, 172)}
    if kind == "layers":
        return dict(shape, batch=_log_int(rng, 1, 48), ctx=_log_int(rng, 128, 2048))
    if kind == "decode":
        return dict(shape, vocab=_log_int(rng, 4000, 32000), pos=_log_int(rng, 16, 2000), tokens=rng.randrange(1, 5))
    return dict(shape, vocab=_log_int(rng, 4000, 32000), tokens=_log_int(rng, 8, 512))


# ---- what a program has in hand before the call ---------------------------------------------------------------
class _Device:
    """A device allocation of the library as a torch tensor that shares its memory."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner  # keeps the allocation alive
        self.__cuda_array_interface__ = {"data": (int(ptr.value), False), "shape": tuple(shape), "typestr": typestr, "version": 3}


def _tensor(storage, shape, typestr="<f4"):
    return torch.as_tensor(_Device(storage, storage.ptr, shape, typestr), device="cuda")


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _weights(dev, g, qtype, order, n, k):
    """Blocks of W ~ N(0, 0.02): through the library's quantizer, or for the formats without one random quants with
    scales of that size."""
    qt = QTYPES[qtype]
    if qt not in abi.K_BLOCK_BYTES:
        w = torch.randn(n, k, generator=g, device="cuda") * 0.02
        q = QStorage(dev, qt, order, n, k, RawBuffer(dev, n * (k // 32) * abi.BLOCK_BYTES[qt]))
        torch.cuda.synchronize()
        abi.check(dev.ctx, dev._lib.cq_quantize_rows(dev.ctx, qt, order, _ptr(w), n, k, q.buf.ptr), "quantize")
    else:
        bb = abi.K_BLOCK_BYTES[qt]
        raw = torch.randint(0, 256, (n * (k // 256), bb), generator=g, device="cuda", dtype=torch.uint8)
        scale = lambda lo, hi: (torch.rand(raw.shape[0], 1, generator=g, device="cuda") * (hi - lo) + lo).half().view(torch.uint8)  # noqa: E731
        if qt == abi.Q4_K:
            raw[:, 0:2], raw[:, 2:4] = scale(1e-4, 2e-4), scale(8e-4, 1.6e-3)
        else:
            raw[:, 208:210] = scale(1e-5, 2e-5)
        q = QStorage(dev, qt, order, n, k, RawBuffer(dev, raw.numel()))
        torch.cuda.synchronize()
        abi.check(dev.ctx, dev._lib.cq_memcpy_d2d(dev.ctx, q.buf.ptr, _ptr(raw), raw.numel()), "copy")
    dev.synchronize()  # before the source goes back to torch
    return q


def _config(case, max_ctx, with_head):
    return DecoderConfig(n_layers=case["layers"], dim=case["dim"], n_heads=case["heads"], n_kv_heads=case["kv_heads"], head_dim=128,
                         ffn=case["ffn"], vocab=case["vocab"] if with_head else 0, max_ctx=max_ctx, with_head=with_head)


def _caches(model, max_ctx):
    shape = (model.batch, max_ctx, model.kv_dim)
    return [_tensor(layer[key], shape) for layer in model.layers for key in ("k", "v")]


def _fill_caches(model, max_ctx, seed):
    """Keys and values as if max_ctx positions had been decoded."""
    for i, layer in enumerate(model.layers):
        for j, key in enumerate(("k", "v")):
            abi.check(model.ctx, model.lib.cq_rand_normal(model.ctx, layer[key].ptr, model.batch * max_ctx * model.kv_dim, 0.0, 1.0,
                                                          seed * 1000 + 2 * i + j), "rand normal")


def prepare(case, seed):
    kind, dev = case["kind"], CudaDevice(0)
    g = _generator(seed)
    st = {"case": case, "dev": dev}
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        st["w"] = _weights(dev, g, case["qtype"], case["order"], n, k)
        st["x"] = torch.randn(m, k, generator=g, device="cuda")
        st["bias"] = torch.randn(n, generator=g, device="cuda") * 0.1 if case["bias"] else None
        st["y"] = torch.empty(m, n, device="cuda")
    elif kind == "forward":
        st["linear"] = QLinear(_weights(dev, g, case["qtype"], 0, case["n"], case["k"]), None, ACTS[case["act"]])
        st["x"] = np.random.default_rng(int(seed)).standard_normal((case["m"], case["k"]), dtype=np.float32)
    elif kind == "attention":
        b, h, hk, sq, sk, d = (case[x] for x in ("b", "h", "hk", "sq", "sk", "d"))
        dt = torch.bfloat16 if case["bf16"] else torch.float16
        st["q"] = torch.randn(b, sq, h, d, generator=g, device="cuda").to(dt)
        st["k"] = torch.randn(b, sk, hk, d, generator=g, device="cuda").to(dt)
        st["v"] = torch.randn(b, sk, hk, d, generator=g, device="cuda").to(dt)
        st["o"], st["lse"] = torch.empty_like(st["q"]), torch.empty(b, h, sq, device="cuda")
    elif kind == "codec":
        n, k, qt = case["n"], case["k"], QTYPES[case["qtype"]]
        st["w"] = torch.randn(n, k, generator=g, device="cuda") * 0.02
        st["blocks"] = torch.empty(n * (k // 32) * abi.BLOCK_BYTES[qt], dtype=torch.uint8, device="cuda")
        st["back"] = torch.empty(n, k, device="cuda")
    elif kind == "decode":
        max_ctx = case["pos"] + case["tokens"]
        model = st["model"] = QuantDecoder(dev, _config(case, max_ctx, True), seed=int(seed))
        _fill_caches(model, max_ctx, int(seed))
        st["ids"] = np.random.default_rng(int(seed)).integers(0, case["vocab"], size=1).astype(np.uint32)
        model.set_state(st["ids"], case["pos"])
        model.step()  # first launches outside the capture
        model.set_state(st["ids"], case["pos"])
        st["graph"] = model.capture(1)
        st["out"] = [_tensor(model.logits, (1, case["vocab"])), _tensor(model.ids, (1,), "<i4")] + _caches(model, max_ctx)
    elif kind == "prompt":
        model = st["model"] = QuantDecoder(dev, _config(case, case["tokens"], True), seed=int(seed))
        st["ids"] = np.random.default_rng(int(seed)).integers(0, case["vocab"], size=case["tokens"]).astype(np.uint32)
        st["out"] = [_tensor(model.logits, (1, case["vocab"]))] + _caches(model, case["tokens"])  # the next token is their arg-max
    elif kind == "layers":
        batch, ctx, dim = case["batch"], case["ctx"], case["dim"]
        model = st["model"] = QuantDecoder(dev, _config(case, ctx, False), seed=int(seed), batch=batch)
        _fill_caches(model, ctx, int(seed))
        st["x"] = torch.randn(batch, dim, generator=g, device="cuda")
        model.set_state(np.zeros(batch, dtype=np.uint32), ctx - 1)
        model.step(advance=False)
        model.set_state(np.zeros(batch, dtype=np.uint32), ctx - 1)
        abi.check(model.ctx, model.lib.cq_capture_begin(model.ctx), "capture begin")
        model.step(advance=False)
        st["graph"] = C.c_void_p()
        abi.check(model.ctx, model.lib.cq_capture_end(model.ctx, C.byref(st["graph"])), "capture end")
        st["out"] = [_tensor(model.x, (batch, dim)), _tensor(model.d, (batch, dim))] + _caches(model, ctx)
    else:
        raise ValueError(f"unknown kind {kind}")
    dev.synchronize()
    torch.cuda.synchronize()
    return st


# ---- one pass ---------------------------------------------------------------------------------------------------
def run(st):
    case, dev = st["case"], st["dev"]
    lib, ctx, kind = dev._lib, dev.ctx, case["kind"]
    if kind == "linear":
        w, x, y = st["w"], st["x"], st["y"]
        m, n, k = case["m"], case["n"], case["k"]
        if st["bias"] is None:
            s = lib.cq_qmatmul(ctx, w.qtype, w.order, ACTS[case["act"]], x.data_ptr(), m, k, k, w.buf.ptr, n, y.data_ptr(), n)
        else:
            s = lib.cq_qlinear(ctx, w.qtype, w.order, ACTS[case["act"]], x.data_ptr(), m, k, k, w.buf.ptr, n, st["bias"].data_ptr(),
                               y.data_ptr(), n)
        abi.check(ctx, s, "linear")
        return y
    if kind == "forward":
        return st["linear"].forward(st["x"])
    if kind == "attention":
        b, h, hk, sq, sk, d = (case[x] for x in ("b", "h", "hk", "sq", "sk", "d"))
        s = lib.cq_flash_attention(ctx, st["q"].data_ptr(), st["k"].data_ptr(), st["v"].data_ptr(), st["o"].data_ptr(), st["lse"].data_ptr(),
                                   None, None, None, sq * h * d, sk * hk * d, sk * hk * d, sq * h * d, 0, h * d, hk * d, hk * d, h * d,
                                   d, d, d, d, b, h, hk, d, d, d ** -0.5, sq, sk, -(-sq // 128) * 128, -(-sk // 128) * 128,
                                   1 if case["bf16"] else 0, 1 if case["causal"] else 0, 0, -1, -1, 0.0)
        abi.check(ctx, s, "attention")
        return st["o"], st["lse"]
    if kind == "codec":
        n, k, qt = case["n"], case["k"], QTYPES[case["qtype"]]
        abi.check(ctx, lib.cq_quantize_rows(ctx, qt, case["order"], st["w"].data_ptr(), n, k, st["blocks"].data_ptr()), "quantize")
        abi.check(ctx, lib.cq_dequantize(ctx, qt, case["order"], st["blocks"].data_ptr(), n * (k // 32), st["back"].data_ptr()), "dequantize")
        return st["blocks"], st["back"]
    model = st["model"]
    if kind == "decode":
        model.set_state(st["ids"], case["pos"])
        model.replay(st["graph"], case["tokens"])
    elif kind == "prompt":
        model.set_state(st["ids"][:1], 0)
        model.prefill(st["ids"])
    else:  # the residual stream of the previous layers comes in, nothing pending
        abi.check(ctx, lib.cq_memcpy_d2d(ctx, model.x.ptr, st["x"].data_ptr(), 4 * st["x"].numel()), "stream in")
        abi.check(ctx, lib.cq_memset(ctx, model.d.ptr, 0, 4 * st["x"].numel()), "nothing pending")
        abi.check(ctx, lib.cq_graph_launch(ctx, st["graph"]), "graph launch")
    return st["out"]


# ---- what a pass cannot do without, and how exactly its results are defined ---------------------------------------
def _block_bytes(qtype, count):
    qt = QTYPES[qtype]
    return count // 256 * abi.K_BLOCK_BYTES[qt] if qt in abi.K_BLOCK_BYTES else count // 32 * abi.BLOCK_BYTES[qt]


def _layer_weights(case):
    hd = 128
    return (case["heads"] + 2 * case["kv_heads"]) * hd * case["dim"] + case["dim"] * case["heads"] * hd + 3 * case["ffn"] * case["dim"]


def _visible(sq, sk, causal):
    """Query-key pairs of one head, the mask aligned to the bottom right."""
    return sum(max(0, min(sk, i + 1 + sk - sq)) for i in range(sq)) if causal else sq * sk


def work(case):
    kind = case["kind"]
    if kind in ("linear", "forward"):
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": _block_bytes(case["qtype"], n * k) + 4 * m * (k + n) + (4 * n if case.get("bias") else 0), "flops": 2 * m * n * k}
    if kind == "attention":
        b, h, hk, sq, sk, d = (case[x] for x in ("b", "h", "hk", "sq", "sk", "d"))
        return {"bytes": 2 * b * d * (2 * sq * h + 2 * sk * hk) + 4 * b * h * sq, "flops": 4 * b * h * d * _visible(sq, sk, case["causal"])}
    if kind == "codec":
        count = case["n"] * case["k"]
        return {"bytes": 2 * (4 * count + _block_bytes(case["qtype"], count)), "flops": 0}
    layers, hd = case["layers"], 128
    weights, kv = layers * _layer_weights(case), layers * 2 * case["kv_heads"] * hd
    if kind == "decode":
        head, steps = case["vocab"] * case["dim"], case["tokens"]
        keys = sum(case["pos"] + 1 + t for t in range(steps))
        return {"bytes": steps * (_block_bytes("q4_0", weights + head) + 4 * (case["vocab"] + case["dim"])) + 4 * kv * keys,
                "flops": 2 * steps * (weights + head) + 4 * layers * case["heads"] * hd * keys}
    if kind == "prompt":
        head, t = case["vocab"] * case["dim"], case["tokens"]
        return {"bytes": _block_bytes("q4_0", weights + head) + 4 * kv * t + 4 * t * case["dim"] + 4 * case["vocab"],
                "flops": 2 * t * weights + 2 * head + 4 * layers * case["heads"] * hd * _visible(t, t, True)}
    b, ctx = case["batch"], case["ctx"]
    return {"bytes": _block_bytes("q4_0", weights) + 4 * b * kv * ctx + 12 * b * case["dim"],
            "flops": 2 * b * weights + 4 * b * layers * case["heads"] * hd * ctx}


def tolerance(case):
    """Relative error in the 2-norm that another correct implementation at the same precision may show: about four times
    what the path shows against a 64-bit evaluation on the same inputs, or (models) against its own steps with
    activations resolved to f32."""
    kind = case["kind"]
    if kind == "codec":
        return "exact"
    if kind == "attention":  # 16-bit probabilities and results: 2.1e-3 in bf16, 2.6e-4 in f16
        return {"rel": 8e-3 if case["bf16"] else 1.2e-3}
    if kind in ("linear", "forward"):  # 15-bit block fixed point 4.2e-5; exact integer dots, f32 sums; f16 operands 2.9e-4
        return {"rel": {"f32": 1.6e-4, "q8_1": 1e-5, "f16": 1.2e-3}[case["act"]]}
    # logits of f16-operand layers 4.8e-3; one token's f32-mode layers 2.5e-4; two layers of a batch 9e-4
    return {"rel": {"prompt": 1.6e-2, "decode": 1e-3, "layers": 4e-3}[kind]}


# ---- the same results in 64 bits, without the library ------------------------------------------------------------
def _exact_weights(g, qtype, n, k):
    """The values that the blocks of ``_weights`` stand for, and the scales of the blocks where those are of one kind (f64).
    The element order inside a block changes nothing here: random bytes come in the files' order only."""
    if qtype not in ("q4_k", "q6_k"):
        v = (torch.randn(n, k, generator=g, device="cuda") * 0.02).view(-1, 32)
        inv = lambda d: torch.where(d != 0, 1.0 / d, torch.zeros_like(d))  # noqa: E731
        if qtype in ("q4_0", "q5_0"):
            half = 8 if qtype == "q4_0" else 16
            d = v.gather(1, v.abs().argmax(1, keepdim=True)) / -half
            q = (v * inv(d) + (half + 0.5)).int().clamp_max(2 * half - 1) - half
            w = d.half().double() * q
        elif qtype == "q4_1":
            lo = v.amin(1, keepdim=True)
            d = (v.amax(1, keepdim=True) - lo) / 15
            w = d.half().double() * ((v - lo) * inv(d) + 0.5).int().clamp_max(15) + lo.half().double()
        else:
            d = v.abs().amax(1, keepdim=True) / 127
            u = (v * inv(d)).double()
            w = d.half().double() * (u.sign() * (u.abs() + 0.5).floor())  # ties away from zero
        return w.reshape(n, k), d.half().double().view(n, -1)
    size = abi.K_BLOCK_BYTES[QTYPES[qtype]]
    raw = torch.randint(0, 256, (n * (k // 256), size), generator=g, device="cuda", dtype=torch.uint8)
    scale = lambda lo, hi: (torch.rand(raw.shape[0], 1, generator=g, device="cuda") * (hi - lo) + lo).half().double()  # noqa: E731
    if qtype == "q4_k":
        d, dmin = scale(1e-4, 2e-4), scale(8e-4, 1.6e-3)
        s = raw[:, 4:16].int()
        sc = torch.cat([s[:, 0:4] & 63, (s[:, 8:12] & 15) | (s[:, 0:4] >> 6 << 4)], 1)
        mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:12] >> 4) | (s[:, 4:8] >> 6 << 4)], 1)
        qs = raw[:, 16:].int().view(-1, 4, 1, 32)
        q = torch.cat([qs & 15, qs >> 4], 2).view(-1, 8, 32)  # 32 low nibbles, then the high ones of the same bytes
        w = (d * sc).unsqueeze(2) * q - (dmin * mn).unsqueeze(2)
    else:
        d = scale(1e-5, 2e-5)
        ql, qh = raw[:, :128].int().view(-1, 2, 2, 32), raw[:, 128:192].int().view(-1, 2, 1, 32)
        sc = raw[:, 192:208].view(torch.int8).double().repeat_interleave(16, 1)
        four = [(ql[:, :, j & 1:(j & 1) + 1] >> (4 * (j >> 1)) & 15) | ((qh >> (2 * j) & 3) << 4) for j in range(4)]
        w = d * sc * (torch.cat(four, 2).reshape(-1, 256) - 32)
    return w.reshape(n, k), None


def _exact_linear(case, x, w, d):
    """x W^T; in the Q8_1 mode of the activations that the mode defines: whole numbers of d8 = amax / 127, and for 4-bit
    weights, whose offset meets a block's sum, that sum in f16 beside them: d4 (sumi d8 - 8 s8)."""
    if case["act"] != "q8_1":
        return x.double() @ w.T
    v = x.reshape(-1, 32)
    d8 = v.abs().amax(1, keepdim=True) / 127
    u = torch.where(d8 != 0, v / d8, torch.zeros_like(v)).double()
    held = d8.half().double() * (u.sign() * (u.abs() + 0.5).floor())
    y = held.view(x.shape) @ w.T
    if case["qtype"] == "q4_0":
        y += (held.sum(1) - v.sum(1, dtype=torch.float64).half().double()).view(x.shape[0], -1) @ (8 * d).T
    return y


def exact(case, seed):
    kind = case["kind"]
    if kind in ("decode", "prompt", "layers"):  # their weights and caches come from the library's own generator
        return None
    g = _generator(seed)
    if kind in ("linear", "forward"):
        m, n, k = case["m"], case["n"], case["k"]
        w, d = _exact_weights(g, case["qtype"], n, k)
        if kind == "forward":
            x = torch.from_numpy(np.random.default_rng(int(seed)).standard_normal((m, k), dtype=np.float32)).cuda()
            return _exact_linear(case, x, w, d).cpu().numpy()
        y = _exact_linear(case, torch.randn(m, k, generator=g, device="cuda"), w, d)
        return y + (torch.randn(n, generator=g, device="cuda") * 0.1).double() if case["bias"] else y
    if kind == "codec":  # the blocks are bytes
        return None, _exact_weights(g, case["qtype"], case["n"], case["k"])[0]
    b, h, hk, sq, sk, dim = (case[x] for x in ("b", "h", "hk", "sq", "sk", "d"))
    dt = torch.bfloat16 if case["bf16"] else torch.float16
    q, key, v = (torch.randn(b, s, heads, dim, generator=g, device="cuda").to(dt) for s, heads in ((sq, h), (sk, hk), (sk, hk)))
    hidden = torch.ones(sq, sk, dtype=torch.bool, device="cuda").triu(1 + sk - sq) if case["causal"] else None
    o = torch.empty(b, sq, h, dim, dtype=torch.float64, device="cuda")
    lse = torch.empty(b, h, sq, dtype=torch.float64, device="cuda")
    for i in range(b):
        for j in range(h):
            s = q[i, :, j].double() @ key[i, :, j * hk // h].double().T * dim ** -0.5
            if hidden is not None:
                s.masked_fill_(hidden, -math.inf)
            lse[i, j] = s.logsumexp(1)
            o[i, :, j] = (s - lse[i, j].unsqueeze(1)).exp_() @ v[i, :, j * hk // h].double()
    return o, lse
