"""The workloads by which the speed of this library is followed, and the ranges they stand for.

Each case is one call (or the short run of calls that a program makes together) through the public entry points:
what a user has in hand is made by ``prepare``, one pass over it is ``run``.  ``listed`` names the fixed cases,
``draw`` gives further ones of the same kinds and ranges.  Kinds:

step      one decoding step of a layer: ``rope_padded`` writes the new keys and values into the padded cache, attention reads it
paged     decode attention over a paged cache in 16-bit, int4 row-wise or fp8 row-wise format
segments  decode attention over a long context kept in several segments: partial attention per segment, then the merge
dense     prefill of equally long sequences, with or without a causal mask, MHA or GQA
varlen    prefill of packed sequences of unequal length (block-diagonal causal mask), log-sum-exp returned
chunk     new tokens of several sequences on top of what their padded cache already holds: ``rope_padded``, then attention
bias      prefill with an additive bias tensor (relative positions), alone or under the causal mask
encoder   attention without a mask over many short sequences with the head dims of vision encoders
"""

from __future__ import annotations

import math

import torch

import xformers_b200.ops as xops
from xformers_b200.ops import fmha
from xformers_b200.ops.fmha import attn_bias as ab

_DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16}


def listed():
    return [
        # a chat-sized decoding step: few sequences, short contexts; launches and host work are what it costs
        dict(name="step_small", kind="step", batch=4, kv=1000, hq=32, hkv=8, d=128, dtype="bf16", lens=1),
        # serving: 64 sequences of mixed length over a paged cache, in each cache format
        dict(name="paged_bf16", kind="paged", fmt="bf16", batch=64, kv_min=1024, kv=32768, hq=64, hkv=8, page=256, dtype="bf16", lens=2),
        dict(name="paged_int4", kind="paged", fmt="int4", batch=64, kv_min=1024, kv=32768, hq=64, hkv=8, page=256, dtype="bf16", lens=2),
        dict(name="paged_fp8", kind="paged", fmt="fp8", batch=64, kv_min=1024, kv=32768, hq=64, hkv=8, page=256, dtype="bf16", lens=2),
        # two long conversations whose caches lie in four segments each, few kv heads, two tokens per step
        dict(name="segments_f16", kind="segments", batch=2, segments=4, kv=16384, mq=2, hq=16, hkv=2, d=128, dtype="f16", lens=3),
        # one short prompt, head dim 64, an odd length: the smallest prefill
        dict(name="dense_small", kind="dense", batch=1, m=333, h=8, hkv=8, d=64, causal=True, lse=False, dtype="f16"),
        # the headline prefill of the benchmark
        dict(name="dense_causal_4k", kind="dense", batch=4, m=4096, h=32, hkv=32, d=128, causal=True, lse=False, dtype="bf16"),
        # one very long document
        dict(name="dense_long", kind="dense", batch=1, m=131072, h=64, hkv=8, d=128, causal=True, lse=False, dtype="bf16"),
        # a training or prefill batch packed without padding
        dict(name="varlen_gqa", kind="varlen", batch=16, m_min=256, m=4096, hq=32, hkv=8, d=128, dtype="bf16", lens=4),
        # chunked prefill: up to 512 new tokens for each of eight sequences with contexts of up to 8192
        dict(name="chunk_bf16", kind="chunk", batch=8, new=512, kv=8192, hq=32, hkv=8, d=128, dtype="bf16", lens=5),
        # relative position bias on a sequence of ordinary length
        dict(name="bias_2k", kind="bias", batch=2, m=2048, h=8, d=128, causal=False, dtype="bf16"),
        # a batch of images, 197 patches each
        dict(name="encoder_d80", kind="encoder", batch=64, m=197, h=16, d=80, dtype="f16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "paged", "paged", "segments", "dense", "dense", "varlen", "chunk", "bias", "encoder"])
    lens = rng.randrange(1, 1 << 30)
    dtype = rng.choice(["bf16", "f16"])
    if kind == "step":
        hkv, g = rng.choice([(8, 4), (2, 8), (4, 7), (8, 8)])
        return dict(kind=kind, batch=_log(rng, 1, 64), kv=_log(rng, 64, 8192), hq=hkv * g, hkv=hkv, d=rng.choice([64, 128]), dtype=dtype, lens=lens)
    if kind == "paged":
        hkv, g = rng.choice([(8, 8), (8, 4), (4, 8), (1, 16)])
        kv = _log(rng, 512, 32768)
        batch = _log(rng, 1, min(256, 64 * 32768 // kv))
        return dict(kind=kind, fmt=rng.choice(["bf16", "int4", "fp8"]), batch=batch, kv_min=max(1, kv // rng.choice([1, 4, 32])), kv=kv, hq=hkv * g, hkv=hkv,
                    page=rng.choice([16, 64, 256]), dtype=dtype, lens=lens)
    if kind == "segments":
        hkv = rng.choice([1, 2])
        return dict(kind=kind, batch=_log(rng, 1, 8), segments=rng.randrange(2, 9), kv=_log(rng, 2048, 32768), mq=rng.choice([1, 2, 4]), hq=16, hkv=hkv, d=128, dtype=dtype, lens=lens)
    if kind == "dense":
        h = rng.choice([4, 8, 16, 32])
        m = _log(rng, 64, 16384)
        batch = _log(rng, 1, max(1, min(32, 65536 // m)))
        return dict(kind=kind, batch=batch, m=m, h=h, hkv=rng.choice([h, max(1, h // 4)]), d=rng.choice([64, 128, 128]), causal=rng.random() < 0.7, lse=rng.random() < 0.3, dtype=dtype)
    if kind == "varlen":
        m = _log(rng, 256, 8192)
        return dict(kind=kind, batch=rng.randrange(2, 25), m_min=max(1, m // 16), m=m, hq=32, hkv=8, d=rng.choice([64, 128]), dtype=dtype, lens=lens)
    if kind == "chunk":
        new = _log(rng, 32, 2048)
        return dict(kind=kind, batch=_log(rng, 1, 16), new=new, kv=_log(rng, 2 * new, 16384), hq=32, hkv=8, d=128, dtype=dtype, lens=lens)
    if kind == "bias":
        return dict(kind=kind, batch=rng.choice([1, 2, 3]), m=_log(rng, 256, 4096), h=rng.choice([4, 8, 12]), d=rng.choice([64, 128]), causal=rng.random() < 0.5, dtype=dtype)
    return dict(kind="encoder", batch=_log(rng, 4, 256), m=rng.randrange(50, 1025), h=rng.choice([4, 8, 16]), d=rng.choice([32, 40, 72, 80, 88, 96, 160, 256]), dtype=dtype)


def _lengths(case, lo, hi, n, salt=0):
    """The lengths belong to the case, not to the seed of its inputs: every pass of a case is the same amount of work."""
    g = torch.Generator().manual_seed(case["lens"] + salt)
    return torch.randint(lo, hi + 1, (n,), generator=g).tolist()


def _randn(gen, dtype, *shape):
    return torch.randn(shape, generator=gen, device="cuda", dtype=dtype)


def _quantize_int4(x):
    """int4 row-wise format: one word of (fp16 scale | fp16 shift << 16), then eight nibbles per word."""
    x = x.float()
    lo, hi = x.amin(-1, keepdim=True), x.amax(-1, keepdim=True)
    scale, shift = ((hi - lo) / 15).half(), lo.half()
    n = ((x - shift.float()) / scale.float() + 0.5).clamp(0, 15).to(torch.uint8)
    packed = n[..., ::2] + (n[..., 1::2] << 4)
    return torch.cat([scale.view(torch.uint8), shift.view(torch.uint8), packed], dim=-1).contiguous().view(torch.int32)


def _quantize_fp8(x):
    """fp8 row-wise format: four e4m3 values per word, and a word of (fp16 scale | fp16 shift << 16) per row beside them."""
    x = x.float()
    shift = x.mean(-1, keepdim=True)
    scale = (x - shift).abs().amax(-1, keepdim=True) / 448.0
    q = ((x - shift) / scale).to(torch.float8_e4m3fn)
    word = torch.cat([scale.half().view(torch.uint8), shift.half().view(torch.uint8)], dim=-1).contiguous().view(torch.int32)
    return q.contiguous().view(torch.int32), word.squeeze(-1)


def _decode_inputs(case):
    return _lengths(case, case["kv_min"], case["kv"], case["batch"])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = _DTYPES[case["dtype"]]
    return _PREPARE[case["kind"]](case, gen, dt)


def _prepare_step(case, gen, dt):
    b, hkv, g, d = case["batch"], case["hkv"], case["hq"] // case["hkv"], case["d"]
    lens = _lengths(case, max(1, case["kv"] // 2), case["kv"], b)
    pad = case["kv"] + 24  # room for the tokens still to come
    return dict(kind="step", xq=_randn(gen, dt, 1, b, hkv, g, d), xk=_randn(gen, dt, 1, b, hkv, 1, d), xv=_randn(gen, dt, 1, b, hkv, 1, d),
                ck=_randn(gen, dt, 1, b * pad, hkv, 1, d), cv=_randn(gen, dt, 1, b * pad, hkv, 1, d), g=g,
                bias=ab.BlockDiagonalCausalWithOffsetPaddedKeysMask.from_seqlens(q_seqlen=[1] * b, kv_padding=pad, kv_seqlen=lens, device="cuda"))


def _prepare_paged(case, gen, dt):
    b, hkv, g, d, page = case["batch"], case["hkv"], case["hq"] // case["hkv"], 128, case["page"]
    lens = _decode_inputs(case)
    pages = [-(-n // page) for n in lens]
    pool = sum(pages)
    order = torch.randperm(pool, generator=gen, device="cuda").int()
    table = torch.zeros(b, max(pages), dtype=torch.int32, device="cuda")
    at = 0
    for i, n in enumerate(pages):
        table[i, :n] = order[at : at + n]
        at += n
    rows = pool * page
    st = dict(kind="paged", fmt=case["fmt"], q=_randn(gen, dt, 1, b, hkv, g, d))
    if case["fmt"] == "bf16":  # the 16-bit cache has the type of the queries
        k, v = _randn(gen, dt, 1, rows, hkv, 1, d), _randn(gen, dt, 1, rows, hkv, 1, d)
    else:
        int4 = case["fmt"] == "int4"
        k, v = (torch.empty(1, rows, hkv, 1, d // 8 + 1 if int4 else d // 4, dtype=torch.int32, device="cuda") for _ in range(2))
        kw, vw = (torch.empty(1, rows, hkv, 1, dtype=torch.int32, device="cuda") for _ in range(2))
        step = max(page, (1 << 20) // (hkv * 8))
        for lo in range(0, rows, step):
            n = min(step, rows - lo)
            for dst, word in ((k, kw), (v, vw)):
                x = _randn(gen, dt, 1, n, hkv, 1, d)
                if int4:
                    dst[:, lo : lo + n] = _quantize_int4(x)
                else:
                    dst[:, lo : lo + n], word[:, lo : lo + n] = _quantize_fp8(x)
        if not int4:
            st.update(kw=kw.expand(-1, -1, -1, g), vw=vw.expand(-1, -1, -1, g))
    st.update(k=k.expand(-1, -1, -1, g, -1), v=v.expand(-1, -1, -1, g, -1),
              bias=ab.PagedBlockDiagonalPaddedKeysMask.from_seqlens([1] * b, lens, table, page))
    return st


def _prepare_segments(case, gen, dt):
    b, mq, hkv, g, d, pad = case["batch"], case["mq"], case["hkv"], case["hq"] // case["hkv"], case["d"], case["kv"]
    parts = []
    for s in range(case["segments"]):
        last = s == case["segments"] - 1
        lens = _lengths(case, max(mq, pad // 8), pad, b) if last else [pad] * b  # earlier segments are full, the last one is being filled
        cls = ab.BlockDiagonalCausalWithOffsetPaddedKeysMask if last else ab.BlockDiagonalPaddedKeysMask
        k, v = (_randn(gen, dt, 1, b * pad, hkv, 1, d).expand(-1, -1, -1, g, -1) for _ in range(2))
        parts.append((k, v, cls.from_seqlens(q_seqlen=[mq] * b, kv_padding=pad, kv_seqlen=lens, device="cuda")))
    return dict(kind="segments", q=_randn(gen, dt, 1, b * mq, hkv, g, d), parts=parts)


def _prepare_dense(case, gen, dt):
    b, m, h, hkv, d = case["batch"], case["m"], case["h"], case["hkv"], case["d"]
    bias = ab.LowerTriangularMask() if case["causal"] else None
    if h == hkv:
        q, k, v = (_randn(gen, dt, b, m, h, d) for _ in range(3))
    else:
        q = _randn(gen, dt, b, m, hkv, h // hkv, d)
        k, v = (_randn(gen, dt, b, m, hkv, 1, d).expand(-1, -1, -1, h // hkv, -1) for _ in range(2))
    return dict(kind="lse" if case["lse"] else "dense", q=q, k=k, v=v, bias=bias)


def _prepare_varlen(case, gen, dt):
    lens = _lengths(case, case["m_min"], case["m"], case["batch"])
    n, hkv, g, d = sum(lens), case["hkv"], case["hq"] // case["hkv"], case["d"]
    k, v = (_randn(gen, dt, 1, n, hkv, 1, d).expand(-1, -1, -1, g, -1) for _ in range(2))
    return dict(kind="lse", q=_randn(gen, dt, 1, n, hkv, g, d), k=k, v=v, bias=ab.BlockDiagonalCausalMask.from_seqlens(lens, device="cuda"))


def _chunk_lengths(case):
    new = _lengths(case, max(1, case["new"] // 4), case["new"], case["batch"])
    total = _lengths(case, case["new"], case["kv"], case["batch"], salt=1)
    return new, total


def _prepare_chunk(case, gen, dt):
    new, total = _chunk_lengths(case)
    n, b, hkv, g, d, pad = sum(new), case["batch"], case["hkv"], case["hq"] // case["hkv"], case["d"], case["kv"]
    return dict(kind="step", xq=_randn(gen, dt, 1, n, hkv, g, d), xk=_randn(gen, dt, 1, n, hkv, 1, d), xv=_randn(gen, dt, 1, n, hkv, 1, d),
                ck=_randn(gen, dt, 1, b * pad, hkv, 1, d), cv=_randn(gen, dt, 1, b * pad, hkv, 1, d), g=g,
                bias=ab.BlockDiagonalCausalWithOffsetPaddedKeysMask.from_seqlens(q_seqlen=new, kv_padding=pad, kv_seqlen=total, device="cuda"))


def _prepare_bias(case, gen, dt):
    b, m, h, d = case["batch"], case["m"], case["h"], case["d"]
    wide = -(-m // 8) * 8  # rows of the bias start on 16-byte boundaries, as a program would lay them out
    bias = _randn(gen, dt, b, h, m, wide)[..., :m]
    q, k, v = (_randn(gen, dt, b, m, h, d) for _ in range(3))
    return dict(kind="dense", q=q, k=k, v=v, bias=ab.LowerTriangularMaskWithTensorBias(bias) if case["causal"] else bias)


def _prepare_encoder(case, gen, dt):
    q, k, v = (_randn(gen, dt, case["batch"], case["m"], case["h"], case["d"]) for _ in range(3))
    return dict(kind="dense", q=q, k=k, v=v, bias=None)


_PREPARE = dict(step=_prepare_step, paged=_prepare_paged, segments=_prepare_segments, dense=_prepare_dense, varlen=_prepare_varlen, chunk=_prepare_chunk,
                bias=_prepare_bias, encoder=_prepare_encoder)


def run(state):
    s = state
    if s["kind"] == "dense":
        return xops.memory_efficient_attention_forward(s["q"], s["k"], s["v"], s["bias"])
    if s["kind"] == "lse":
        return fmha.memory_efficient_attention_forward_requires_grad(s["q"], s["k"], s["v"], s["bias"])
    if s["kind"] == "step":
        q = xops.rope_padded(s["xq"], s["xk"], s["xv"], s["ck"], s["cv"], s["bias"])
        k, v = (c.expand(-1, -1, -1, s["g"], -1) for c in (s["ck"], s["cv"]))
        return xops.memory_efficient_attention_forward(q, k, v, s["bias"]), s["ck"], s["cv"]
    if s["kind"] == "segments":
        parts = [fmha.memory_efficient_attention_partial(s["q"], k, v, bias) for k, v, bias in s["parts"]]
        return fmha.merge_attentions([o for o, _ in parts], [l for _, l in parts])
    if s["fmt"] == "fp8":
        inp = fmha.triton_splitk.InputsFp8(query=s["q"], key=s["k"], value=s["v"], attn_bias=s["bias"], k_fp8_scale_shift=s["kw"], v_fp8_scale_shift=s["vw"])
        return fmha._memory_efficient_attention_forward(inp, op=fmha.triton_splitk.FwOp)
    return xops.memory_efficient_attention_forward(s["q"], s["k"], s["v"], s["bias"])


def _attention_work(pairs, rows_q, rows_kv, hq, hkv, d, row_bytes):
    """`pairs`: visible (query, key) pairs of one head; rows read and written once each, 16-bit queries and outputs."""
    return {"flops": 4.0 * pairs * hq * d, "bytes": 2.0 * rows_q * hq * d * 2 + 2.0 * rows_kv * hkv * row_bytes}


def work(case):
    kind = case["kind"]
    if kind in ("dense", "bias", "encoder"):
        b, m, h, d = case["batch"], case["m"], case["h"], case["d"]
        pairs = b * (m * (m + 1) // 2 if case.get("causal") else m * m)
        w = _attention_work(pairs, b * m, b * m, h, case.get("hkv", h), d, 2 * d)
        if kind == "bias":
            w["bytes"] += 2.0 * pairs * h
        if case.get("lse"):
            w["bytes"] += 4.0 * b * m * h
        return w
    if kind == "varlen":
        lens = _lengths(case, case["m_min"], case["m"], case["batch"])
        w = _attention_work(sum(n * (n + 1) // 2 for n in lens), sum(lens), sum(lens), case["hq"], case["hkv"], case["d"], 2 * case["d"])
        w["bytes"] += 4.0 * sum(lens) * case["hq"]
        return w
    if kind == "paged":
        lens = _decode_inputs(case)
        row = {"bf16": 256, "int4": 68, "fp8": 132}[case["fmt"]]
        w = _attention_work(sum(lens), case["batch"], sum(lens), case["hq"], case["hkv"], 128, row)
        w["bytes"] += 4.0 * sum(-(-n // case["page"]) for n in lens)
        return w
    if kind == "segments":
        b, mq, pad, n = case["batch"], case["mq"], case["kv"], case["segments"]
        lens = _lengths(case, max(mq, pad // 8), pad, b)
        keys = b * pad * (n - 1) + sum(lens)
        w = _attention_work(mq * keys, b * mq, keys, case["hq"], case["hkv"], case["d"], 2 * case["d"])
        w["bytes"] += 4.0 * b * mq * case["hq"]
        return w
    if kind == "step":
        new = [1] * case["batch"]
        total = _lengths(case, max(1, case["kv"] // 2), case["kv"], case["batch"])
    else:
        new, total = _chunk_lengths(case)
    pairs = sum(q * (k - q) + q * (q + 1) // 2 for q, k in zip(new, total))
    w = _attention_work(pairs, sum(new), sum(total), case["hq"], case["hkv"], case["d"], 2 * case["d"])
    # the rotary pass reads the new queries and writes them rotated; reads the new keys and values and writes them into the cache
    w["bytes"] += 2.0 * sum(new) * (case["hq"] + 2 * case["hkv"]) * case["d"] * 2
    return w


def tolerance(case):
    """What another correct implementation may be off by: relative 2-norm, and the largest error over the root mean square
    of the result.  About four times what these paths differ by from a 64-bit computation (bf16: 1.8e-3 to 2.8e-3 and up to
    2.8e-2; f16: 2.4e-4 to 3.3e-4 and up to 4.3e-3; f16 queries over a quantised cache up to 9.3e-4): the probabilities
    and the output are rounded to the 16-bit type."""
    if case["dtype"] == "bf16":
        return {"rel": 1e-2, "max": 1.2e-1}
    return {"rel": 4e-3 if case.get("fmt") in ("int4", "fp8") else 1.4e-3, "max": 2e-2}
