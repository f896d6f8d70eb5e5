"""The host front (csrc/front.cpp) against the Python operators it stands in for: the same operator, arguments and kernels, so
outputs and log-sum-exps must agree bit for bit, with the same shapes and strides; and it leaves alone what it does not cover."""

import types

import pytest
import torch

from gpu_utils import gpu, require_cuda
import xformers_b200.ops as xops
from xformers_b200 import _lib
from xformers_b200.ops import fmha
from xformers_b200.ops.fmha import attn_bias as ab


def _both(monkeypatch, call, takes=True):
    """(result through the front, result through Python); checks whether the front took the call."""
    seen = []
    real = fmha.front.forward
    monkeypatch.setattr(fmha.front, "forward", lambda *a, **k: seen.append(real(*a, **k)) or seen[-1])
    a = call()
    assert (seen[-1] is not None) == takes
    monkeypatch.setattr(fmha.front, "forward", lambda *a, **k: None)
    b = call()
    monkeypatch.setattr(fmha.front, "forward", real)
    return a, b


def _same(a, b):
    a, b = (x if isinstance(x, tuple) else (x,) for x in (a, b))
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert x.dtype == y.dtype and x.shape == y.shape and x.stride() == y.stride() and torch.equal(x, y)


def _mk(gen, *shape, dtype=torch.bfloat16):
    return torch.randn(*shape, generator=gen).to(dtype).cuda()


def _bias(name, q_lens, k_lens, pad, page):
    """A bias object by name; key rows it needs."""
    dev, n = "cuda", len(q_lens)
    if name.startswith("Paged"):
        per = -(-pad // page)
        table = torch.randperm(n * per, generator=torch.Generator().manual_seed(1)).int().view(n, per).to(dev)
        cls = getattr(ab, name)
        if "Local" in name:
            return cls.from_seqlens_local(q_lens, k_lens, table, page, 20), n * per * page
        return cls.from_seqlens(q_lens, k_lens, table, page), n * per * page
    cls = getattr(ab, name)
    if "Gappy" in name:
        starts = [i * pad for i in range(n + 1)]
        if "Local" in name:
            return cls.from_seqlens_local(q_seqlen=q_lens, kv_seqstarts=starts, kv_seqlen=k_lens, window_left=9, window_right=3, device=dev), n * pad
        return cls.from_seqlens(q_seqlen=q_lens, kv_seqstarts=starts, kv_seqlen=k_lens, device=dev), n * pad
    if "Padded" in name:
        if name == "BlockDiagonalLocalAttentionPaddedKeysMask":
            return cls.from_seqlens_local(q_seqlen=q_lens, kv_padding=pad, kv_seqlen=k_lens, window_left=9, window_right=3, device=dev), n * pad
        if "Local" in name:
            return cls.from_seqlens_local(q_seqlen=q_lens, kv_padding=pad, kv_seqlen=k_lens, window_size=20, device=dev), n * pad
        return cls.from_seqlens(q_seqlen=q_lens, kv_padding=pad, kv_seqlen=k_lens, device=dev), n * pad
    base = ab.BlockDiagonalMask.from_seqlens(q_lens, k_lens, device=dev)
    make = {"BlockDiagonalMask": lambda: base, "BlockDiagonalCausalMask": base.make_causal,
            "BlockDiagonalCausalFromBottomRightMask": base.make_causal_from_bottomright,
            "BlockDiagonalCausalLocalAttentionMask": lambda: base.make_local_attention(20),
            "BlockDiagonalCausalLocalAttentionFromBottomRightMask": lambda: base.make_local_attention_from_bottomright(20)}
    return make[name](), sum(k_lens)


@gpu
@pytest.mark.parametrize("layout", ["gqa", "mqa", "mha"])
@pytest.mark.parametrize("mq", [1, 3, 40])
@pytest.mark.parametrize("name", [t.__name__ for t, spec in fmha.front._BIASES.items() if spec[0] >= fmha.front._VARLEN])
def test_front_gives_what_python_gives_on_sequences(name, mq, layout, monkeypatch):
    require_cuda()
    paged = name.startswith("Paged")
    gen = torch.Generator().manual_seed(mq)
    q_lens, k_lens, pad, page = [mq] * 3, [50, 90, 64], 96, 32
    bias, rows = _bias(name, q_lens, k_lens, pad, page)
    heads = {"gqa": (2, 4), "mqa": (4,), "mha": (3,)}[layout]
    if paged and mq * (1 if layout == "mha" else 4) > 64:
        pytest.skip("more query rows than the decode operator takes")
    q = _mk(gen, 1, sum(q_lens), *heads, 64)
    if layout == "mha":
        k, v = (_mk(gen, 1, rows, *heads, 64) for _ in range(2))
    else:
        k, v = (_mk(gen, 1, rows, *heads[:-1], 1, 64).expand(1, rows, *heads, 64) for _ in range(2))
    _same(*_both(monkeypatch, lambda: xops.memory_efficient_attention_forward(q, k, v, bias)))
    _same(*_both(monkeypatch, lambda: fmha.memory_efficient_attention_partial(q, k, v, bias, scale=0.2)))
    _same(*_both(monkeypatch, lambda: fmha.memory_efficient_attention_forward_requires_grad(q, k, v, bias, output_dtype=torch.float32)))


@gpu
@pytest.mark.parametrize("five", [False, True])
@pytest.mark.parametrize("kind", ["none", "causal", "bottom_right", "window", "window_br", "band", "tensor", "causal_tensor"])
@pytest.mark.parametrize("mq", [2, 70])
def test_front_gives_what_python_gives_on_dense_batches(kind, mq, five, monkeypatch):
    require_cuda()
    gen = torch.Generator().manual_seed(mq)
    heads, n = ((2, 3) if five else (3,)), 130
    q = _mk(gen, 2, mq, *heads, 72, dtype=torch.float16)
    k, v = (_mk(gen, 2, n, *heads, 72, dtype=torch.float16) for _ in range(2))
    t = _mk(gen, 2, *heads, mq, n, dtype=torch.float32)
    bias = {"none": None, "causal": ab.LowerTriangularMask(), "bottom_right": ab.LowerTriangularFromBottomRightMask(),
            "window": ab.LowerTriangularMaskLocalAttention(20), "window_br": ab.LowerTriangularFromBottomRightLocalAttentionMask(20),
            "band": ab.LocalAttentionFromBottomRightMask(5, 4), "tensor": t, "causal_tensor": ab.LowerTriangularMaskWithTensorBias(t)}[kind]
    _same(*_both(monkeypatch, lambda: xops.memory_efficient_attention_forward(q, k, v, bias)))
    _same(*_both(monkeypatch, lambda: fmha.memory_efficient_attention_forward_requires_grad(q, k, v, bias, op=fmha.b200.FwOp)))


@gpu
def test_front_on_quantised_caches_rope_and_merge(monkeypatch):
    require_cuda()
    import oracle

    gen = torch.Generator().manual_seed(5)
    bias, rows = _bias("PagedBlockDiagonalCausalWithOffsetPaddedKeysMask", [1] * 3, [50, 90, 64], 96, 32)
    for heads in ((8, 4), (8,)):
        q = _mk(gen, 1, 3, *heads, 128)
        kv = (8, 1) if len(heads) == 2 else (1,)
        grown = (1, rows, *heads)
        raw = torch.randn(1, rows, *kv, 128, generator=gen)
        k4 = oracle.quantize_kv_int4(raw).cuda()
        v4 = k4.flip(1)
        _same(*_both(monkeypatch, lambda: xops.memory_efficient_attention_forward(q, k4.expand(*grown, -1), v4.expand(*grown, -1), bias)))
        k8 = torch.randint(0, 1 << 30, (1, rows, *kv, 32), generator=gen).int().bitwise_and(0x3F3F3F3F).cuda()
        w8 = torch.full((1, rows, *kv), 0x00002C00, dtype=torch.int32).cuda()
        inp = fmha.common.InputsFp8(q, k8.expand(*grown, -1), k8.flip(1).expand(*grown, -1), bias, k_fp8_scale_shift=w8.expand(*grown), v_fp8_scale_shift=w8.expand(*grown))
        _same(*_both(monkeypatch, lambda: fmha._memory_efficient_attention_forward(inp, op=fmha.triton_splitk.FwOp)))

    stub = types.SimpleNamespace(split_k=_lib.front.split_k, rope=lambda *a: None, merge=lambda *a: None, dense=lambda *a: None, varlen=lambda *a: None)
    for dtype, int4, paged in ((torch.bfloat16, False, False), (torch.float32, False, True), (torch.float16, True, True)):
        cls = "PagedBlockDiagonalCausalWithOffsetPaddedKeysMask" if paged else "BlockDiagonalCausalWithOffsetPaddedKeysMask"
        rb, rr = _bias(cls, [2, 5, 1], [50, 90, 64], 96, 32)
        xq = _mk(gen, 1, 8, 2, 4, 64, dtype=dtype)
        xk, xv = (_mk(gen, 1, 8, 2, 1, 64, dtype=dtype) for _ in range(2))
        got = []
        for f in (_lib.front, stub):
            monkeypatch.setattr(_lib, "front", f)
            ck, cv = (torch.zeros(1, rr, 2, 1, 9 if int4 else 64, dtype=torch.int32 if int4 else dtype, device="cuda") for _ in range(2))
            got.append((xops.rope_padded(xq, xk, xv, ck, cv, rb, theta=5000.0, adjacents=False), ck, cv))
        monkeypatch.undo()
        _same(*got)
    parts, lses = [_mk(gen, 1, 6, 2, 3, 64) for _ in range(3)], [_mk(gen, 1, 2, 3, 6, dtype=torch.float32) for _ in range(3)]
    got = []
    for f in (_lib.front, stub):
        monkeypatch.setattr(_lib, "front", f)
        got.append(fmha.merge_attentions(parts, lses, output_dtype=torch.float32))
    monkeypatch.undo()
    _same(*got)


@gpu
def test_front_leaves_the_unusual_to_python(monkeypatch):
    """Parameters, 3-D inputs, operators with a fixed split count, status checks: the Python path serves these."""
    require_cuda()
    gen = torch.Generator().manual_seed(6)
    q, k, v = (_mk(gen, 1, 33, 4, 64) for _ in range(3))
    run = lambda q, k, v, **kw: lambda: xops.memory_efficient_attention_forward(q, k, v, ab.LowerTriangularMask(), **kw)
    _both(monkeypatch, run(torch.nn.Parameter(q, requires_grad=False), k, v), takes=False)
    _both(monkeypatch, run(*(x[0].transpose(0, 1).contiguous() for x in (q, k, v))), takes=False)
    _both(monkeypatch, run(q, k, v, op=fmha.b200.FwOp_Generic), takes=False)
    monkeypatch.setenv("XFB200_CHECK_STATUS", "1")
    _both(monkeypatch, run(q, k, v), takes=False)
    monkeypatch.setenv("XFB200_CHECK_STATUS", "0")
    _both(monkeypatch, run(q, k, v), takes=True)
    with pytest.raises(ValueError):  # the Python path's message, not a crash
        xops.memory_efficient_attention_forward(q, k[:, :, :2], v, None)


@gpu
@pytest.mark.parametrize("op", [None, "named"])
def test_front_leaves_changed_operators_to_python(op, monkeypatch):
    """What a program sets on the operator classes themselves counts: settings and methods."""
    require_cuda()
    gen = torch.Generator().manual_seed(7)
    decode, prefill = fmha.b200_splitk.FwOp, fmha.b200.FwOp
    qd = _mk(gen, 1, 1, 2, 4, 128)
    kd, vd = (_mk(gen, 1, 4096, 2, 1, 128).expand(-1, -1, -1, 4, -1) for _ in range(2))
    q, k, v = (_mk(gen, 1, 33, 4, 64) for _ in range(3))
    step = lambda: xops.memory_efficient_attention_forward(qd, kd, vd, None, op=op and decode)
    prompt = lambda: xops.memory_efficient_attention_forward(q, k, v, ab.LowerTriangularMask(), op=op and prefill)
    splits, paths = [], []
    for call, cls, name, value in ((step, decode, "SPLIT_K", 3), (step, decode, "get_split_k", classmethod(lambda c, *a, **kw: splits.append(a) or 2)),
                                   (prompt, prefill, "KERNEL_PATH", _lib.PREFILL_MMA_SYNC), (prompt, prefill, "_WAIT_BUDGET_KCYCLES", 100000),
                                   (prompt, prefill, "apply", classmethod(lambda c, inp, needs_gradient: paths.append(1) or (torch.zeros_like(inp.query), None)))):
        with monkeypatch.context() as m:
            m.setattr(cls, name, value)
            _both(m, call, takes=False)
        _both(monkeypatch, call, takes=True)
    assert splits and len(paths) == 2


@gpu
def test_calls_without_the_front(monkeypatch):
    """Every kind of call that the front serves, with no front at all."""
    require_cuda()
    gen = torch.Generator().manual_seed(9)
    bias, rows = _bias("BlockDiagonalCausalWithOffsetPaddedKeysMask", [1] * 3, [50, 90, 64], 96, 32)
    xq, xk, xv = _mk(gen, 1, 3, 2, 4, 64), _mk(gen, 1, 3, 2, 1, 64), _mk(gen, 1, 3, 2, 1, 64)
    q, k, v = (_mk(gen, 1, 33, 4, 64) for _ in range(3))
    got = []
    for f in (_lib.front, None):
        monkeypatch.setattr(_lib, "front", f)
        ck, cv = (torch.ones(1, rows, 2, 1, 64, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        r = xops.rope_padded(xq, xk, xv, ck, cv, bias)
        o, l = fmha.memory_efficient_attention_partial(r, ck.expand(-1, -1, -1, 4, -1), cv.expand(-1, -1, -1, 4, -1), bias)
        got.append((ck, cv, r, o, l, *fmha.merge_attentions([o, o], [l, l]), xops.memory_efficient_attention_forward(q, k, v, ab.LowerTriangularMask())))
    monkeypatch.undo()
    _same(*got)
