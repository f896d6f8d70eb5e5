"""Launches that begin before the kernel ahead of them has ended, and the order and size of the prefill kernel's work items:
results must be those of calls that are waited for, and of the oracle."""

import time

import pytest
import torch

import xformers_b200.ops as xops
from gpu_utils import assert_o_lse, gpu, rand_qkv, ref, require_cuda
from xformers_b200.ops import fmha
from xformers_b200.ops.fmha import attn_bias as ab


@gpu
@pytest.mark.parametrize("capture", [False, True])
@pytest.mark.parametrize("kv_heads,mq", [(8, 1), (1, 2)])
def test_steps_back_to_back(kv_heads, mq, capture):
    """Decoding steps whose every kernel reads what the one before it wrote (cache, lengths, partials, scratch that the
    allocator hands out again)."""
    require_cuda()
    B, pad, G, D, steps = 3, 2048, 8, 128, 12
    g = torch.Generator(device="cuda").manual_seed(11)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=torch.bfloat16)
    xq, xk, xv = rnd(1, B * mq, kv_heads, G, D), rnd(1, B * mq, kv_heads, 1, D), rnd(1, B * mq, kv_heads, 1, D)
    ck0, cv0 = rnd(1, B * pad, kv_heads, 1, D), rnd(1, B * pad, kv_heads, 1, D)
    lens0 = [5, 1400, 2000]

    def run(wait, graph):
        ck, cv, x = ck0.clone(), cv0.clone(), xq.clone()
        bias = ab.BlockDiagonalCausalWithOffsetPaddedKeysMask.from_seqlens(q_seqlen=[mq] * B, kv_padding=pad, kv_seqlen=lens0, device="cuda")
        k, v = (c.expand(-1, -1, -1, G, -1) for c in (ck, cv))

        def step():
            q = xops.rope_padded(x, xk, xv, ck, cv, bias)
            if wait:
                torch.cuda.synchronize()
            parts = [fmha.memory_efficient_attention_partial(q, k, v, bias) for _ in range(2)]
            if wait:
                torch.cuda.synchronize()
            out, lse = fmha.merge_attentions([o for o, _ in parts], [l for _, l in parts])
            x.copy_(out)
            bias.k_seqinfo.seqlen.add_(1)
            return out, lse

        outs = []
        if graph:
            warm = torch.cuda.Stream()
            with torch.cuda.stream(warm):
                step()
            warm.synchronize()
            cg = torch.cuda.CUDAGraph()
            with torch.cuda.graph(cg):
                res = step()
            ck.copy_(ck0), cv.copy_(cv0), x.copy_(xq), bias.k_seqinfo.seqlen.copy_(torch.tensor(lens0, dtype=torch.int32, device="cuda"))
            for _ in range(steps):
                cg.replay()
                outs.append(tuple(t.clone() for t in res))
        else:
            for _ in range(steps):
                outs.append(tuple(t.clone() for t in step()))
        return outs, ck, cv

    got, ck, cv = run(False, capture)
    want, ck_w, cv_w = run(True, False)
    assert torch.equal(ck, ck_w) and torch.equal(cv, cv_w)
    for (o, l), (ow, lw) in zip(got, want):
        assert torch.equal(o, ow) and torch.equal(l, lw)


@gpu
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33])
@pytest.mark.parametrize("heads", [2, 8])
def test_order_of_sequences(n, heads):
    """Packed batches on both sides of the number of sequences that a warp ranks; empty ones, equal ones, keys without queries."""
    require_cuda()
    g = torch.Generator().manual_seed(n)
    ql = torch.randint(0, 200, (n,), generator=g).tolist()
    kl = [q + int(torch.randint(0, 600, (1,), generator=g)) for q in ql]
    ql[0], kl[0] = 150, 150
    if n > 2:
        ql[1], kl[1] = 0, 300
        ql[2], kl[2] = 150, 150
    q, k, v = rand_qkv(1, sum(kl), sum(kl), 1, heads, 128, torch.bfloat16, seed=n)
    q = q[:, : sum(ql)]
    bias = ab.BlockDiagonalCausalFromBottomRightMask.from_seqlens(ql, kl, device="cuda")
    out, lse = fmha.memory_efficient_attention_forward_requires_grad(q, k, v, bias, op=fmha.b200.FwOp)
    ro, rl = ref(q, k, v, bias)
    assert_o_lse(out, lse, ro, rl, torch.bfloat16, f"{n} sequences")


@gpu
@pytest.mark.parametrize("mask", ["none", "causal", "bottom_right", "window"])
@pytest.mark.parametrize("m", [1, 128, 129, 2304, 2305])
@pytest.mark.parametrize("D", [64, 80, 128])
def test_items_of_one_tile(D, m, mask):
    """8 heads: up to 2304 rows (144 tiles) a work item is one tile of 128 rows, from 2305 rows on it is two."""
    require_cuda()
    keys = {"none": 300, "causal": m, "bottom_right": m + 77, "window": m}[mask]
    bias = {"none": None, "causal": ab.LowerTriangularMask(), "bottom_right": ab.LowerTriangularFromBottomRightMask(),
            "window": ab.LowerTriangularFromBottomRightLocalAttentionMask(100) if m > 1 else ab.LowerTriangularMask()}[mask]
    q, k, v = (t[:, :, 0] for t in rand_qkv(1, m, keys, 1, 8, D, torch.float16, seed=m, gqa=False))
    out, lse = fmha.memory_efficient_attention_forward_requires_grad(q, k, v, bias, op=fmha.b200.FwOp)
    ro, rl = ref(q, k, v, bias)
    assert_o_lse(out, lse, ro, rl, torch.float16, f"{mask} m={m}")


@gpu
@pytest.mark.parametrize("m,heads", [(200, 4), (2500, 16)])
def test_prefills_back_to_back(m, heads):
    """Prefill calls that read the output of the one before, on launches smaller and larger than the machine."""
    require_cuda()
    q0, k, v = (t[:, :, 0] for t in rand_qkv(1, m, m, 1, heads, 128, torch.bfloat16, seed=3, gqa=False))

    def run(wait):
        q, outs = q0, []
        for _ in range(8):
            q = fmha.memory_efficient_attention_forward(q, k, v, ab.LowerTriangularMask(), op=fmha.b200.FwOp)
            q = fmha.memory_efficient_attention_forward(q, q, v, None, op=fmha.b200.FwOp) * 3
            if wait:
                torch.cuda.synchronize()
            outs.append(q)
        return outs

    for a, b in zip(run(False), run(True)):
        assert torch.equal(a, b)


@gpu
def test_capture_behind_copies_and_joined_streams():
    """Captured launches whose predecessor is a copy, and whose stream has just joined another one."""
    require_cuda()
    q, k, v = (t[:, :, 0] for t in rand_qkv(1, 300, 300, 1, 4, 128, torch.bfloat16, seed=5, gqa=False))
    qg, kg, vg = rand_qkv(2, 1, 3000, 2, 8, 128, torch.bfloat16, seed=6)
    x, y = torch.zeros_like(q), torch.zeros_like(qg)

    def work(side):
        main = torch.cuda.current_stream()
        x.copy_(q)
        a = fmha.memory_efficient_attention_forward(x, k, v, ab.LowerTriangularMask(), op=fmha.b200.FwOp)
        side.wait_stream(main)
        with torch.cuda.stream(side):
            y.copy_(qg)
            b, lse = fmha.memory_efficient_attention_partial(y, kg, vg, op=fmha.b200_splitk.FwOp)
        c = fmha.memory_efficient_attention_forward(a, k, v, None, op=fmha.b200.FwOp)
        main.wait_stream(side)
        d, _ = fmha.memory_efficient_attention_partial(b, kg, vg, op=fmha.b200_splitk.FwOp)
        m, _ = fmha.merge_attentions([b, d], [lse, lse])
        return c, m

    side = torch.cuda.Stream()
    want = [t.clone() for t in work(side)]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = work(side)
    for _ in range(5):
        x.zero_(), y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@gpu
def test_free_sms_stay_free_between_two_launches():
    """Two launches that leave SMs free, one behind the other: a kernel of another stream runs beside the first of them, it does
    not wait for its end (as it does where the second one's CTAs already sit on those SMs)."""
    require_cuda()
    q, k, v = (t[:, :, 0] for t in rand_qkv(1, 16384, 16384, 1, 32, 128, torch.bfloat16, seed=8, gqa=False))
    inp = fmha.Inputs(q, k, v, None)
    x, side = torch.zeros(1024, device="cuda"), torch.cuda.Stream()
    shares = []
    for _ in range(4):  # (the first loads the kernels)
        start, small, end = (torch.cuda.Event(enable_timing=True) for _ in range(3))
        torch.cuda.synchronize()
        start.record()
        for _ in range(2):
            fmha.b200.FwOp._apply(inp, False, sm_margin=8)  # 3.5 ms each
        end.record()
        time.sleep(0.0005)  # both are with the GPU now
        with torch.cuda.stream(side):
            x.add_(1)
            small.record()
        torch.cuda.synchronize()
        shares.append(start.elapsed_time(small) / start.elapsed_time(end))
    assert min(shares[1:]) < 0.3, f"the other stream's kernel ended after {shares} of both launches"
