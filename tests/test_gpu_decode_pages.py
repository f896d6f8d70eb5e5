"""Decode over paged caches with many pages per chunk: the copy warp's look-ahead through the page table (windows of 32 entries)
against the padded cache, bit for bit, and against the oracle."""

import pytest
import torch

import oracle
from gpu_utils import assert_o_lse, gpu, require_cuda
from xformers_b200.ops import fmha
from xformers_b200.ops.fmha import attn_bias as ab

S = fmha.b200_splitk


@gpu
@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("split_k", [None, 1])
@pytest.mark.parametrize("page", [1, 4, 8, 16, 24, 48, 1536])
@pytest.mark.parametrize("kv_heads,group", [(8, 8), (1, 16), (2, 4)])
def test_small_pages(kv_heads, group, page, split_k, quant):
    require_cuda()
    dtype, D, max_t = torch.bfloat16, 128, 1536
    lens = [max_t, 1, 1499, 513]  # more than two windows of 16-token pages, and their edge
    B = len(lens)
    g = torch.Generator().manual_seed(78)
    q = torch.randn(1, B, kv_heads, group, D, generator=g).to(dtype).cuda()
    kf, vf = (torch.randn(1, B * max_t, kv_heads, 1, D, generator=g) for _ in range(2))
    if quant:
        k_pad, v_pad = oracle.quantize_kv_int4(kf), oracle.quantize_kv_int4(vf)
        k_ref, v_ref = oracle.dequantize_kv_int4(k_pad), oracle.dequantize_kv_int4(v_pad)
    else:
        k_pad, v_pad = kf.to(dtype), vf.to(dtype)
        k_ref, v_ref = k_pad.float(), v_pad.float()
    expand = lambda t: t.expand(-1, -1, -1, group, -1)
    pad_bias = ab.BlockDiagonalPaddedKeysMask.from_seqlens([1] * B, max_t, lens, device="cuda")
    n_pages = B * (max_t // page)
    perm = torch.randperm(n_pages, generator=g).int().view(B, -1)
    k_pg, v_pg = (oracle.scatter_to_pages(t, perm, page, [max_t] * B, max_t, n_pages) for t in (k_pad, v_pad))
    bias = pad_bias.make_paged(perm.cuda(), page, ab.PagedBlockDiagonalPaddedKeysMask)
    op = S.FwOp if split_k is None else type("Op", (S.FwOp,), {"SPLIT_K": split_k})
    run = lambda k, v, b: fmha.memory_efficient_attention_forward_requires_grad(q, expand(k.cuda()), expand(v.cuda()), b, op=op)
    out, lse = run(k_pg, v_pg, bias)
    ro, rl = oracle.ref_attention_with_lse(q.float().cpu(), expand(k_ref), expand(v_ref), pad_bias.to("cpu"))
    assert_o_lse(out, lse, ro, rl, dtype, f"pages of {page}")
    out_pad, lse_pad = run(k_pad, v_pad, pad_bias)
    assert torch.equal(out, out_pad) and torch.equal(lse, lse_pad), "page placement must not change a single bit"


@gpu
def test_nan_behind_a_vanishing_weight():
    """A NaN in V makes the output NaN whatever the weight of its chunk, also one that underflows to zero in the merge."""
    require_cuda()
    q = torch.ones(1, 1, 1, 8, 128, device="cuda", dtype=torch.bfloat16)
    k = torch.zeros(1, 512, 1, 1, 128, device="cuda", dtype=torch.bfloat16)
    k[:, 300] = 40.0  # a score of 450; the keys of the other chunks weigh exp(-450)
    v = torch.ones(1, 512, 1, 1, 128, device="cuda", dtype=torch.bfloat16)
    v[0, 5, 0, 0, 7] = float("nan")
    bias = ab.BlockDiagonalPaddedKeysMask.from_seqlens([1], 512, [512], device="cuda")
    op = type("Op", (S.FwOp,), {"SPLIT_K": 4})
    out = fmha.memory_efficient_attention_forward(q, k.expand(-1, -1, -1, 8, -1), v.expand(-1, -1, -1, 8, -1), bias, op=op)
    assert out[..., 7].isnan().all() and (out[..., :7] == 1).all() and (out[..., 8:] == 1).all()
