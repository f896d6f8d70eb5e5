"""The consumers of the quantised caches at the edges of their tiles: sub-tiles, pairs of sub-tiles and stages cut anywhere,
8 and more query rows per kv head, every number of kv heads per CTA, and queries of extreme magnitude."""

import pytest
import torch

import oracle
from gpu_utils import assert_o_lse, gpu, require_cuda
from xformers_b200.ops import fmha
from xformers_b200.ops.fmha import attn_bias as ab

S = fmha.triton_splitk
LENS = [1, 15, 16, 17, 31, 32, 33, 64, 127, 129, 255, 256, 257, 300]


def _run(fmt, kv_heads, group, D, dtype, mag, mq=1, split_k=1):
    g = torch.Generator().manual_seed(5)
    B, pad = len(LENS), 320
    lens = [max(n, mq) for n in LENS]
    q = (torch.randn(1, B * mq, kv_heads, group, D, generator=g) * mag).to(dtype)
    kf, vf = (torch.randn(1, B * pad, kv_heads, 1, D, generator=g) for _ in range(2))
    expand = lambda t: t.expand(-1, -1, -1, group, *t.shape[4:])
    bias = ab.BlockDiagonalCausalWithOffsetPaddedKeysMask.from_seqlens(q_seqlen=[mq] * B, kv_padding=pad, kv_seqlen=lens, device="cuda")
    op = type("Op", (S.FwOp,), {"SPLIT_K": split_k})
    scale = D**-0.5 / mag
    if fmt == "int4":
        kc, vc = oracle.quantize_kv_int4(kf), oracle.quantize_kv_int4(vf)
        k_ref, v_ref = oracle.dequantize_kv_int4(kc), oracle.dequantize_kv_int4(vc)
        out, lse = fmha.memory_efficient_attention_forward_requires_grad(q.cuda(), expand(kc.cuda()), expand(vc.cuda()), bias, scale=scale, op=op)
    else:
        def quantise(x):
            x8, sc, sh = oracle.quantize_fp8_asymmetric(x.reshape(-1, D))
            words = oracle.combine_scale_shift(sc, sh)
            return x8, words, oracle.dequantize_fp8_asymmetric(x8, *oracle.split_scale_shift(words)).view(x.shape)

        (k8, kss, k_ref), (v8, vss, v_ref) = quantise(kf), quantise(vf)
        rows = lambda x8: expand(oracle.pack_fp8_words(x8).view(1, B * pad, kv_heads, 1, D // 4).cuda())
        word = lambda w: expand(w.view(1, B * pad, kv_heads, 1).cuda())
        inp = S.InputsFp8(query=q.cuda(), key=rows(k8), value=rows(v8), attn_bias=bias, scale=scale, k_fp8_scale_shift=word(kss), v_fp8_scale_shift=word(vss))
        out, ctx = fmha._memory_efficient_attention_forward_requires_grad(inp, op=op)
        lse = ctx.lse
    ro, rl = oracle.ref_attention_with_lse(q.float(), expand(k_ref), expand(v_ref), bias.to("cpu"), scale)
    assert_o_lse(out, lse, ro, rl, dtype, f"{fmt} {kv_heads}x{group} D={D}")


@gpu
@pytest.mark.parametrize("split_k", [1, 3])
@pytest.mark.parametrize("group,mq", [(8, 1), (9, 1), (16, 1), (17, 1), (4, 3)])
@pytest.mark.parametrize("kv_heads", [1, 2, 4, 8])
@pytest.mark.parametrize("fmt,D", [("int4", 64), ("int4", 128), ("fp8", 128)])
def test_quantised_tile_edges(fmt, D, kv_heads, group, mq, split_k):
    require_cuda()
    _run(fmt, kv_heads, group, D, torch.bfloat16 if group % 2 else torch.float16, 1.0, mq, split_k)


# Queries are brought to f16 by a power of two per row.  fp8: only downwards, so small ones must be normal f16 values.
@gpu
@pytest.mark.parametrize("fmt,dtype,mag", [("int4", torch.bfloat16, 2.0**-90), ("int4", torch.bfloat16, 2.0**110), ("int4", torch.float16, 2.0**-8),
                                           ("int4", torch.float16, 2.0**13), ("fp8", torch.bfloat16, 2.0**110), ("fp8", torch.float16, 2.0**13)])
def test_quantised_query_magnitudes(fmt, dtype, mag):
    require_cuda()
    _run(fmt, 2, 8, 128, dtype, mag)


def _int4_rows(scale, shift, n):
    """Rows of the int4 format: [rows] scales and shifts, [rows, D] nibbles -> [rows, 1 + D / 8] words."""
    half = lambda x: x.half().view(torch.int16).long() & 0xFFFF
    packed = (n.long().view(n.shape[0], -1, 8) << torch.arange(0, 32, 4)).sum(-1)
    w = torch.cat([(half(scale) | half(shift) << 16)[:, None], packed], 1)
    return torch.where(w >= 1 << 31, w - (1 << 32), w).int()


@gpu
@pytest.mark.parametrize("peaks", ["one per sub-tile", "any weight"])
@pytest.mark.parametrize("kv_heads,group", [(1, 8), (2, 16), (8, 4)])
@pytest.mark.parametrize("D", [64, 128])
def test_int4_columns_are_equally_accurate(D, kv_heads, group, peaks):
    """f32 output.  The tensor core cuts the products of a sub-tile off against the largest of them, so their place in the 16
    bits counts: neighbouring columns that hold the same values must give the same bits.  The weights are powers of two (f16
    holds them and V's scales exactly), so that these cuts and those of the running sum are the error."""
    require_cuda()
    N = 4096
    g = torch.Generator().manual_seed(D)
    q = torch.zeros(1, 1, kv_heads, group, D, dtype=torch.bfloat16)
    q[..., 0] = 1
    kn = torch.zeros(N, D, dtype=torch.int32)
    kn[:, 0] = 2
    kn[::16, 0] = 15
    if peaks == "any weight":
        kn[:, 0] = torch.randint(0, 16, (N,), generator=g)
    vn = torch.randint(0, 16, (N, D // 2), generator=g).repeat_interleave(2, -1)
    vs = 1 + torch.randint(0, 1024, (N,), generator=g) / 1024.0
    cache = lambda words: words.cuda().view(1, N, 1, 1, -1).expand(-1, -1, kv_heads, -1, -1).contiguous().expand(-1, -1, -1, group, -1)
    k, v = cache(_int4_rows(torch.ones(N), torch.full((N,), -15.0), kn)), cache(_int4_rows(vs, torch.zeros(N), vn))
    out, _ = fmha.memory_efficient_attention_partial(q.cuda(), k, v, None, scale=0.6931471805599453, op=S.FwOp_S1, output_dtype=torch.float32)
    assert torch.equal(out[..., 0::2], out[..., 1::2])
    p = torch.exp2(kn[:, 0].double() - 15)
    want = (p[:, None] * vn.double() * vs[:, None].double()).sum(0) / p.sum()
    # a warp adds its sub-tiles of 16 keys (8 warps share the heads) to f32 sums that are cut off, not rounded: 2^-23 each; one
    # more 2^-22 for the exponentials and the sum over the warps.  Measured: 3.1e-6, 6.2e-6, 2.6e-5 with 1, 2, 8 kv heads.
    assert ((out.double().cpu() - want) / want).abs().max() <= N // 16 * kv_heads // 8 * 2.0**-23 + 2.0**-22
