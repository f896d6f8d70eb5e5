"""The order in which the prefill kernel takes the sequences of a packed batch."""

import pytest
import torch

from gpu_utils import assert_o_lse, gpu, rand_qkv, ref, require_cuda
from xformers_b200.ops import fmha
from xformers_b200.ops.fmha import attn_bias as ab


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
