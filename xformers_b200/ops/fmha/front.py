"""Way from the public entry points to the host front (csrc/front.cpp).

Every function here returns the call's result, or ``None`` when the front does
not take the call: the entry point then goes through :class:`~.common.Inputs`,
the dispatcher and the operator classes, which run it or raise its error.  The
tables only say how a bias object of a given type is read.
"""

from __future__ import annotations

from typing import Any, Optional, Tuple

import torch

from ... import _lib
from . import attn_bias as ab
from . import b200, b200_splitk
from .common import InputsFp8

_DENSE, _TENSOR, _VARLEN, _PADDED, _PAGED = range(5)
_PLAIN, _CAUSAL_WINDOW, _BAND = range(3)
WANT_LSE, PARTIAL, _DECODE, _PREFILL, _FORCE_DECODE, _FORCE_PREFILL = 1, 2, 4, 8, 16, 32
_BOTH = _DECODE | _PREFILL
_NONE, _TL, _BR, _LOCAL = _lib.MASK_NONE, _lib.MASK_CAUSAL_TOP_LEFT, _lib.MASK_CAUSAL_BOTTOM_RIGHT, _lib.MASK_LOCAL_BOTTOM_RIGHT

# bias type -> (how its sequences are read, operators that take it, mask, window attributes)
_BIASES = {
    type(None): (_DENSE, _BOTH, _NONE, _PLAIN),
    torch.Tensor: (_TENSOR, _BOTH, _NONE, _PLAIN),
    ab.LowerTriangularMaskWithTensorBias: (_TENSOR, _PREFILL, _TL, _PLAIN),
    ab.LowerTriangularMask: (_DENSE, _PREFILL, _TL, _PLAIN),
    ab.LowerTriangularFromBottomRightMask: (_DENSE, _PREFILL, _BR, _PLAIN),
    ab.LowerTriangularMaskLocalAttention: (_DENSE, _PREFILL, _TL, _CAUSAL_WINDOW),
    ab.LowerTriangularFromBottomRightLocalAttentionMask: (_DENSE, _PREFILL, _BR, _CAUSAL_WINDOW),
    ab.LocalAttentionFromBottomRightMask: (_DENSE, _PREFILL, _LOCAL, _BAND),
    ab.BlockDiagonalMask: (_VARLEN, _PREFILL, _NONE, _PLAIN),
    ab.BlockDiagonalCausalMask: (_VARLEN, _PREFILL, _TL, _PLAIN),
    ab.BlockDiagonalCausalFromBottomRightMask: (_VARLEN, _PREFILL, _BR, _PLAIN),
    ab.BlockDiagonalCausalLocalAttentionMask: (_VARLEN, _PREFILL, _TL, _CAUSAL_WINDOW),
    ab.BlockDiagonalCausalLocalAttentionFromBottomRightMask: (_VARLEN, _PREFILL, _BR, _CAUSAL_WINDOW),
    ab.BlockDiagonalPaddedKeysMask: (_PADDED, _BOTH, _NONE, _PLAIN),
    ab.BlockDiagonalCausalWithOffsetPaddedKeysMask: (_PADDED, _BOTH, _BR, _PLAIN),
    ab.BlockDiagonalCausalLocalAttentionPaddedKeysMask: (_PADDED, _BOTH, _BR, _CAUSAL_WINDOW),
    ab.BlockDiagonalLocalAttentionPaddedKeysMask: (_PADDED, _PREFILL, _LOCAL, _BAND),
    ab.BlockDiagonalGappyKeysMask: (_PADDED, _BOTH, _NONE, _PLAIN),
    ab.BlockDiagonalCausalWithOffsetGappyKeysMask: (_PADDED, _BOTH, _BR, _PLAIN),
    ab.BlockDiagonalLocalAttentionFromBottomRightGappyKeysMask: (_PADDED, _PREFILL, _LOCAL, _BAND),
    ab.PagedBlockDiagonalPaddedKeysMask: (_PAGED, _DECODE, _NONE, _PLAIN),
    ab.PagedBlockDiagonalCausalWithOffsetPaddedKeysMask: (_PAGED, _DECODE, _BR, _PLAIN),
    ab.PagedBlockDiagonalCausalLocalPaddedKeysMask: (_PAGED, _DECODE, _BR, _CAUSAL_WINDOW),
}
_GAPPY = (ab.BlockDiagonalGappyKeysMask, ab.BlockDiagonalCausalWithOffsetGappyKeysMask, ab.BlockDiagonalLocalAttentionFromBottomRightGappyKeysMask)
# operators a caller may name
_OPS = {
    None: 0,
    b200_splitk.FwOp: _FORCE_DECODE,
    b200.FwOp: _FORCE_PREFILL,
    (b200_splitk.FwOp, None): _FORCE_DECODE,
    (b200.FwOp, None): _FORCE_PREFILL,
}
_Tensor = torch.Tensor
_DECODE_CLS, _PREFILL_CLS = b200_splitk.FwOp.__dict__, b200.FwOp.__dict__  # (views: they follow the classes)
_SPLIT, _DECODE_APPLY, _DECODE_REASONS = (_DECODE_CLS[n] for n in ("get_split_k", "apply", "not_supported_reasons"))
_PREFILL_APPLY, _PREFILL_REASONS = (_PREFILL_CLS[n] for n in ("apply", "not_supported_reasons"))


def _as_shipped() -> bool:
    """The front knows the operators as they are; settings and methods replaced on the classes themselves are the Python path's."""
    d, p = _DECODE_CLS, _PREFILL_CLS
    return (d["SPLIT_K"] is None and d["NUM_GROUPS"] == 1 and d["get_split_k"] is _SPLIT and d["apply"] is _DECODE_APPLY
            and d["not_supported_reasons"] is _DECODE_REASONS and p["KERNEL_PATH"] == _lib.PREFILL_AUTO and not p["_WAIT_BUDGET_KCYCLES"]
            and not p["_DEBUG_FLAGS"] and p["apply"] is _PREFILL_APPLY and p["not_supported_reasons"] is _PREFILL_REASONS)


def forward(q, k, v, bias: Any, p: float, scale: Optional[float], op: Any, output_dtype: Optional[torch.dtype], flags: int,
            k_words: Optional[torch.Tensor] = None, v_words: Optional[torch.Tensor] = None) -> Optional[Tuple[torch.Tensor, Optional[torch.Tensor]]]:
    """``(out, lse or None)`` of an attention call, or ``None``."""
    front, spec, force = _lib.front, _BIASES.get(type(bias)), _OPS.get(op)
    # (a tensor subclass -- a parameter, a fake tensor -- goes the long way)
    if front is None or spec is None or force is None or p != 0.0 or type(q) is not _Tensor or type(k) is not _Tensor or type(v) is not _Tensor:
        return None
    if not _as_shipped():
        return None
    family, takes, mask, window = spec
    flags |= takes | force
    left, right = -1, 0
    if window == _CAUSAL_WINDOW:
        left = bias._window_size - 1
    elif window == _BAND:
        left, right = bias.window_left, bias.window_right
    if family == _DENSE:
        return front.dense(q, k, v, None, flags, mask, left, right, scale, output_dtype)
    if family == _TENSOR:
        return front.dense(q, k, v, bias if mask == _NONE else bias._bias, flags, mask, left, right, scale, output_dtype)
    qi, ki = bias.q_seqinfo, bias.k_seqinfo
    n = len(qi.seqstart_py) - 1
    if family == _VARLEN:
        return front.varlen(q, k, v, qi.seqstart, ki.seqstart, None, n, qi.max_seqlen, qi.min_seqlen, 0, False, flags, mask, left, right, scale, output_dtype,
                            None, 0, None, None)
    tables, page = (bias.block_tables, bias.page_size) if family == _PAGED else (None, 0)
    return front.varlen(q, k, v, qi.seqstart, ki.seqstart, ki.seqlen, n, qi.max_seqlen, qi.min_seqlen, ki.padding, type(bias) in _GAPPY, flags, mask, left,
                        right, scale, output_dtype, tables, page, k_words, v_words)


def forward_inputs(inp, op: Any, flags: int):
    """The same for a prepared ``Inputs`` / ``InputsFp8`` object."""
    if inp.is_partial:
        flags |= PARTIAL
    if type(inp) is InputsFp8:
        if type(inp.k_fp8_scale_shift) is not _Tensor or type(inp.v_fp8_scale_shift) is not _Tensor or inp.attn_bias is None:
            return None
        return forward(inp.query, inp.key, inp.value, inp.attn_bias, inp.p, inp.scale, op, inp.output_dtype, flags, inp.k_fp8_scale_shift, inp.v_fp8_scale_shift)
    return forward(inp.query, inp.key, inp.value, inp.attn_bias, inp.p, inp.scale, op, inp.output_dtype, flags)
