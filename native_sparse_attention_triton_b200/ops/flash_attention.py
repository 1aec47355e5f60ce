"""Dense varlen attention (flash_attention_varlen) on the shared strided-causal kernel.

Signature follows native_sparse_attention/ops/triton/flash_attention.py:895-935 of the reference.
`gqa_interleave=True` is rejected: the reference's forward and backward disagree on that head mapping.
"""
from typing import Optional

import torch

from .. import _lib


def flash_attention_varlen(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, cu_seqlens_q: torch.Tensor,
                           cu_seqlens_k: torch.Tensor, max_seqlen_q: int, max_seqlen_k: int, causal: bool = False,
                           sm_scale: Optional[float] = None, gqa_interleave: bool = False) -> torch.Tensor:
    """Varlen GQA attention; causal means key j is visible to query i iff j <= i within a sequence."""
    if gqa_interleave:
        raise NotImplementedError("gqa_interleave=True is not supported")
    return _lib.host().flash_attention_varlen(q, k, v, cu_seqlens_q, cu_seqlens_k, int(max_seqlen_q), int(max_seqlen_k), bool(causal), sm_scale)
