"""Attention over the KV blocks selected per query token (topk_sparse_attention).

Signature follows native_sparse_attention/ops/triton/topk_sparse_attention.py:1182-1217 of the reference.
"""
from typing import Optional

import torch

from .. import _lib


def topk_sparse_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, topk_idx: torch.Tensor, block_size: int,
                          cu_seqlens: torch.Tensor, softmax_scale: Optional[float] = None) -> torch.Tensor:
    """Each query attends, causally, to the keys of its selected blocks.

    Args:
        q: [total_len, num_q_heads, head_dim]
        k, v: [total_len, num_kv_heads, head_dim]
        topk_idx: int32 [num_kv_heads, total_len, topk], valid block ids first, -1 padding; the keys of an id given twice
            count twice, forward and backward, as in the single-token operator
        block_size: keys per block (multiple of 64)
        cu_seqlens: int32 [batch + 1]
        softmax_scale: default 1/sqrt(head_dim)
    Returns:
        attention output [total_len, num_q_heads, head_dim]
    """
    assert block_size in (32, 64, 128, 256), "block_size must be 32, 64, 128 or 256"
    return _lib.host().topk_sparse_attention(q, k, v, topk_idx, int(block_size), cu_seqlens, softmax_scale)
