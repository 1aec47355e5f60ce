"""Single-token (decode) operators against dense KV caches.

Signatures follow the reference:
  flash_attention_decode        native_sparse_attention/ops/triton/flash_attention_decode.py:142-217
  compressed_attention_decode   native_sparse_attention/ops/torch/compressed_attention_decode.py:65-153
  topk_sparse_attention_decode  native_sparse_attention/ops/triton/topk_sparse_attention_decode.py:151-237
Cache tensors may be strided views ([batch, len, kv_heads, d] slices of a larger cache).
"""
from typing import Optional, Tuple

import torch

from .. import _lib


def flash_attention_decode(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, seqlens: torch.Tensor,
                           sm_scale: Optional[float] = None) -> torch.Tensor:
    """One query token per sequence attends to the first seqlens[b] rows of its cache.

    q [batch, num_q_heads, d]; k, v [batch, cache_len, num_kv_heads, d]; seqlens int32 [batch].
    """
    return _lib.host().flash_attention_decode(q, k, v, seqlens, sm_scale)


def topk_sparse_attention_decode(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, topk_idx: torch.Tensor,
                                 block_size: int, seqlens: torch.Tensor, sm_scale: Optional[float] = None) -> torch.Tensor:
    """One query token per sequence attends to the rows of its selected blocks below seqlens[b].

    topk_idx int32 [num_kv_heads, batch, topk], -1 padding.
    """
    return _lib.host().topk_sparse_attention_decode(q, k, v, topk_idx, int(block_size), seqlens, sm_scale)


def compressed_attention_decode(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, seqlens: torch.Tensor,
                                compress_seqlens: torch.Tensor, kernel_size: int, kernel_stride: int, block_size: int,
                                topk: int, init_blocks: int = 1, local_blocks: int = 2,
                                sm_scale: Optional[float] = None, max_seqlen: Optional[int] = None) -> Tuple[torch.Tensor, torch.Tensor]:
    """Single-token attention over the compressed cache and block selection for the current token.

    seqlens counts the current token; compress_seqlens is the number of valid compressed rows.
    Returns (o [batch, num_q_heads, d], topk_idx int32 [num_kv_heads, batch, min(topk, num_blocks)]).
    num_blocks = ceil(max(seqlens) / block_size) as in the reference, which costs a device-to-host copy; a caller that must
    not synchronise passes max_seqlen (an upper bound, e.g. the cache capacity): the width of topk_idx then follows the
    bound and the entries beyond a sequence's blocks are -1.
    """
    return _lib.host().compressed_attention_decode(q, k, v, seqlens, compress_seqlens, kernel_size, kernel_stride, block_size, topk,
                                                   init_blocks, local_blocks, sm_scale, max_seqlen)
