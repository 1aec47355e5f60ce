"""Attention between queries and compressed keys/values, plus top-k block selection.

Signature and semantics follow native_sparse_attention/ops/triton/compressed_attention.py:1182-1331
of the reference.  The block scores are never materialised: one kernel recomputes QK^T against the
final log-sum-exp, reduces over the query heads of each KV group and selects in shared memory.
"""
import warnings
from typing import Tuple, Union

import torch

from .. import _lib


def compressed_attention(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    kernel_size: int,
    kernel_stride: int,
    block_size: int,
    topk: int,
    cu_seqlens_q: torch.Tensor,
    cu_seqlens_k: torch.Tensor,
    max_seqlen_q: int = None,
    max_seqlen_k: int = None,
    sm_scale: float = None,
    init_blocks: int = 1,
    local_blocks: int = 2,
    parallel_topk_compute: Union[str, bool] = "auto",
) -> Tuple[torch.Tensor, torch.Tensor]:
    """Attention output over compressed K/V and the block ids each query keeps for sparse attention.

    Args:
        q: [total_q_len, num_q_heads, head_dim]
        k, v: [total_kv_len, num_kv_heads, head_dim] (compressed)
        kernel_size, kernel_stride: the compression window and hop that produced k, v
        block_size: selection block size of topk_sparse_attention
        topk: blocks kept per query (<= 0: no selection, topk_idx is None)
        cu_seqlens_q, cu_seqlens_k: int32 [batch + 1]
        max_seqlen_q, max_seqlen_k: optional maxima (computed with one host sync when None)
        sm_scale: softmax scale, default 1/sqrt(head_dim)
        init_blocks, local_blocks: always-selected leading blocks / trailing blocks ending at the query's own
        parallel_topk_compute: accepted for compatibility; selection never materialises scores here
    Returns:
        (attention output like q, topk_idx int32 [num_kv_heads, total_q_len, min(topk, num_blocks)])
    """
    if topk <= 0:
        warnings.warn("topk <= 0, returned topk_idx will be None")
    max_seqlen_q, max_seqlen_k = (None if m is None else int(m) for m in (max_seqlen_q, max_seqlen_k))
    return _lib.host().compressed_attention(q, k, v, kernel_size, kernel_stride, block_size, topk, cu_seqlens_q, cu_seqlens_k,
                                            max_seqlen_q, max_seqlen_k, sm_scale, init_blocks, local_blocks)
