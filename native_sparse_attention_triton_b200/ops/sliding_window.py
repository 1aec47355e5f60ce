"""Sliding-window branch of the NSA layer: causal varlen GQA attention where query t sees keys t - window_size .. t.

The reference has no operator of its own for this branch: its layer calls the third-party
flash_attn.flash_attn_varlen_func(..., causal=True, window_size=(window_size, -1))
(native_sparse_attention/module/native_sparse_attention.py:213-223), which this function replaces with the same
tcgen05 kernels as flash_attention_varlen plus a lower bound on the visible keys.  head_dim 128 only.
"""
from typing import Optional

import torch

from .. import _lib


def sliding_window_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, cu_seqlens: torch.Tensor, max_seqlen: int,
                             window_size: int, sm_scale: Optional[float] = None) -> torch.Tensor:
    """q [total, Hq, d], k/v [total, Hkv, d] (self-attention: one cu_seqlens); key j is visible to query i of the same
    sequence iff i - window_size <= j <= i, i.e. window_size + 1 keys, as flash_attn's window_size=(window_size, -1) with
    causal=True gives."""
    return _lib.host().sliding_window_attention(q, k, v, cu_seqlens, int(max_seqlen), int(window_size), sm_scale)
