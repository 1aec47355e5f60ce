"""Key/value compression operators: linear projection, weighted pooling, average pooling.

Signatures, argument meaning and assertion behaviour follow the reference's
native_sparse_attention/ops/triton/linear_compress.py:497-525 and
native_sparse_attention/ops/triton/weighted_pool.py:301-363.  Unlike the reference the
position-embedding bias is folded into the kernel epilogue and its gradient is produced by the same
backward pass.  The lengths of a cu_seqlens tensor are read on the host once per tensor and version.
"""
from typing import Optional, Tuple

import torch

from .. import _lib

_LINEAR, _WEIGHTED, _AVERAGE = 0, 1, 2


def linear_compress(x: torch.Tensor, w: torch.Tensor, cu_seqlens: torch.Tensor, kernel_size: int, kernel_stride: int,
                    pe: Optional[torch.Tensor] = None) -> Tuple[torch.Tensor, torch.Tensor]:
    """Compress keys/values with a per-head linear projection of each window.

    Args:
        x: [total_len, num_heads, head_dim]
        w: [num_heads, kernel_size * head_dim, head_dim]
        cu_seqlens: int32 [batch + 1]
        kernel_size / kernel_stride: window length and hop
        pe: optional intra-block position embedding [num_heads, kernel_size, head_dim]
    Returns:
        (compressed [total_compressed, num_heads, head_dim], y_cu_seqlens int32 [batch + 1])
    """
    return _lib.host().compress(x, w, cu_seqlens, kernel_size, kernel_stride, pe, _LINEAR)


def weightedpool_compress(x: torch.Tensor, w: torch.Tensor, cu_seqlens: torch.Tensor, kernel_size: int,
                          kernel_stride: int, pe: Optional[torch.Tensor] = None):
    """Compress keys/values with a per-head weighted sum over each window; w is [num_heads, kernel_size]."""
    return _lib.host().compress(x, w, cu_seqlens, kernel_size, kernel_stride, pe, _WEIGHTED)


def avgpool_compress(x: torch.Tensor, w, cu_seqlens: torch.Tensor, kernel_size: int, kernel_stride: int,
                     pe: Optional[torch.Tensor] = None):
    """Compress keys/values with the mean of each window; w must be None."""
    assert w is None, "don't need additional weight for avgpool"
    return _lib.host().compress(x, None, cu_seqlens, kernel_size, kernel_stride, pe, _AVERAGE)
