"""Rotary position embedding of a varlen batch in one kernel (forward and backward).

Mirrors ``RotaryEmbedding.forward(x, cu_seqlens, step=0, stride=1)`` of the reference
(native_sparse_attention/module/rope.py:197-209): ``x * cos + rotate_half(x) * sin`` with the position of every row
derived from ``cu_seqlens`` -- token t of its sequence at ``t * stride`` when ``step == 0``, row b of a decode step at
``(seqlen_b + step - 1) * stride`` otherwise (:158-195).  The frequencies stay the caller's: ``inv_freq`` and
``attention_scaling`` are what the reference obtains from ``ROPE_INIT_FUNCTIONS`` (:88-90); the cos/sin values are
computed from them on the fly (fp32 angle, rounded to the tensor's dtype as the reference's cached tables are), so there
is no table, no Python loop over the batch and no host synchronisation.
"""
import torch

from .. import _lib


def rope(x: torch.Tensor, inv_freq: torch.Tensor, cu_seqlens: torch.Tensor, step: int = 0, stride: int = 1,
         attention_scaling: float = 1.0) -> torch.Tensor:
    """x [rows, heads, d] (d 64 or 128, bf16/fp16), inv_freq fp32 [d / 2], cu_seqlens int32 [batch + 1] -> rotated copy.
    With step > 0, rows == batch (one new token per sequence) and cu_seqlens holds the PREFILL lengths, as in the
    reference's decode loop."""
    return _lib.host().rope(x, inv_freq, cu_seqlens, int(step), int(stride), attention_scaling)
