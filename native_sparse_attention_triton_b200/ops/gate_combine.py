"""Gated sum of the three branch outputs of an NSA layer (compressed, selected, sliding-window).

The reference has no operator for this step: its layer evaluates
    gate[..., 0:1] * compressed_attn_output + gate[..., 1:2] * sparse_attn_output + gate[..., 2:3] * sliding_attn_output
in eager PyTorch (native_sparse_attention/module/native_sparse_attention.py:226-232; the inference path does the same at
native_sparse_attention/infer/nsa_inference.py:146-150).  This function computes the same expression, forward and
backward, in one pass over HBM each, with fp32 arithmetic and a single rounding.
"""
import torch

from .. import _lib


def gate_combine(gate: torch.Tensor, o_cmp: torch.Tensor, o_sel: torch.Tensor, o_win: torch.Tensor) -> torch.Tensor:
    """gate [n, h, 3] (already through the sigmoid), o_* [n, h, d] -> [n, h, d] contiguous, so that the head concat that
    feeds the output projection is a view.  d is 64 or 128; 16-bit inputs of one dtype."""
    return _lib.host().gate_combine(gate, o_cmp, o_sel, o_win)
