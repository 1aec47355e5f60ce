"""Lengths and sizes may be whole numbers of any type: floats (a maximum taken over a float array), numpy scalars, 0-dim tensors.  No
GPU: an accepted call gets as far as the refusal of CPU tensors."""
import numpy as np
import pytest
import torch

from native_sparse_attention_triton_b200 import ops

WHOLE = [int, float, np.int64, np.float32, torch.tensor, lambda x: torch.tensor(float(x))]


@pytest.mark.parametrize("kind", range(len(WHOLE)))
def test_whole_numbers_of_any_type(kind):
    n = WHOLE[kind]
    q, k, cu = torch.zeros(70, 4, 128).bfloat16(), torch.zeros(70, 2, 128).bfloat16(), torch.tensor([0, 70], dtype=torch.int32)
    cu_k, idx = torch.tensor([0, 3], dtype=torch.int32), torch.zeros(2, 70, 1, dtype=torch.int32)
    one = torch.tensor([70], dtype=torch.int32)
    calls = [
        lambda: ops.compressed_attention(q, k[:3], k[:3], 32, 16, 64, 4, cu, cu_k, n(70), n(3)),
        lambda: ops.flash_attention_varlen(q, k, k, cu, cu, n(70), n(70), n(1), 0.1),
        lambda: ops.sliding_window_attention(q, k, k, cu, n(70), n(64)),
        lambda: ops.rope(q, torch.ones(64), cu, n(0), n(1)),
        lambda: ops.topk_sparse_attention(q, k, k, idx, n(64), cu),
        lambda: ops.topk_sparse_attention_decode(q[:1], k[None], k[None], idx[:, :1], n(64), one),
    ]
    for call in calls:
        with pytest.raises(RuntimeError, match="CUDA tensors only"):
            call()


def test_block_sizes_that_are_none():
    q, k = torch.zeros(70, 4, 128).bfloat16(), torch.zeros(70, 2, 128).bfloat16()
    for bs in (16, 64.5, 100, 512):
        with pytest.raises(AssertionError):
            ops.topk_sparse_attention(q, k, k, torch.zeros(2, 70, 1, dtype=torch.int32), bs, torch.tensor([0, 70], dtype=torch.int32))
