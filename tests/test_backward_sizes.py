"""Scratch sizes of the backward passes, and the division of work that they are made for."""
import pytest

from native_sparse_attention_triton_b200 import _lib


def align_up(n):
    return (n + 255) // 256 * 256


def item_entries(N, batch, Hq, Hkv, d, topk, block_size):
    """Entries of the table of work items: what nsa_topk_sparse_attn_bwd_workspace asks for beside the other buffers."""
    G = Hq // Hkv
    fused = G >= 4 and G & (G - 1) == 0
    per_token = 4 * G * d + (4 * G * d if fused else 0)
    window = 1024
    while 2 * window * per_token <= 64 << 20:
        window *= 2
    bins = Hkv * -(-N // window) * (N // block_size + batch) + 1
    others = align_up(N * Hq * 8) + 2 * align_up(N * Hkv * d * 4) + 4 * align_up(bins * 4) + align_up(Hkv * N * topk * 4)
    others += align_up(N * Hq * d * 4) if fused else 0
    size = _lib.lib().nsa_topk_sparse_attn_bwd_workspace(N, batch, Hq, Hkv, d, topk, block_size)
    return (size - others) // 4, bins


@pytest.mark.parametrize("N,Hq,Hkv,topk,chunk", [
    (977, 24, 2, 8, 64), (6000, 20, 2, 16, 256), (3000, 9, 1, 12, 64), (16384, 48, 4, 16, 512), (3000, 15, 1, 12, 64),  # mma.sync pass
    (4096, 12, 4, 16, 256), (977, 4, 2, 8, 64),
    (977, 32, 2, 8, 32), (16384, 64, 4, 16, 256), (7097, 32, 8, 16, 512), (2000, 16, 1, 16, 64), (65536, 16, 2, 16, 512),  # tcgen05 pass
])
def test_tokens_of_a_work_item(N, Hq, Hkv, topk, chunk):
    entries, bins = item_entries(N, 1, Hq, Hkv, 128, topk, 64)
    assert entries == align_up((Hkv * N * topk // chunk + bins) * 4) // 4
