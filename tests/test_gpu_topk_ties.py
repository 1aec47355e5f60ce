"""Block selection by a bitwise threshold (up to 256 candidate blocks): ties, which zero queries make of every interior block; candidate
counts on both sides of 32, 64, 128 and 256; scores on both sides of 2; widths from one free choice to more than there are blocks."""
import pytest
import torch

from oracle import nsa_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,topk", [(1, 4), (4, 16), (1, 33)])
@pytest.mark.parametrize("n", [33 * 64, 65 * 64 + 1, 130 * 64 - 5, 258 * 64])
def test_selection(n, Hq, topk):
    import native_sparse_attention_triton_b200 as pkg
    ks, st, bs, d = 16, 16, 64, 64
    if n > 130 * 64 and Hq > 1:
        pytest.skip("the oracle's score matrix for one head is enough at this length")
    g = torch.Generator().manual_seed(n + topk)
    m = (n - ks) // st + 1
    q, k, v = [torch.randn(r, h, d, generator=g).half() for r, h in ((n, Hq), (m, 1), (m, 1))]
    q[::7] = 0
    q[3::7] *= 6      # nearly all of a row's mass on one block
    cu, cu_k = torch.tensor([0, n], dtype=torch.int32), torch.tensor([0, m], dtype=torch.int32)
    _, idx = pkg.ops.compressed_attention(q.cuda(), k.cuda(), v.cuda(), ks, st, bs, topk, cu.cuda(), cu_k.cuda(), n, m)
    _, ref, scores = O.compressed_attention(q.float(), k.float(), v.float(), ks, st, bs, topk, cu, cu_k, return_scores=True)
    idx = idx.cpu()
    bad, differing, rows = O.compare_topk_idx(idx, ref, scores, tie_tol=1e-3)
    assert bad == 0, (bad, differing, rows)
    assert torch.equal(idx >= 0, ref >= 0)
    a = torch.where(idx >= 0, idx, torch.arange(idx.shape[-1]).int() + 100000)
    assert bool((a[..., 1:] > a[..., :-1]).all())   # ascending, -1 last
    assert pkg.device_status() == 0
