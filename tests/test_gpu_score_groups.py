"""Block selection on the tcgen05 score pass for groups of eight query heads."""
import pytest
import torch

from native_sparse_attention_triton_b200 import device_status, ops

pytestmark = pytest.mark.gpu


def _cu(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return cu


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("lens", [[15, 16, 17, 31, 33], [700, 4000]])
def test_scores_of_groups_of_eight(d, lens):
    """Selection with eight query heads per KV head (16 tokens in a row tile, three folds per thread) against float64 scores."""
    from oracle import nsa_oracle as oracle

    g = torch.Generator(device="cuda").manual_seed(d)
    cq, windows = _cu(lens), [max(0, (n - 32) // 16 + 1) for n in lens]
    ck = _cu(windows)
    q = torch.randn(cq[-1], 16, d, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(ck[-1], 2, d, generator=g, device="cuda").bfloat16() for _ in range(2))
    cu_q, cu_k = (torch.tensor(c, dtype=torch.int32, device="cuda") for c in (cq, ck))
    _, idx = ops.compressed_attention(q, k, v, 32, 16, 64, 8, cu_q, cu_k, max(lens), max(windows), None, 1, 2)
    _, want, scores = oracle.compressed_attention(q.float().cpu(), k.float().cpu(), v.float().cpu(), 32, 16, 64, 8, cu_q.cpu(), cu_k.cpu(),
                                                  max(lens), max(windows), None, 1, 2, return_scores=True)
    bad, _, _ = oracle.compare_topk_idx(idx.cpu(), want, scores, tie_tol=1e-3)
    assert bad == 0
    assert device_status() == 0
