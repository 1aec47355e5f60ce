"""Backward of the selected-block attention with output gradients of other strides, down to an expanded gradient's strides of 0: a
token's rows come as TMA boxes.  Gradients against autograd over the fp32 oracle, for every group size of the tcgen05 pass, lists
of one token, of a row tile and one more, and longer than a work item; one KV head's items are one CTA's, many or few."""
import pytest
import torch

from oracle import nsa_oracle as O
from tests.helpers import MEAN_TOL, assert_close_16bit, grad_tol

pytestmark = pytest.mark.gpu


def gradient(kind, N, Hq, d, g, dtype):
    if kind == "expanded tokens":
        return torch.randn(1, Hq, d, generator=g).to(dtype).cuda().expand(N, Hq, d)
    if kind == "expanded":
        return torch.randn(d, generator=g).to(dtype).cuda().expand(N, Hq, d)
    if kind == "padded rows":
        return torch.randn(N, Hq + 1, d + 8, generator=g).to(dtype).cuda()[:, 1:, :d]
    return torch.randn(Hq, N, d, generator=g).to(dtype).cuda().transpose(0, 1)  # heads outermost


@pytest.mark.parametrize("kind", ["expanded tokens", "expanded", "padded rows", "heads outermost"])
@pytest.mark.parametrize("G,d,lens,topk,dtype", [
    (16, 128, [1, 65, 700], 4, torch.bfloat16),
    (16, 64, [9, 300], 3, torch.float16),
    (8, 128, [577, 17], 5, torch.float16),
    (8, 64, [400], 4, torch.bfloat16),
    (4, 128, [33, 600], 6, torch.bfloat16),
    (4, 64, [200, 128, 1], 2, torch.float16),
])
def test_gradient_strides(G, d, lens, topk, dtype, kind):
    import native_sparse_attention_triton_b200 as pkg
    Hkv, bs, N = 2, 64, sum(lens)
    g = torch.Generator().manual_seed(G + d)
    host = [torch.randn(N, h, d, generator=g).to(dtype) for h in (G * Hkv, Hkv, Hkv)]
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
    idx = torch.full((Hkv, N, topk), -1, dtype=torch.int32)
    at = 0
    for n in lens:
        for t in range(n):
            for h in range(Hkv):
                # every token takes block 0: its list is the longest there can be
                rest = torch.randperm(t // bs, generator=g)
                ids = torch.cat([torch.zeros(1, dtype=torch.long), torch.tensor([t // bs]), rest]).unique(sorted=False)[:topk].sort().values
                idx[h, at + t, :len(ids)] = ids.int()
        at += n
    do = gradient(kind, N, G * Hkv, d, g, dtype)
    dev = [t.cuda().requires_grad_(True) for t in host]
    ref = [t.float().requires_grad_(True) for t in host]
    pkg.ops.topk_sparse_attention(*dev, idx.cuda(), bs, cu.cuda()).backward(do)
    O.topk_sparse_attention(*ref, idx, bs, cu).backward(do.float().cpu())
    for name, a, b in zip(("dq", "dk", "dv"), dev, ref):
        assert_close_16bit(a.grad, b.grad, name, grad_tol(name, False), MEAN_TOL)
    assert pkg.device_status() == 0
