"""dK/dV passes at head_dim 64 on the tensor-core kernels, which stack two operands to fill a 128-row product: gradients against
autograd over the fp32 oracle at the edges of row tiles, key tiles, blocks of two tiles and groups of 4, 8 and 16 (and, dense, 1)."""
import pytest
import torch

from oracle import nsa_oracle as O
from tests.helpers import MEAN_TOL, assert_close_16bit, grad_tol

pytestmark = pytest.mark.gpu


def leaves(seed, lens, Hq, Hkv, d, dtype):
    g = torch.Generator().manual_seed(seed)
    N = sum(lens)
    host = [torch.randn(N, h, d, generator=g).to(dtype) for h in (Hq, Hkv, Hkv, Hq)]
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
    dev = [t.cuda().requires_grad_(True) for t in host[:3]]
    ref = [t.float().requires_grad_(True) for t in host[:3]]
    return cu, dev, ref, host[3]


def check(dev, ref):
    import native_sparse_attention_triton_b200 as pkg
    for name, a, b in zip(("dq", "dk", "dv"), dev, ref):
        assert_close_16bit(a.grad, b.grad, name, grad_tol(name, False), MEAN_TOL)
    assert pkg.device_status() == 0


@pytest.mark.parametrize("Hq,Hkv,bs,topk,lens,dtype", [
    (16, 1, 64, 4, [1, 8, 65], torch.bfloat16),        # 8 tokens per row tile
    (16, 2, 64, 5, [129, 500], torch.float16),         # 16
    (8, 2, 128, 3, [385, 33], torch.bfloat16),         # 32; two key tiles per block
    (16, 1, 64, 16, [1700], torch.bfloat16),           # lists longer than a work item, several items per CTA
    (4, 2, 64, 4, [200], torch.bfloat16),              # groups of two: the kernel of mma.sync warps
])
def test_selected_blocks(Hq, Hkv, bs, topk, lens, dtype):
    import native_sparse_attention_triton_b200 as pkg
    cu, dev, ref, do = leaves(Hq + topk, lens, Hq, Hkv, 64, dtype)
    g = torch.Generator().manual_seed(2)
    idx = torch.full((Hkv, sum(lens), topk), -1, dtype=torch.int32)
    at = 0
    for n in lens:
        for t in range(n):
            for h in range(Hkv):
                ids = torch.cat([torch.tensor([t // bs]), torch.randperm(t // bs, generator=g)])[:topk].sort().values
                idx[h, at + t, :len(ids)] = ids.int()
        at += n
    pkg.ops.topk_sparse_attention(*dev, idx.cuda(), bs, cu.cuda()).backward(do.cuda())
    O.topk_sparse_attention(*ref, idx, bs, cu).backward(do.float())
    check(dev, ref)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("Hq,Hkv,lens,dtype", [
    (16, 1, [1, 7, 130], torch.bfloat16),
    (8, 8, [129, 300], torch.float16),                 # groups of one: 128 tokens per row tile
    (16, 2, [777], torch.bfloat16),
])
def test_dense(Hq, Hkv, lens, dtype, causal):
    import native_sparse_attention_triton_b200 as pkg
    cu, dev, ref, do = leaves(Hq + sum(lens), lens, Hq, Hkv, 64, dtype)
    pkg.ops.flash_attention_varlen(*dev, cu.cuda(), cu.cuda(), max(lens), max(lens), causal).backward(do.cuda())
    O.flash_attention_varlen(*ref, cu, cu, causal=causal).backward(do.float())
    check(dev, ref)


@pytest.mark.parametrize("d", [64, 128])
def test_gradient_at_an_odd_offset(d):
    """A contiguous view whose address is no multiple of 16 bytes gives what its copy gives (up to the order of atomic sums)."""
    import native_sparse_attention_triton_b200 as pkg
    N, Hq, Hkv, bs = 300, 8, 2, 64
    g = torch.Generator().manual_seed(4)
    q, k, v = [torch.randn(N, h, d, generator=g).bfloat16().cuda().requires_grad_(True) for h in (Hq, Hkv, Hkv)]
    cu = torch.tensor([0, N], dtype=torch.int32).cuda()
    t = torch.arange(N)
    idx = torch.stack([torch.zeros(N, dtype=torch.int64), torch.where(t < bs, -1, t // bs)], 1).int()[None].expand(Hkv, N, 2).contiguous().cuda()
    odd = torch.randn(N * Hq * d + 1, generator=g).bfloat16().cuda()[1:].view(N, Hq, d)
    assert odd.data_ptr() % 16 and odd.is_contiguous()
    for o in (pkg.ops.topk_sparse_attention(q, k, v, idx, bs, cu), pkg.ops.flash_attention_varlen(q, k, v, cu, cu, N, N, causal=True)):
        for a, b in zip(torch.autograd.grad(o, (q, k, v), odd, retain_graph=True), torch.autograd.grad(o, (q, k, v), odd.clone())):
            assert float((a.float() - b.float()).norm()) <= 1e-3 * float(b.float().norm())
    assert pkg.device_status() == 0
