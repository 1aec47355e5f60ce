"""The two kernels of the selected-block forward divide the tokens of a sequence by their position (unions of neighbouring tokens'
selections before it, private walks behind it): outputs at the edges of row tiles, blocks, sequences and of that division, against
the fp32 oracle."""
import pytest
import torch

from oracle import nsa_oracle as O

pytestmark = pytest.mark.gpu


def selection(g, lens, hkv, bs, topk):
    """First block, own block and its predecessor, the rest at random; a few tokens without any and one with only its own block."""
    out = torch.full((hkv, sum(lens), topk), -1, dtype=torch.int32)
    at = 0
    for n in lens:
        for t in range(n):
            own = t // bs
            for h in range(hkv):
                pool = torch.randperm(own + 1, generator=g)[:topk].tolist()
                ids = sorted(set([0, max(own - 1, 0), own] + pool))
                ids = ids[:topk - 1] + [own] if len(ids) > topk else ids
                ids = sorted(set(ids))
                if t % 97 == 13:
                    ids = []
                elif t % 97 == 14:
                    ids = [own]
                out[h, at + t, :len(ids)] = torch.tensor(ids, dtype=torch.int32)
        at += n
    return out


@pytest.mark.parametrize("Hq,Hkv,d,bs,topk,lens,dtype", [
    (16, 1, 128, 64, 4, [1, 17, 129, 200], torch.bfloat16),
    (8, 2, 64, 64, 3, [300, 64, 63], torch.float16),
    (4, 1, 128, 128, 3, [385, 65], torch.bfloat16),
    (2, 1, 128, 64, 5, [513], torch.float16),
    (3, 3, 64, 64, 4, [257, 31], torch.bfloat16),      # groups of one: a row tile is 128 tokens
    (6, 2, 128, 64, 4, [150], torch.bfloat16),         # a group that is no power of two: private walks only
    (16, 1, 64, 64, 4, [2600], torch.bfloat16),        # crosses the division (head_dim 64, top-4)
])
def test_sparse_forward_positions(Hq, Hkv, d, bs, topk, lens, dtype):
    import native_sparse_attention_triton_b200 as pkg
    g = torch.Generator().manual_seed(sum(lens) + Hq)
    N = sum(lens)
    rnd = lambda h: torch.randn(N, h, d, generator=g).to(dtype)
    q, k, v = rnd(Hq), rnd(Hkv), rnd(Hkv)
    idx = selection(g, lens, Hkv, bs, topk)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
    o = pkg.ops.topk_sparse_attention(q.cuda(), k.cuda(), v.cuda(), idx.cuda(), bs, cu.cuda())
    ref = O.topk_sparse_attention(q.float(), k.float(), v.float(), idx, bs, cu)
    err = (o.float().cpu() - ref).abs() / ref.abs().clamp(min=1.0)
    # P and the result are rounded to 16 bits once each; |o| <= max |v|
    assert float(err.max()) <= 2e-2 and float(err.mean()) <= 2e-3, (float(err.max()), float(err.mean()))
    assert pkg.device_status() == 0


def test_lengths_remembered_on_the_host_choose_nothing_but_speed():
    """cu_seqlens that were written to behind the version counter after the host has seen them (as a graph replay does): the same
    rows as three short sequences first, then as one that crosses the division."""
    import native_sparse_attention_triton_b200 as pkg
    Hq, Hkv, d, bs, topk, N = 16, 1, 64, 64, 4, 2600
    g = torch.Generator().manual_seed(7)
    rnd = lambda h: torch.randn(N, h, d, generator=g).bfloat16()
    q, k, v = rnd(Hq), rnd(Hkv), rnd(Hkv)
    cu = torch.tensor([0, 900, 1800, N], dtype=torch.int32).cuda()
    pkg.ops.avgpool_compress(k.cuda(), None, cu, 32, 16, None)
    one = torch.tensor([0, N, N, N], dtype=torch.int32)
    cu.data.copy_(one)
    idx = selection(g, [N], Hkv, bs, topk)
    o = pkg.ops.topk_sparse_attention(q.cuda(), k.cuda(), v.cuda(), idx.cuda(), bs, cu)
    ref = O.topk_sparse_attention(q.float(), k.float(), v.float(), idx, bs, torch.tensor([0, N], dtype=torch.int32))
    err = (o.float().cpu() - ref).abs() / ref.abs().clamp(min=1.0)
    assert float(err.max()) <= 2e-2 and float(err.mean()) <= 2e-3, (float(err.max()), float(err.mean()))


@pytest.mark.parametrize("where,value", [("v", float("inf")), ("k", float("-inf")), ("k", float("nan"))])
def test_non_finite_rows_stay_with_those_who_selected_them(where, value):
    """One key or value row of block 3 that is not finite: tokens whose selection leaves that block out get what they get without it."""
    import native_sparse_attention_triton_b200 as pkg
    Hq, Hkv, d, bs, topk, lens = 8, 2, 128, 64, 4, [700, 450]
    g = torch.Generator().manual_seed(3)
    N = sum(lens)
    rnd = lambda h: torch.randn(N, h, d, generator=g).bfloat16().cuda()
    q, k, v = rnd(Hq), rnd(Hkv), rnd(Hkv)
    idx = selection(g, lens, Hkv, bs, topk)
    cu = torch.tensor([0, lens[0], N], dtype=torch.int32).cuda()
    run = lambda: pkg.ops.topk_sparse_attention(q, k, v, idx.cuda(), bs, cu).float().cpu()
    clean = run()
    (v if where == "v" else k)[3 * bs + 5, 0, 7] = value
    o = run()
    hit = (idx == 3).any(-1)
    hit[:, lens[0]:] = False      # block 3 of the second sequence is another one
    hit[1] = False                # the row belongs to the first KV head
    away = ~hit.repeat_interleave(Hq // Hkv, 0).T
    err = (o - clean).abs()[away] / clean.abs().clamp(min=1.0)[away]
    assert float(err.max()) <= 2e-2, float(err.max())
    seen = hit.clone()
    seen[:, :3 * bs + 64] = False  # in the row's own block the causal mask decides
    assert int(seen.sum()) > 50
    if value != float("-inf"):
        assert not torch.isfinite(o[seen.repeat_interleave(Hq // Hkv, 0).T]).all()
