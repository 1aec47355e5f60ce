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


def private_walk(q, k, v, idx, bs, lens):
    """The walk of sparse_fwd.cu, one (token, KV head) pair at a time in fp32 torch: 64 keys per step in the order of the selection, the
    running maximum as reference, probabilities rounded to 16 bits before the product with V, the sum of the unrounded ones."""
    N, Hq, d = q.shape
    Hkv = k.shape[1]
    G, T = Hq // Hkv, idx.shape[-1]
    out, at = torch.zeros_like(q), 0
    for n in lens:
        pos = torch.arange(n, device=q.device)
        for h in range(Hkv):
            qf, kf, vf = q[at:at + n, h * G:(h + 1) * G].float(), k[at:at + n, h].float(), v[at:at + n, h].float()
            m = torch.full((n, G), -float("inf"), device=q.device)
            l, o = torch.zeros(n, G, device=q.device), torch.zeros(n, G, d, device=q.device)
            for j in range(T):
                for half in range(bs // 64):
                    key = idx[h, at:at + n, j].long()[:, None] * bs + half * 64 + torch.arange(64, device=q.device)
                    seen = (idx[h, at:at + n, j] >= 0)[:, None] & (key <= pos[:, None])
                    key = key.clamp(0, n - 1)
                    s = torch.einsum("ngd,nkd->ngk", qf, kf[key]) * (d ** -0.5 * 1.4426950408889634)
                    s = s.masked_fill(~seen[:, None], -float("inf"))
                    mn = torch.maximum(m, s.amax(-1))
                    ref = torch.where(mn == -float("inf"), torch.zeros_like(mn), mn)
                    p, c = torch.exp2(s - ref[..., None]), torch.exp2(m - ref)
                    l, o, m = l * c + p.sum(-1), o * c[..., None] + torch.einsum("ngk,nkd->ngd", p.to(q.dtype).float(), vf[key]), mn
            out[at:at + n, h * G:(h + 1) * G] = torch.where(l[..., None] > 0, o / l[..., None], torch.zeros_like(o)).to(q.dtype)
        at += n
    return out


@pytest.mark.parametrize("Hq,Hkv,d,topk,lens,dtype", [
    (8, 2, 128, 8, [900, 700], torch.bfloat16),
    (8, 2, 128, 8, [900, 700], torch.float16),
    (16, 1, 64, 6, [1500], torch.bfloat16),
])
def test_unions_are_no_less_exact_than_private_walks(Hq, Hkv, d, topk, lens, dtype):
    """Error of the output against 64 bits beside that of the private walk, and of the lse, which the backward reads."""
    import native_sparse_attention_triton_b200 as pkg
    from native_sparse_attention_triton_b200 import _lib
    g = torch.Generator().manual_seed(11)
    N, bs, G = sum(lens), 64, Hq // Hkv
    rnd = lambda h: torch.randn(N, h, d, generator=g).to(dtype).cuda()
    q, k, v = rnd(Hq), rnd(Hkv), rnd(Hkv)
    idx = selection(g, lens, Hkv, bs, topk).cuda()
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32).cuda()
    o, lse = torch.empty_like(q), torch.empty(N, Hq, device="cuda")
    strides = _lib.strides_array(*[x for t in (q, k, v, o) for x in t.stride()[:2]], *idx.stride())
    rc = _lib.lib().nsa_topk_sparse_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), idx.data_ptr(), cu.data_ptr(), o.data_ptr(),
                                             lse.data_ptr(), N, len(lens), Hq, Hkv, d, topk, bs, strides, d ** -0.5,
                                             _lib.DTYPE_BF16 if dtype == torch.bfloat16 else _lib.DTYPE_FP16,
                                             torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    exact, exact_lse = torch.zeros(N, Hq, d, device="cuda", dtype=torch.float64), torch.zeros(N, Hq, device="cuda", dtype=torch.float64)
    at = 0
    for n in lens:
        nb = (n + bs - 1) // bs
        for h in range(Hkv):
            ids = idx[h, at:at + n].long()
            took = torch.zeros(n, nb + 1, dtype=torch.bool, device="cuda").scatter_(1, torch.where(ids < 0, nb, ids), True)
            mask = took[:, :nb].repeat_interleave(bs, 1)[:, :n] & torch.ones(n, n, dtype=torch.bool, device="cuda").tril()
            s = torch.einsum("ngd,md->ngm", q[at:at + n, h * G:(h + 1) * G].double(), k[at:at + n, h].double()) * d ** -0.5
            s = s.masked_fill(~mask[:, None], -float("inf"))
            exact[at:at + n, h * G:(h + 1) * G] = s.softmax(-1).nan_to_num(0.0) @ v[at:at + n, h].double()
            exact_lse[at:at + n, h * G:(h + 1) * G] = torch.logsumexp(s, -1) * 1.4426950408889634
        at += n
    rel = lambda x: float((x.double() - exact).norm() / exact.norm())
    # the same roundings of other sums: over a million outputs the two norms agree to a few parts in ten thousand
    assert rel(o) <= 1.002 * rel(private_walk(q, k, v, idx, bs, lens)), (rel(o), rel(private_walk(q, k, v, idx, bs, lens)))
    seen = torch.isfinite(exact_lse)
    assert torch.equal(seen, torch.isfinite(lse))
    # fp32: logits of magnitude 8 to 2^-21, exponentials of the unit to 2^-22, a sum of up to 512 terms
    worst = float((lse.double() - exact_lse)[seen].abs().max())
    assert worst <= 6e-6, worst
    assert pkg.device_status() == 0


@pytest.mark.parametrize("Hq,Hkv,d,topk,lens,dtype", [
    (8, 2, 128, 5, [300, 200], torch.bfloat16),
    (3, 3, 64, 4, [257], torch.float16),        # groups of one: 256 tokens per CTA
    (16, 1, 64, 4, [2600], torch.bfloat16),     # crosses the division
])
def test_blocks_given_twice_count_twice(Hq, Hkv, d, topk, lens, dtype):
    """Some tokens give a block two or three times: output and gradients against attention whose logits carry the logarithm of the
    number of times, and the single-token operator on the last token's row."""
    import native_sparse_attention_triton_b200 as pkg
    g = torch.Generator().manual_seed(23)
    N, bs, G = sum(lens), 64, Hq // Hkv
    rnd = lambda h: torch.randn(N, h, d, generator=g).to(dtype).cuda()
    q, k, v, do = rnd(Hq), rnd(Hkv), rnd(Hkv), rnd(Hq)
    idx = selection(g, lens, Hkv, bs, topk)
    for t in range(N):
        if t % 3 == 0 or t == N - 1:
            for h in range(Hkv):
                ids = [x for x in idx[h, t].tolist() if x >= 0]
                ids = (ids + ids[-1:] * (1 + t % 2) + ids)[:topk]
                idx[h, t] = torch.tensor(ids + [-1] * (topk - len(ids)), dtype=torch.int32)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32).cuda()
    a = [x.clone().requires_grad_(True) for x in (q, k, v)]
    o = pkg.ops.topk_sparse_attention(*a, idx.cuda(), bs, cu)
    grads = torch.autograd.grad(o, a, do)
    b = [x.double().requires_grad_(True) for x in (q, k, v)]
    outs, at = [], 0
    for n in lens:
        nb = (n + bs - 1) // bs
        ids = idx[:, at:at + n].long().cuda()
        times = torch.zeros(Hkv, n, nb + 1, device="cuda").scatter_add_(2, torch.where(ids < 0, nb, ids), torch.ones(ids.shape, device="cuda"))
        times = times[..., :nb].repeat_interleave(bs, 2)[..., :n] * torch.ones(n, n, device="cuda").tril()
        s = torch.einsum("nhgd,mhd->hgnm", b[0][at:at + n].view(n, Hkv, G, d), b[1][at:at + n]) * d ** -0.5
        s = s + times.double().log()[:, None]
        empty = (times.sum(-1) == 0)[:, None, :, None]
        p = torch.where(empty, 0.0, s.masked_fill(empty, 0.0).softmax(-1))
        outs.append(torch.einsum("hgnm,mhd->nhgd", p, b[2][at:at + n]).reshape(n, Hq, d))
        at += n
    want = torch.cat(outs)
    for name, x, y in zip(("o", "dq", "dk", "dv"), (o,) + grads, (want,) + torch.autograd.grad(want, b, do.double())):
        rel = float((x.detach().double() - y.detach()).norm() / y.detach().norm())
        # P, dS and the results are rounded to 16 bits: 2^-9 (2^-12 in fp16) each, two or three times; once instead of twice is 0.1
        assert rel <= (8e-3 if dtype == torch.bfloat16 else 1e-3), (name, rel)
    n = lens[-1]
    last = pkg.ops.topk_sparse_attention_decode(q[-1:], k[N - n:][None], v[N - n:][None], idx[:, -1:].cuda(), bs,
                                                torch.tensor([n], dtype=torch.int32).cuda())
    err = (last[0].double() - want[-1].detach()).abs() / want[-1].detach().abs().clamp(min=1.0)
    assert float(err.max()) <= 2e-2
    assert pkg.device_status() == 0


def test_rows_outside_the_sequences_are_written():
    """Padding rows behind the last sequence: they continue it, as they do where the private walk takes every token."""
    import native_sparse_attention_triton_b200 as pkg
    from native_sparse_attention_triton_b200 import _lib
    Hq, Hkv, d, bs, topk, N, used = 8, 2, 128, 64, 4, 700, 530
    g = torch.Generator().manual_seed(29)
    rnd = lambda h: torch.randn(N, h, d, generator=g).bfloat16().cuda()
    q, k, v = rnd(Hq), rnd(Hkv), rnd(Hkv)
    idx = selection(g, [200, N - 200], Hkv, bs, topk).cuda()
    out = []
    for end in (used, N):
        cu = torch.tensor([0, 200, end], dtype=torch.int32).cuda()
        o, lse = torch.full_like(q, 7.0), torch.full((N, Hq), 7.0, device="cuda")
        strides = _lib.strides_array(*[x for t in (q, k, v, o) for x in t.stride()[:2]], *idx.stride())
        rc = _lib.lib().nsa_topk_sparse_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), idx.data_ptr(), cu.data_ptr(), o.data_ptr(),
                                                 lse.data_ptr(), N, 2, Hq, Hkv, d, topk, bs, strides, d ** -0.5, _lib.DTYPE_BF16,
                                                 torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        out.append(o.float())
    err = (out[0] - out[1]).abs() / out[1].abs().clamp(min=1.0)
    assert float(err.max()) <= 2e-2, float(err.max())
    assert torch.equal(out[0][:256], out[1][:256])
    assert pkg.device_status() == 0
