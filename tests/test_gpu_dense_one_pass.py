"""dQ, dK and dV of dense attention in one pass (3072 keys and more): gradients against fp32 torch on the GPU over every group size,
lengths at and beside the edges of key tiles, row tiles and token chunks, both masks, and against the two-pass kernels, which the same
call takes with the smaller workspace."""
import math

import pytest
import torch

from tests.helpers import MEAN_TOL, assert_close_16bit, grad_tol

pytestmark = pytest.mark.gpu


def reference(q, k, v, do, lens, causal):
    """fp32 gradients, sequence by sequence."""
    out, at = [[], [], []], 0
    for n in lens:
        qs, ks, vs = [t[at:at + n].float().requires_grad_(True) for t in (q, k, v)]
        G = q.shape[1] // k.shape[1]
        s = torch.einsum("qhgd,khd->hgqk", qs.view(n, -1, G, q.shape[2]), ks) / math.sqrt(q.shape[2])
        if causal:
            s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
        o = torch.einsum("hgqk,khd->qhgd", s.softmax(-1), vs).reshape(n, q.shape[1], q.shape[2])
        for acc, g in zip(out, torch.autograd.grad([o], [qs, ks, vs], [do[at:at + n].float()])):
            acc.append(g)
        at += n
    return [torch.cat(x) for x in out]


@pytest.mark.parametrize("Hq,Hkv,lens,causal,dtype", [
    (16, 1, [3072], True, torch.bfloat16),             # 8 tokens per row tile
    (16, 2, [3201], True, torch.float16),              # 16; a key tile of one key
    (8, 2, [3583, 1700], True, torch.bfloat16),        # 32
    (4, 2, [3100, 3000], False, torch.float16),        # 64
    (2, 2, [4097, 2049, 5000], True, torch.bfloat16),  # 128
    (16, 1, [3073], False, torch.bfloat16),
])
def test_gradients(Hq, Hkv, lens, causal, dtype):
    import native_sparse_attention_triton_b200 as pkg
    N, d = sum(lens), 128
    g = torch.Generator(device="cuda").manual_seed(Hq + N)
    q, k, v, do = [torch.randn(N, h, d, generator=g, device="cuda").to(dtype) for h in (Hq, Hkv, Hkv, Hq)]
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    for t in (q, k, v):
        t.requires_grad_(True)
    # the rule takes these calls to the one pass: its workspace is the larger one
    sizes = (N, N, len(lens), max(lens), Hq, Hkv, d)
    lib = pkg._lib.lib()
    assert lib.nsa_varlen_attn_bwd_workspace_one_pass(*sizes) > lib.nsa_varlen_attn_bwd_workspace(N, N, Hq, Hkv, d)
    pkg.ops.flash_attention_varlen(q, k, v, cu, cu, max(lens), max(lens), causal=causal).backward(do)
    for name, t, ref in zip(("dq", "dk", "dv"), (q, k, v), reference(q.detach(), k.detach(), v.detach(), do, lens, causal)):
        assert_close_16bit(t.grad, ref.cpu(), name, grad_tol(name, False), MEAN_TOL)
    assert pkg.device_status() == 0


def test_compressed_keys_and_the_smaller_workspace():
    """Strided causal mask: 3073 keys of 16 tokens each; the two-pass kernels, chosen by the workspace, give the same gradients.
    Both round fp32 sums to 16 bits once: they differ by single roundings (2^-8 of a value) where the sums' order does."""
    import native_sparse_attention_triton_b200 as pkg
    lib = pkg._lib.lib()
    N, m, Hq, Hkv, d = 3073 * 16 + 5, 3073, 8, 2, 128
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v, do = [torch.randn(n, h, d, generator=g, device="cuda").bfloat16() for n, h in ((N, Hq), (m, Hkv), (m, Hkv), (N, Hq))]
    cu_q, cu_k = (torch.tensor([0, n], dtype=torch.int32, device="cuda") for n in (N, m))
    o, lse = torch.empty_like(q), torch.empty(N, Hq, device="cuda")
    P, scale = lambda t: t.data_ptr(), 1 / math.sqrt(d)
    rows, kv = [Hq * d, d], [Hkv * d, d]
    fwd = pkg._lib.strides_array(*rows, *kv, *kv, *rows)
    assert lib.nsa_varlen_attn_fwd(P(q), P(k), P(v), P(cu_q), P(cu_k), P(o), P(lse), N, m, 1, N, Hq, Hkv, d, 1, 16, 16, fwd, scale, 0, None) == 0
    bwd = pkg._lib.strides_array(*rows, *kv, *kv, *rows, *rows, *rows, *kv, *kv)
    grads = []
    for size in (lib.nsa_varlen_attn_bwd_workspace_one_pass(N, m, 1, m, Hq, Hkv, d), lib.nsa_varlen_attn_bwd_workspace(N, m, Hq, Hkv, d)):
        out = [torch.empty_like(t) for t in (q, k, v)]
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        assert lib.nsa_varlen_attn_bwd(P(q), P(k), P(v), P(o), P(do), P(lse), P(cu_q), P(cu_k), *(P(t) for t in out), P(ws), size, N, m, 1, N, m,
                                       Hq, Hkv, d, 1, 16, 16, bwd, scale, 0, None) == 0
        torch.cuda.synchronize()
        grads.append(out)
    for a, b in zip(*grads):
        assert (a.float() - b.float()).norm() <= 2 ** -8 * b.float().norm()
    assert pkg.device_status() == 0


@pytest.mark.parametrize("Hq,Hkv,lens_q,lens_k,dtype", [
    (16, 1, [200, 5], [3500, 3100], torch.bfloat16),   # fewer queries than keys
    (8, 4, [4000, 0, 1], [3072, 3300, 3200], torch.float16),  # a sequence without queries, one with a single one
])
def test_other_lengths_and_strides(Hq, Hkv, lens_q, lens_k, dtype):
    """No mask, queries and keys of different lengths, all inputs and the gradient strided views."""
    import native_sparse_attention_triton_b200 as pkg
    d, Nq, Nk = 128, sum(lens_q), sum(lens_k)
    g = torch.Generator(device="cuda").manual_seed(Nq)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dtype)
    q = rnd(Hq, Nq, d).transpose(0, 1)              # heads outermost
    k, v = rnd(Nk, 2, Hkv, d).unbind(1)             # packed pairs
    do = rnd(Nq, Hq + 1, d + 8)[:, 1:, :d]          # padded rows
    leaves = [t.detach().requires_grad_(True) for t in (q, k, v)]
    cu = [torch.tensor([0] + torch.tensor(n).cumsum(0).tolist(), dtype=torch.int32, device="cuda") for n in (lens_q, lens_k)]
    assert pkg._lib.lib().nsa_varlen_attn_bwd_workspace_one_pass(Nq, Nk, len(lens_k), max(lens_k), Hq, Hkv, d) > \
        pkg._lib.lib().nsa_varlen_attn_bwd_workspace(Nq, Nk, Hq, Hkv, d)
    pkg.ops.flash_attention_varlen(*leaves, *cu, max(lens_q), max(lens_k), causal=False).backward(do)
    ref = [t.detach().float().requires_grad_(True) for t in (q, k, v)]
    outs, aq, ak = [], 0, 0
    for nq, nk in zip(lens_q, lens_k):
        qs, ks, vs = ref[0][aq:aq + nq], ref[1][ak:ak + nk], ref[2][ak:ak + nk]
        s = torch.einsum("qhgd,khd->hgqk", qs.reshape(nq, Hkv, Hq // Hkv, d), ks) / math.sqrt(d)
        outs.append(torch.einsum("hgqk,khd->qhgd", s.softmax(-1), vs).reshape(nq, Hq, d))
        aq, ak = aq + nq, ak + nk
    torch.cat(outs).backward(do.float())
    for name, a, b in zip(("dq", "dk", "dv"), leaves, ref):
        assert_close_16bit(a.grad, b.grad.cpu(), name, grad_tol(name, False), MEAN_TOL)
    assert pkg.device_status() == 0
