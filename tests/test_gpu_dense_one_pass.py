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


def both_forms(lens_q, lens_k, Hq, Hkv, causal, window, stride):
    """The backward as a call that takes one pass, and one that takes two: chosen by the workspace.  Returns (call, its gradients) each
    and the inputs."""
    import native_sparse_attention_triton_b200 as pkg
    lib = pkg._lib.lib()
    N, m, B, d = sum(lens_q), sum(lens_k), len(lens_q), 128
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v, do = [torch.randn(n, h, d, generator=g, device="cuda").bfloat16() for n, h in ((N, Hq), (m, Hkv), (m, Hkv), (N, Hq))]
    cu_q, cu_k = (torch.tensor([0] + torch.tensor(n).cumsum(0).tolist(), dtype=torch.int32, device="cuda") for n in (lens_q, lens_k))
    o, lse = torch.empty_like(q), torch.empty(N, Hq, device="cuda")
    P, scale = lambda t: t.data_ptr(), 1 / math.sqrt(d)
    rows, kv = [Hq * d, d], [Hkv * d, d]
    fwd = pkg._lib.strides_array(*rows, *kv, *kv, *rows)
    assert lib.nsa_varlen_attn_fwd(P(q), P(k), P(v), P(cu_q), P(cu_k), P(o), P(lse), N, m, B, max(lens_q), Hq, Hkv, d, causal, window, stride, fwd, scale,
                                   0, None) == 0
    bwd = pkg._lib.strides_array(*rows, *kv, *kv, *rows, *rows, *rows, *kv, *kv)
    sizes = lib.nsa_varlen_attn_bwd_workspace_one_pass(N, m, B, max(lens_k), Hq, Hkv, d), lib.nsa_varlen_attn_bwd_workspace(N, m, Hq, Hkv, d)
    assert sizes[0] > sizes[1]

    def form(size):
        out = [torch.empty_like(t) for t in (q, k, v)]
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")

        def call():
            assert lib.nsa_varlen_attn_bwd(P(q), P(k), P(v), P(o), P(do), P(lse), P(cu_q), P(cu_k), *(P(t) for t in out), P(ws), size, N, m, B, max(lens_q),
                                           max(lens_k), Hq, Hkv, d, causal, window, stride, bwd, scale, 0, torch.cuda.current_stream().cuda_stream) == 0
        return call, out
    return form(sizes[0]), form(sizes[1]), (q, k, v, do)


def test_compressed_keys_and_the_smaller_workspace():
    """Strided causal mask: 3073 keys of 16 tokens each, against fp32 sums over every key; the two-pass kernels, chosen by the workspace,
    give the same gradients.  Both round fp32 sums to 16 bits once: they differ by single roundings (2^-8 of a value) where the sums'
    order does."""
    import native_sparse_attention_triton_b200 as pkg
    N, m, Hq, Hkv = 3073 * 16 + 5, 3073, 8, 2
    (one, a), (two, b), (q, k, v, do) = both_forms([N], [m], Hq, Hkv, 1, 16, 16)
    one(), two()
    for x, y in zip(a, b):
        assert (x.float() - y.float()).norm() <= 2 ** -8 * y.float().norm()
    # fp32, a block of queries and a head at a time: key j is seen from token 16 j + 15 on
    ref = [torch.zeros(t.shape, device="cuda") for t in (q, k, v)]
    first = torch.arange(m, device="cuda") * 16 + 15
    for at in range(0, N, 8192):
        t = slice(at, min(N, at + 8192))
        hidden = first[None, :] > torch.arange(at, t.stop, device="cuda")[:, None]
        for h in range(Hq):
            leaves = [x.float().requires_grad_(True) for x in (q[t, h], k[:, h // (Hq // Hkv)], v[:, h // (Hq // Hkv)])]
            s = (leaves[0] @ leaves[1].T / math.sqrt(128)).masked_fill(hidden, float("-inf"))
            p = s.softmax(-1).nan_to_num(0.0)  # the first 15 tokens see no key
            gq, gk, gv = torch.autograd.grad([p @ leaves[2]], leaves, [do[t, h].float()])
            ref[0][t, h] = gq.nan_to_num(0.0)
            ref[1][:, h // (Hq // Hkv)] += gk.nan_to_num(0.0)
            ref[2][:, h // (Hq // Hkv)] += gv
    for name, x, r in zip(("dq", "dk", "dv"), a, ref):
        assert_close_16bit(x, r.cpu(), name, grad_tol(name, False), MEAN_TOL)
    assert pkg.device_status() == 0


@pytest.mark.parametrize("Hq,Hkv,lens,causal", [
    (2, 2, [3072], 1),           # CTAs of 8 row tiles, the least
    (8, 8, [3072] * 4, 1),       # 16, the most for groups of one and two
    (4, 1, [5000, 3071], 1),     # 16
    (16, 1, [6100], 1),          # 32
    (16, 1, [9000], 0),          # 64, the most
    (16, 1, [24600], 1),
])
def test_cta_lengths(Hq, Hkv, lens, causal):
    """One pass against two, as above, with CTAs of every length."""
    import native_sparse_attention_triton_b200 as pkg
    (one, a), (two, b), _ = both_forms(lens, lens, Hq, Hkv, causal, 1, 1)
    one(), two()
    for x, y in zip(a, b):
        assert (x.float() - y.float()).norm() <= 2 ** -8 * y.float().norm()
    assert pkg.device_status() == 0


def test_one_query_head_per_key_head_is_not_slower():
    """Groups of one, whose row tiles are 128 tokens: in turn with the two passes, where CTAs of few row tiles took 1.07 of their time
    (as long as the CTAs should be: 0.71)."""
    (one, _), (two, _), _ = both_forms([3072] * 4, [3072] * 4, 8, 8, 1, 1, 1)
    times = [[], []]
    for i in range(20):
        for call, ts in zip((one, two), times):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record(), call(), end.record()
            end.synchronize()
            ts.append(start.elapsed_time(end))
    one_ms, two_ms = (sorted(ts)[len(ts) // 2] for ts in times)
    assert one_ms < two_ms


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


@pytest.mark.parametrize("lens", [[3100], [1500, 700]])  # one pass, two passes
@pytest.mark.parametrize("expanded", ["tokens", "tokens and heads"])
def test_expanded_gradient(lens, expanded):
    """The gradient of a sum over tokens, or over tokens and heads: strides of 0."""
    import native_sparse_attention_triton_b200 as pkg
    N, Hq, Hkv, d = sum(lens), 8, 2, 128
    g = torch.Generator(device="cuda").manual_seed(N)
    q, k, v = [torch.randn(N, h, d, generator=g, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv)]
    w = torch.randn(1, 1 if expanded == "tokens and heads" else Hq, d, generator=g, device="cuda").bfloat16()
    do = w.expand(N, Hq, d)
    leaves = [t.detach().requires_grad_(True) for t in (q, k, v)]
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    pkg.ops.flash_attention_varlen(*leaves, cu, cu, max(lens), max(lens), causal=True).backward(do)
    for name, t, ref in zip(("dq", "dk", "dv"), leaves, reference(q, k, v, do, lens, True)):
        assert_close_16bit(t.grad, ref.cpu(), name, grad_tol(name, False), MEAN_TOL)
    assert pkg.device_status() == 0


def kernels(call):
    """Names of the kernels that a call launches."""
    import native_sparse_attention_triton_b200 as pkg
    pkg._lib.profile(True)
    try:
        call()
        torch.cuda.synchronize()
        return set(pkg._lib.profile_collect())
    finally:
        pkg._lib.profile(False)


def test_two_passes_where_the_larger_workspace_does_not_fit():
    import native_sparse_attention_triton_b200 as pkg
    N, Hq, Hkv, d = 3072, 64, 4, 128
    g = torch.Generator(device="cuda").manual_seed(9)
    q, k, v, do = [torch.randn(N, h, d, generator=g, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv, Hq)]
    leaves = [t.requires_grad_(True) for t in (q, k, v)]
    cu = torch.tensor([0, N], dtype=torch.int32, device="cuda")
    grads = lambda: torch.autograd.grad([pkg.ops.flash_attention_varlen(*leaves, cu, cu, N, N, causal=True)], leaves, [do])
    want = []
    assert "dense_bwd_tc" in kernels(lambda: want.extend(t.cpu() for t in grads()))
    o = pkg.ops.flash_attention_varlen(*leaves, cu, cu, N, N, causal=True)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total, held = torch.cuda.get_device_properties(0).total_memory, torch.cuda.memory_reserved()
    filler, got = [], []
    try:
        torch.cuda.set_per_process_memory_fraction(held / total)
        for size in (32 << 20, 4 << 20, 2 << 20):  # room in the pieces that the process holds
            try:
                while True:
                    filler.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                pass
        # 100 MiB more are enough for dq, dk and dv (48 + 3 + 3) and the smaller workspace (14); the larger one is 110
        torch.cuda.set_per_process_memory_fraction((held + (100 << 20)) / total)
        ran = kernels(lambda: got.extend(torch.autograd.grad([o], leaves, [do])))
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert "dense_dq_tc" in ran and "dense_bwd_tc" not in ran
    for x, y in zip((t.cpu() for t in got), want):
        assert (x.float() - y.float()).norm() <= 2 ** -8 * y.float().norm()
    assert pkg.device_status() == 0


def test_dq_repeats_itself_where_that_is_asked_for():
    import native_sparse_attention_triton_b200 as pkg
    N, Hq, Hkv, d = 3500, 32, 2, 128
    g = torch.Generator(device="cuda").manual_seed(10)
    q, k, v, do = [torch.randn(N, h, d, generator=g, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv, Hq)]
    cu = torch.tensor([0, N], dtype=torch.int32, device="cuda")
    o = pkg.ops.flash_attention_varlen(q.requires_grad_(True), k, v, cu, cu, N, N, causal=True)
    got = []
    torch.use_deterministic_algorithms(True)
    try:
        ran = kernels(lambda: got.extend(torch.autograd.grad([o], [q], [do], retain_graph=True)[0] for _ in range(3)))
    finally:
        torch.use_deterministic_algorithms(False)
    assert "dense_bwd_tc" not in ran
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    assert "dense_bwd_tc" in kernels(lambda: torch.autograd.grad([o], [q], [do]))
