"""Decode kernels that put a cluster of CTAs on each (sequence, KV head) pair: the three operators against the fp32 oracle at the
sizes where the work is dealt out differently (cluster sizes 1 to 16, four and eight warps, the split-KV kernel's range, lengths
at the edges of the 32-row sub-tiles), and the fused decode step against the operators it replaces."""
import pytest
import torch

from oracle import nsa_oracle as O

pytestmark = pytest.mark.gpu

# |o| <= max |v| of 16-bit values; P and the result are rounded once each: 2^-8 relative for bf16, plus fp32 summation
TOL = 2e-2


def close(a, b):
    err = (a.float().cpu() - b.float()).abs() / b.float().abs().clamp(min=1.0)
    assert float(err.max()) <= TOL and float(err.mean()) <= 2e-3, (float(err.max()), float(err.mean()))


@pytest.mark.parametrize("B,Hkv,G,d,L,dtype", [
    (1, 1, 16, 128, 4100, torch.bfloat16),   # one pair: clusters of 16, eight warps
    (3, 2, 4, 64, 700, torch.float16),
    (5, 1, 3, 128, 95, torch.bfloat16),      # a group that is no power of two
    (40, 4, 1, 128, 130, torch.bfloat16),    # 160 pairs: clusters of one CTA
    (150, 3, 2, 64, 65, torch.bfloat16),     # 450 pairs: compressed on the split-KV kernel
    (31, 4, 8, 128, 4200, torch.bfloat16),   # 124 pairs of long rows: dense on the split-KV kernel
])
def test_operators_against_oracle(B, Hkv, G, d, L, dtype):
    import native_sparse_attention_triton_b200 as pkg
    ops = pkg.ops
    ks, st, bs, topk = 32, 16, 64, 6
    g = torch.Generator().manual_seed(B + L)
    rnd = lambda *s: torch.randn(*s, generator=g).to(dtype)
    q, k, v = rnd(B, Hkv * G, d), rnd(B, L, Hkv, d), rnd(B, L, Hkv, d)
    lens = torch.randint(1, L + 1, (B,), generator=g)
    edges = [1, 31, 32, 33, 64, L]
    lens[:min(B, len(edges))] = torch.tensor(edges)[:B].clamp(max=L)
    lens[-1] = L
    lens = lens.int()
    Lc = (L - ks) // st + 1
    ck, cv = rnd(B, Lc, Hkv, d), rnd(B, Lc, Hkv, d)
    clens = torch.clamp((lens - ks) // st + 1, min=0).int()
    f, c = (lambda t: t.float()), (lambda t: t.cuda())
    close(ops.flash_attention_decode(c(q), c(k), c(v), c(lens)), O.flash_attention_decode(f(q), f(k), f(v), lens))
    o, idx = ops.compressed_attention_decode(c(q), c(ck), c(cv), c(lens), c(clens), ks, st, bs, topk, max_seqlen=L)
    o_ref, idx_ref = O.compressed_attention_decode(f(q), f(ck), f(cv), lens, clens, ks, st, bs, topk, 1, 2)[:2]
    close(o, o_ref)
    idx = idx.cpu()
    # block scores of N(0, 1) inputs differ by far more than fp32 rounding: the selections agree but for a rare tie
    assert float((idx != idx_ref[..., :idx.shape[-1]]).float().mean()) <= 2e-3
    close(ops.topk_sparse_attention_decode(c(q), c(k), c(v), c(idx), bs, c(lens)), O.topk_sparse_attention_decode(f(q), f(k), f(v), idx, bs, lens))
    assert pkg.device_status() == 0


@pytest.mark.parametrize("mode,lens,Hq,Hkv,d,ks,st,bs,topk,window,dtype", [
    ("weighted", [5, 31, 200], 16, 1, 128, 32, 16, 64, 4, 32, torch.bfloat16),
    ("avg", [64, 1], 8, 8, 64, 16, 16, 64, 8, 100, torch.float16),
    ("linear", [33, 300, 16], 8, 2, 128, 32, 32, 128, 3, 64, torch.bfloat16),
    ("linear", [47], 4, 1, 64, 64, 32, 64, 16, 33, torch.float16),
])
def test_fused_step_equals_operators(monkeypatch, mode, lens, Hq, Hkv, d, ks, st, bs, topk, window, dtype):
    """40 steps of the fused kernel and of the separate launches from the same prefilled state.  Copies are exact; a pooled row
    is the same fp32 sum rounded twice, a projected one differs in summation order; outputs round three branches to 16 bits."""
    import native_sparse_attention_triton_b200 as pkg
    from native_sparse_attention_triton_b200 import infer
    from native_sparse_attention_triton_b200.kv_cache import NSACache
    ops = pkg.ops
    g = torch.Generator(device="cuda").manual_seed(len(lens) + ks)
    rnd = lambda *s, scale=1.0: (torch.randn(*s, generator=g, device="cuda") * scale).to(dtype)
    B, N = len(lens), sum(lens)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    fn = {"linear": ops.linear_compress, "weighted": ops.weightedpool_compress, "avg": ops.avgpool_compress}[mode]
    w = {"linear": lambda: rnd(Hkv, ks * d, d, scale=(ks * d) ** -0.5), "weighted": lambda: rnd(Hkv, ks, scale=ks ** -0.5), "avg": lambda: None}[mode]
    rope = infer.RotaryEmbedding(1.0 / (10000.0 ** (torch.arange(0, d, 2, dtype=torch.float32, device="cuda") / d)))
    caches = [NSACache(B + 1, 512, Hkv, d, ks, st, window, dtype) for _ in range(2)]
    common = dict(rope=rope, compress_weight=(w(), w()), compress_func=(fn, fn), intra_block_pe=rnd(Hkv, ks, d, scale=0.02), kernel_size=ks,
                  kernel_stride=st, block_size=bs, topk=topk, init_blocks=1, local_blocks=2, window_size=window)
    key, value = rnd(N, Hkv, d), rnd(N, Hkv, d)
    for c in caches:   # the prefill's caches, without its sliding-window branch (head_dim 128 only)
        c.prepare_compress(cu, 0, key, value)
        ck, cu_k = fn(key, common["compress_weight"][0], cu, ks, st, common["intra_block_pe"])
        cv, _ = fn(value, common["compress_weight"][1], cu, ks, st)
        c.update_kv(cu, 0, ops.rope(ck, rope.inv_freq, cu_k, 0, st), cv, ops.rope(key, rope.inv_freq, cu), value, ops.rope(key, rope.inv_freq, cu),
                    value, cu_k)
    tol = 4e-2 if dtype == torch.bfloat16 else 6e-3
    for step in range(1, 41):
        rows = [rnd(B, Hq, d), rnd(B, Hkv, d), rnd(B, Hkv, d), torch.rand(B, Hq, 3, generator=g, device="cuda").to(dtype)]
        fused = infer.nsa_infer(cu, step, *rows, cache=caches[0], **common)
        with monkeypatch.context() as m:
            m.setattr(infer, "_fused_decode_step", lambda *a, **k: None)
            apart = infer.nsa_infer(cu, step, *rows, cache=caches[1], **common)
        err = (fused.float() - apart.float()).abs() / apart.float().abs().clamp(min=1.0)
        assert float(err.max()) <= tol and float(err.mean()) <= tol / 10, (step, float(err.max()), float(err.mean()))
        for a, b in zip(caches[0]._tensors(), caches[1]._tensors()):
            if a.dtype == torch.int32:
                assert torch.equal(a, b), step
    a, b = caches
    assert torch.equal(a.sparse_kv_cache, b.sparse_kv_cache) and torch.equal(a.sliding_kv_cache, b.sliding_kv_cache)
    assert torch.equal(a.before_compress_kv_cache, b.before_compress_kv_cache)
    assert float((a.compress_kv_cache.float() - b.compress_kv_cache.float()).abs().max()) <= (2e-2 if dtype == torch.bfloat16 else 3e-3) * 4
    assert pkg.device_status() == 0


@pytest.mark.parametrize("mode", ["weighted", "avg", "linear"])
def test_step_reads_the_parameters_it_is_given(mode):
    """Weights and position embedding overwritten behind the version counter between two steps that complete a window, and calls
    that the separate operators refuse."""
    import native_sparse_attention_triton_b200 as pkg
    from native_sparse_attention_triton_b200 import infer
    from native_sparse_attention_triton_b200.kv_cache import NSACache
    ops = pkg.ops
    B, Hq, Hkv, d, ks, st = 2, 8, 2, 128, 16, 16
    g = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s, scale=1.0: (torch.randn(*s, generator=g, device="cuda") * scale).bfloat16()
    fn = {"linear": ops.linear_compress, "weighted": ops.weightedpool_compress, "avg": ops.avgpool_compress}[mode]
    w = {"linear": lambda: rnd(Hkv, ks * d, d, scale=(ks * d) ** -0.5), "weighted": lambda: rnd(Hkv, ks, scale=ks ** -0.5), "avg": lambda: None}[mode]
    wk, wv, pe = w(), w(), rnd(Hkv, ks, d)
    rope = infer.RotaryEmbedding(torch.zeros(d // 2, device="cuda"))    # no rotation: the cached rows are the compressed ones
    cache = NSACache(B, 128, Hkv, d, ks, st, 32, torch.bfloat16)
    args = dict(rope=rope, cache=cache, compress_weight=(wk, wv), compress_func=(fn, fn), intra_block_pe=pe, kernel_size=ks, kernel_stride=st,
                block_size=64, topk=4, init_blocks=1, local_blocks=2, window_size=32)
    cu = torch.zeros(B + 1, dtype=torch.int32, device="cuda")
    keys = []
    for step in range(1, 2 * ks + 1):
        if step == ks + 1:
            for t in (wk, pe):
                if t is not None:
                    t.data.copy_(rnd(*t.shape, scale=float(t.float().std())))
        rows = [rnd(B, Hq, d), rnd(B, Hkv, d), rnd(B, Hkv, d), rnd(B, Hq, 3)]
        keys.append(rows[1])
        infer.nsa_infer(cu, step, *rows, **args)
    x = torch.stack(keys[ks:], 1).reshape(B * ks, Hkv, d)
    want = fn(x, wk, torch.arange(B + 1, dtype=torch.int32, device="cuda") * ks, ks, st, pe)[0]
    got = cache.compress_kv_cache[0, :B, 1]
    # both round a sum of about 1 + |pe| to 16 bits once or twice
    assert float((got.float() - want.float()).abs().max()) <= 4e-2
    with pytest.raises(AssertionError):
        infer.nsa_infer(cu, 1, *[r[:1] for r in rows], **args)            # fewer rows than sequences
    with pytest.raises(AssertionError):
        infer.nsa_infer(cu, 1, *rows, **{**args, "block_size": 40})       # no multiple of kernel_size


def test_forward_mode_is_refused():
    import native_sparse_attention_triton_b200 as pkg
    import torch.autograd.forward_ad as fwAD
    x = torch.randn(64, 2, 64, device="cuda").half()
    cu = torch.tensor([0, 64], dtype=torch.int32, device="cuda")
    with fwAD.dual_level():
        with pytest.raises(RuntimeError):
            pkg.ops.avgpool_compress(fwAD.make_dual(x, torch.ones_like(x)), None, cu, 32, 16, None)
        with pytest.raises(RuntimeError):
            pkg.ops.rope(fwAD.make_dual(x, torch.ones_like(x)), torch.ones(32, device="cuda"), cu)
