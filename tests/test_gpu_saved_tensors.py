"""Saved tensors of the operators' autograd nodes under hooks: activation checkpointing, which computes the forward again while the
backward unpacks them, and hooks that hand out copies."""
import pytest
import torch
from torch.utils.checkpoint import checkpoint

pytestmark = pytest.mark.gpu
KS, ST, BS, TOPK, LENS = 32, 16, 64, 4, [100, 333]


def layer(ops, cu, inv_freq, x, wk, wv, pe, gate):
    """Every operator with a backward, fed by torch's own arithmetic so that what is recomputed has a graph of its own."""
    q = (x * 0.5).repeat_interleave(4, 1)
    k, v = x * 1.5, x + 0.25
    ck, cu_k = ops.linear_compress(k, wk * 1.0, cu, KS, ST, pe * 1.0)
    cv, _ = ops.weightedpool_compress(v, wv * 1.0, cu, KS, ST)
    q, k, ck = ops.rope(q, inv_freq, cu), ops.rope(k, inv_freq, cu), ops.rope(ck, inv_freq, cu_k, 0, ST)
    o_cmp, idx = ops.compressed_attention(q, ck, cv, KS, ST, BS, TOPK, cu, cu_k, max(LENS), 20, None, 1, 2)
    o_sel = ops.topk_sparse_attention(q, k, v, idx, BS, cu)
    o_win = ops.sliding_window_attention(q, k, v, cu, max(LENS), 64)
    o = ops.flash_attention_varlen(q, k, v, cu, cu, max(LENS), max(LENS), causal=True)
    return ops.gate_combine(gate * 1.0, o_cmp, o_sel, o_win) + o


@pytest.mark.parametrize("how", ["checkpoint", "hooks"])
def test_gradients_are_those_without_hooks(how):
    import native_sparse_attention_triton_b200 as pkg
    g = torch.Generator(device="cuda").manual_seed(2)
    N, H, d = sum(LENS), 2, 128
    rnd = lambda *s, scale=1.0: (torch.randn(*s, generator=g, device="cuda") * scale).bfloat16()
    leaves = [rnd(N, H, d), rnd(H, KS * d, d, scale=(KS * d) ** -0.5), rnd(H, KS, scale=KS ** -0.5), rnd(H, KS, d, scale=0.02),
              torch.rand(N, 4 * H, 3, generator=g, device="cuda").bfloat16()]
    cu = torch.tensor([0, LENS[0], N], dtype=torch.int32, device="cuda")
    inv_freq = 1.0 / (10000.0 ** (torch.arange(0, d, 2, device="cuda") / d))
    dy = rnd(N, 4 * H, d)
    f = lambda *a: layer(pkg.ops, cu, inv_freq, *a)

    def grads(run):
        a = [t.clone().requires_grad_(True) for t in leaves]
        return torch.autograd.grad(run(*a), a, dy)

    want = grads(f)
    packed = []
    if how == "checkpoint":
        got = grads(lambda *a: checkpoint(f, *a, use_reentrant=False))
    else:
        with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(1) or t.cpu(), lambda t: t.cuda()):
            got = grads(f)
        assert len(packed) > 30
    for name, x, y in zip(("x", "wk", "wv", "pe", "gate"), got, want):
        if name == "pe":   # shifts all compressed keys alike, which a softmax does not see: the summed rounding of the key gradients
            continue
        # the same kernels on the same values; only sums of atomic additions differ in order
        assert float((x.float() - y.float()).norm()) <= 2e-3 * float(y.float().norm()), name
    assert pkg.device_status() == 0
