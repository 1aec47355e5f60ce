"""Dense attention forward on persistent CTAs: batches whose items are many, empty, or without a visible key, against float64."""
import pytest
import torch

from native_sparse_attention_triton_b200 import device_status, ops

pytestmark = pytest.mark.gpu


def _cu(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return cu


def _exact(q, k, v, cq, ck, visible):
    g = q.shape[1] // k.shape[1]
    out = torch.zeros(q.shape, dtype=torch.float64, device=q.device)
    for b in range(len(cq) - 1):
        x = q[cq[b]:cq[b + 1]].double()
        y, z = (t[ck[b]:ck[b + 1]].double().repeat_interleave(g, 1) for t in (k, v))
        see = visible(x.shape[0], y.shape[0])
        s = (torch.einsum("qhd,khd->hqk", x, y) / q.shape[2] ** 0.5).masked_fill(~see, float("-inf"))
        out[cq[b]:cq[b + 1]] = torch.einsum("hqk,khd->qhd", torch.softmax(s, -1).nan_to_num(0.0), z)
    return out


# row tiles of 128 rows, two per item: lengths around 128 / G and 256 / G tokens; runs of sequences without a compressed key (shorter
# than 32), longer than the ring of items; more items than SMs; more sequences than two turns of the search for an item (1024)
LENS = [[17], [7, 8, 9, 15, 16, 17, 31, 32, 33], [3] * 70 + [40] * 9, [200] + [5] * 12 + [1111, 64, 129, 2000], [0, 300, 0, 0, 47],
        [1 + i * 37 % 23 if i % 7 else 0 for i in range(1100)]]


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("heads", [(16, 1, 128, torch.bfloat16), (32, 8, 64, torch.float16), (4, 4, 128, torch.float16)])
@pytest.mark.parametrize("kind", ["causal", "full", "window", "compressed"])
def test_items(lens, heads, kind):
    hq, hkv, d, dtype = heads
    if kind == "window" and d != 128:
        pytest.skip("the sliding window is built for head_dim 128")
    g = torch.Generator(device="cuda").manual_seed(len(lens))
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dtype)
    cq = _cu(lens)
    windows = [max(0, (n - 32) // 16 + 1) for n in lens]
    ck = _cu(windows) if kind == "compressed" else cq
    if ck[-1] == 0:
        pytest.skip("no compressed key")
    q, k, v = randn(cq[-1], hq, d), randn(ck[-1], hkv, d), randn(ck[-1], hkv, d)
    cu_q, cu_k = (torch.tensor(c, dtype=torch.int32, device="cuda") for c in (cq, ck))
    at = lambda n: torch.arange(n, device="cuda")
    causal = lambda nq, nk: at(nk)[None] <= at(nq)[:, None]
    if kind == "compressed":
        o = ops.compressed_attention(q, k, v, 32, 16, 64, 4, cu_q, cu_k, max(lens), max(windows), None, 1, 2)[0]
        visible = lambda nq, nk: at(nk)[None] * 16 + 31 <= at(nq)[:, None]
    elif kind == "window":
        o = ops.sliding_window_attention(q, k, v, cu_q, max(lens), 100)
        visible = lambda nq, nk: causal(nq, nk) & (at(nk)[None] >= at(nq)[:, None] - 100)
    else:
        o = ops.flash_attention_varlen(q, k, v, cu_q, cu_k, max(lens), max(lens), causal=kind == "causal")
        visible = causal if kind == "causal" else lambda nq, nk: torch.ones(nq, nk, dtype=torch.bool, device="cuda")
    exact = _exact(q, k, v, cq, ck, visible)
    # output and probabilities are rounded to 16 bits: 2^-9 (bf16) or 2^-12 (fp16) of a value each, in the 2-norm; 2 of them
    assert (o.double() - exact).norm() <= 2 * (2.0 ** -9 if dtype is torch.bfloat16 else 2.0 ** -12) * exact.norm()
    assert device_status() == 0
