"""Block selection on the tcgen05 score pass: groups of eight query heads, and groups of sixteen with wide folds."""
import pytest
import torch

from native_sparse_attention_triton_b200 import _lib, device_status, ops

pytestmark = pytest.mark.gpu


def _cu(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return cu


def _launches(run):
    """Names of the library's kernels that run() launches."""
    _lib.profile(True)
    try:
        run()
        return set(_lib.profile_collect())
    finally:
        _lib.profile(False)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("lens", [[15, 16, 17, 31, 33], [639, 641, 655, 1023], [700, 4000]])
def test_scores_of_groups_of_eight(d, lens):
    """Selection with eight query heads per KV head (16 tokens in a row tile, three folds per thread) against the oracle's scores."""
    from oracle import nsa_oracle as oracle

    g = torch.Generator(device="cuda").manual_seed(d)
    cq, windows = _cu(lens), [max(0, (n - 32) // 16 + 1) for n in lens]
    ck = _cu(windows)
    q = torch.randn(cq[-1], 16, d, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(ck[-1], 2, d, generator=g, device="cuda").bfloat16() for _ in range(2))
    cu_q, cu_k = (torch.tensor(c, dtype=torch.int32, device="cuda") for c in (cq, ck))
    out = []
    names = _launches(lambda: out.append(ops.compressed_attention(q, k, v, 32, 16, 64, 8, cu_q, cu_k, max(lens), max(windows), None, 1, 2)))
    assert "score_topk_tc" in names and "score_topk" not in names
    _, want, scores = oracle.compressed_attention(q.float().cpu(), k.float().cpu(), v.float().cpu(), 32, 16, 64, 8, cu_q.cpu(), cu_k.cpu(),
                                                  max(lens), max(windows), None, 1, 2, return_scores=True)
    bad, _, _ = oracle.compare_topk_idx(out[0][1].cpu(), want, scores, tie_tol=1e-3)
    assert bad == 0
    assert device_status() == 0


def wrongest_choice(ks, st, bs, hq, hkv, d, n, topk, alike):
    """Selection of one sequence of n tokens from float64 log-sum-exps, against float64 block scores: the largest (best block left out -
    worst block taken) / best block left out over the rows, and the kernels that ran.  With `alike` the query heads of a group are the
    same, so that nothing averages out over them."""
    g = torch.Generator(device="cuda").manual_seed(ks + st + d)
    G, m, nb = hq // hkv, (n - ks) // st + 1, (n + bs - 1) // bs
    q = torch.randn(n, hkv, 1 if alike else G, d, generator=g, device="cuda").bfloat16().expand(n, hkv, G, d).reshape(n, hq, d).contiguous()
    k = torch.randn(m, hkv, d, generator=g, device="cuda").bfloat16()
    t, j = torch.arange(n, device="cuda")[:, None], torch.arange(m, device="cuda")[None]
    seen = j * st + ks - 1 <= t
    a, c = ks // st, bs // st
    block, key = torch.arange(nb, device="cuda")[None], torch.arange(m, device="cuda")[:, None]
    first = key - (block * c - (a - 1))                  # the key's place among the a + c - 1 that touch the block
    fold = torch.stack([first + 1, a + c - 1 - first, torch.full_like(first, min(a, c))]).amin(0).clamp(min=0).double()
    lse, scores = torch.full((n, hq), -torch.inf, dtype=torch.float64, device="cuda"), torch.zeros(hkv, n, nb, dtype=torch.float64, device="cuda")
    for h in range(hq):
        s = (q[:, h].double() @ k[:, h // G].double().T / d ** 0.5).masked_fill(~seen, -torch.inf)
        lse[:, h] = torch.logsumexp(s, 1) / torch.log(torch.tensor(2.0, dtype=torch.float64))
        scores[h // G] += torch.softmax(s, 1).nan_to_num(0.0) @ fold
    lse = lse.float().contiguous()
    idx = torch.empty(hkv, n, min(topk, nb), dtype=torch.int32, device="cuda")
    cu_q, cu_k = (torch.tensor([0, x], dtype=torch.int32, device="cuda") for x in (n, m))
    strides = _lib.strides_array(q.stride(0), q.stride(1), k.stride(0), k.stride(1), *idx.stride())
    rc = []
    names = _launches(lambda: rc.append(_lib.lib().nsa_compressed_attn_topk(
        q.data_ptr(), k.data_ptr(), lse.data_ptr(), cu_q.data_ptr(), cu_k.data_ptr(), idx.data_ptr(), n, m, 1, n, hq, hkv, d, ks, st, bs, topk, 1, 2,
        strides, d ** -0.5, _lib.DTYPE_BF16, torch.cuda.current_stream().cuda_stream)))
    assert rc == [0] and device_status() == 0
    taken = torch.zeros(hkv, n, nb + 1, dtype=torch.bool, device="cuda")
    taken.scatter_(2, torch.where(idx < 0, nb, idx).long(), True)
    taken = taken[..., :nb]
    own = (torch.arange(n, device="cuda") // bs)[:, None]
    visible, forced = block <= own, (block == 0) | ((block <= own) & (block > own - 2))
    assert not (taken & ~visible).any() and (taken | ~(forced & visible)).all()
    assert (taken.sum(2) == (own[:, 0] + 1).clamp(max=idx.shape[2])).all()
    left = torch.where(visible & ~taken, scores, -1.0).amax(2)
    worst = torch.where(taken & ~forced, scores, torch.inf).amin(2)
    return torch.where((left > 0) & worst.isfinite(), (left - worst) / left, 0.0).max().item(), names


# 8 tokens x 65 or 64 blocks per 128 keys: more pairs than the fold held on the kernels with exact exponentials before it
@pytest.mark.parametrize("fold", [(64, 32, 64), (32, 32, 64)])
@pytest.mark.parametrize("heads", [(64, 4, 128), (16, 1, 64)])
@pytest.mark.parametrize("alike", [True, False])
def test_wide_folds_keep_exact_exponentials(fold, heads, alike):
    wrong, names = wrongest_choice(*fold, *heads, 8192, 32, alike)
    assert "score_topk_tc" in names and "score_topk" not in names
    # An exponent of up to 16 in size is rounded to 2^-20 twice (logit, log-sum-exp); sums and the exponential unit (2^-22) add less than
    # that again: 4 x 2^-20 ln 2 for a score, and two scores are compared.  A cubic in every second pair makes it several times that.
    assert wrong <= 8 * 2.0 ** -20 * 0.6932
