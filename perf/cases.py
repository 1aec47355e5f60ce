"""The work that users of this framework have it do, as measurable cases.

Five kinds, each through the public entry points as a program calls them:

* ``train``    -- forward and backward of a layer's attention: compression of keys and values, compressed attention with
                  block selection, selected-block attention and, with ``layer``, the rotary embedding, the sliding-window
                  branch and the gated sum around them;
* ``generate`` -- ``nsa_infer``: the prefill of a batch of prompts, then decode steps on the KV cache, launched one by one or
                  replayed from a ``DecodeGraph``;
* ``decode``   -- the three single-token operators on caches of their own (a server with its own cache layout);
* ``dense``    -- ``flash_attention_varlen`` forward and backward;
* ``compress`` -- one compression operator, forward and backward, on long batches.

``listed()`` names twelve cases of these; ``draw()`` gives others of the same ranges: 128 to 65 536 tokens in one to eight
sequences of even or ragged lengths, the head layouts 64/4, 32/2, 32/8, 16/2 and 16/1, head_dim 64 and 128, bf16 and fp16,
the three compressions with kernel / stride / block 32/16/64 and, more rarely, 16/16/64, 64/32/64 and 32/32/128.
"""
import math

import torch

from native_sparse_attention_triton_b200 import ops
from native_sparse_attention_triton_b200.infer import DecodeGraph, RotaryEmbedding, nsa_infer
from native_sparse_attention_triton_b200.kv_cache import NSACache

DEVICE = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
COMPRESS = {"linear": ops.linear_compress, "weighted": ops.weightedpool_compress, "avg": ops.avgpool_compress}


# ------------------------------------------------------------------------------------------------------------------ cases
def _case(kind, lens, hq, hkv, d=128, dtype="bf16", ks=32, st=16, bs=64, **more):
    return dict(kind=kind, lens=",".join(str(n) for n in lens), hq=hq, hkv=hkv, d=d, dtype=dtype, ks=ks, st=st, bs=bs, **more)


def listed():
    named = [
        # fine-tuning on short samples: every kernel is small, what counts is launches and host time
        ("layer_short_samples", _case("train", [200, 777], 32, 2, compress="weighted", topk=8, layer=True, window=512)),
        # packed training batch of ragged documents, linear compression
        ("chain_packed_16k", _case("train", [1024, 7168, 8192], 64, 4, compress="linear", topk=16, layer=False, window=0)),
        # long-context training: the sequence length and widths of the headline benchmark
        ("chain_one_64k", _case("train", [65536], 64, 4, compress="linear", topk=16, layer=False, window=0)),
        # one sequence of the 8 x 32 768-token layer configuration, with rotary embedding, window and gates
        ("layer_one_32k", _case("train", [32768], 64, 4, compress="linear", topk=8, layer=True, window=512)),
        # a model with groups of four query heads, fp16, lengths of the operators' own tests (one of odd size)
        ("layer_gqa4_fp16", _case("train", [1000, 2001, 4096], 32, 8, dtype="fp16", compress="avg", topk=16, layer=True, window=512)),
        # a model with head_dim 64
        ("chain_head_dim_64", _case("train", [333, 2500, 5000], 16, 2, d=64, compress="linear", topk=8, layer=False, window=0)),
        # dense causal attention of the first layers of a hybrid model, and what sparse attention is compared with
        ("dense_causal_8k", _case("dense", [8192], 64, 4, causal=True)),
        # compression alone over a layer's batch of eight 32 768-token sequences
        ("compress_8x32k", _case("compress", [32768] * 8, 64, 4, compress="weighted")),
        # chat turns: short ragged prompts, then tokens one at a time from a Python loop
        ("generate_short_prompts", _case("generate", [512, 77, 300, 450], 32, 2, compress="weighted", topk=8, window=512, steps=16, graph=False)),
        # long prompts of the generation configuration, decode steps replayed from a CUDA graph
        ("generate_4x8k_graph", _case("generate", [8192] * 4, 32, 2, compress="weighted", topk=8, window=512, steps=32, graph=True)),
        # one layer's three single-token operators for four sequences, as in that configuration
        ("decode_batch_4", _case("decode", [8256] * 4, 32, 2, topk=8, cache=8320)),
        # a serving batch: 76 sequences of 1 to 8192 tokens, the shape of the decode operators' self-test
        ("decode_batch_76", _case("decode", [min(8192, i * 37 % 76 * 128 + 1) for i in range(76)], 32, 4, topk=16, cache=8192)),
    ]
    return [dict(name=n, **c) for n, c in named]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _split(rng, total, seqs):
    """`total` tokens in `seqs` sequences: even lengths, or ragged ones of any size from 1 up."""
    if rng.random() < 0.4:
        return [max(1, total // seqs)] * seqs
    weights = [rng.uniform(0.05, 1.0) for _ in range(seqs)]
    return [max(1, int(total * w / sum(weights))) for w in weights]


def draw(rng):
    kind = rng.choice(["train"] * 8 + ["generate"] * 4 + ["decode"] * 4 + ["dense"] * 2 + ["compress"] * 2)
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16"])
    d = rng.choice([128, 128, 128, 64])
    hq, hkv = rng.choice([(64, 4), (64, 4), (32, 2), (32, 2), (32, 8), (16, 2), (16, 1)])
    ks, st, bs = rng.choice([(32, 16, 64)] * 7 + [(16, 16, 64), (64, 32, 64), (32, 32, 128)])
    compress = rng.choice(["linear", "linear", "weighted", "avg"])
    topk = rng.choice([8, 8, 16, 16, 12, 24])
    common = dict(dtype=dtype, d=d, ks=ks, st=st, bs=bs)
    if kind == "train":
        lens = _split(rng, _log_uniform(rng, 256, 65536 if d == 128 and topk <= 16 else 16384), rng.choice([1, 1, 2, 3, 4, 8]))
        if max(lens) > 32768:
            layer = False   # the largest listed case is a chain without the layer's other branches
        else:
            layer = d == 128 and rng.random() < 0.6   # the sliding-window branch is built for head_dim 128
        lens[0] = max(lens[0], 2 * ks)
        return _case("train", lens, hq, hkv, **common, compress=compress, topk=topk, layer=layer, window=rng.choice([128, 512, 512]) if layer else 0)
    if kind == "generate":
        common["d"] = 128
        lens = _split(rng, _log_uniform(rng, 128, 32768), rng.choice([1, 2, 4, 4, 7, 8]))
        lens[0] = max(lens[0], 2 * ks)
        return _case("generate", lens, hq, hkv, **common, compress=compress, topk=topk, window=rng.choice([128, 512, 512]),
                     steps=rng.randint(4, 32), graph=rng.random() < 0.5)
    if kind == "decode":
        cache = _log_uniform(rng, 512, 8192)
        batch = _log_uniform(rng, 1, 256)
        lens = [cache if rng.random() < 0.2 else rng.randint(1, cache) for _ in range(batch)]
        return _case("decode", lens, hq, hkv, **common, topk=topk, cache=cache)
    if kind == "dense":
        lens = _split(rng, _log_uniform(rng, 128, 8192), rng.choice([1, 1, 2, 4]))
        return _case("dense", lens, hq, hkv, **common, causal=rng.random() < 0.8)
    lens = _split(rng, _log_uniform(rng, 1024, 524288 if compress != "linear" else 262144), rng.choice([1, 4, 8]))
    lens[0] = max(lens[0], 2 * ks)
    return _case("compress", lens, hq, hkv, **common, compress=compress)


# ----------------------------------------------------------------------------------------------------------------- inputs
def _lens(c):
    return [int(n) for n in c["lens"].split(",")]


def _windows(n, c):
    return 0 if n < c["ks"] else (n - c["ks"]) // c["st"] + 1


class _Maker:
    """Seeded tensors on the GPU."""

    def __init__(self, seed, dtype):
        self.g = torch.Generator(device=DEVICE).manual_seed(seed)
        self.dtype = dtype

    def normal(self, *shape, scale=1.0):
        return (torch.randn(*shape, generator=self.g, device=DEVICE, dtype=torch.float32) * scale).to(self.dtype)

    def uniform(self, *shape):
        return torch.rand(*shape, generator=self.g, device=DEVICE, dtype=torch.float32).to(self.dtype)

    def keys(self, rows, heads, d):
        """Keys of a text: neighbours share a direction (one per 64 tokens), so that pooled keys and block scores differ from
        one another as they do in a model, and each has one of its own."""
        shared = torch.randn((rows + 63) // 64, heads, d, generator=self.g, device=DEVICE).repeat_interleave(64, 0)[:rows]
        return ((torch.randn(rows, heads, d, generator=self.g, device=DEVICE) + shared) * 0.5 ** 0.5).to(self.dtype)

    def weights(self, c):
        """(weight of k, weight of v, position embedding) of a compression."""
        h, ks, d = c["hkv"], c["ks"], c["d"]
        if c["compress"] == "linear":
            w = [self.normal(h, ks * d, d, scale=1 / math.sqrt(ks * d)) for _ in range(2)]
        elif c["compress"] == "weighted":
            w = [self.normal(h, ks, scale=1 / math.sqrt(ks)) for _ in range(2)]
        else:
            w = [None, None]
        return w[0], w[1], self.normal(h, ks, d, scale=0.02)

    def selection(self, lens, hkv, bs, topk):
        """Block ids as the selection gives them, int32 [hkv, tokens, width]: the first block, the two that end at the query's
        own, others at random among those before it; ascending, padded with -1."""
        width = min(topk, (max(lens) + bs - 1) // bs)
        out = torch.full((hkv, sum(lens), width), -1, dtype=torch.int32, device=DEVICE)
        at = 0
        for n in lens:
            nb = (n + bs - 1) // bs
            take = min(width, nb)
            ids = torch.arange(nb, device=DEVICE)
            own = (torch.arange(n, device=DEVICE) // bs)[:, None]
            for h in range(hkv):
                key = torch.rand(n, nb, generator=self.g, device=DEVICE)
                key = torch.where((ids[None] == 0) | (ids[None] > own - 2), 2.0, key).masked_fill_(ids[None] > own, -1.0)
                score, pick = key.topk(take, dim=1)
                pick = torch.where(score < 0, nb, pick).sort(1).values
                out[h, at:at + n, :take] = torch.where(pick == nb, -1, pick).to(torch.int32)
            at += n
        return out


def _cu(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return torch.tensor(cu, dtype=torch.int32, device=DEVICE)


def _inv_freq(d):
    return 1.0 / (500000.0 ** (torch.arange(0, d, 2, dtype=torch.float32, device=DEVICE) / d))


def prepare(case, seed):
    return {"train": _prepare_train, "generate": _prepare_generate, "decode": _prepare_decode, "dense": _prepare_dense,
            "compress": _prepare_compress}[case["kind"]](case, _Maker(seed, DTYPES[case["dtype"]]))


def _prepare_train(c, m):
    lens = _lens(c)
    n, hq, hkv, d = sum(lens), c["hq"], c["hkv"], c["d"]
    s = dict(c=c, cu=_cu(lens), max_q=max(lens), max_k=max(_windows(x, c) for x in lens), q=m.normal(n, hq, d), k=m.keys(n, hkv, d),
             v=m.normal(n, hkv, d))
    s["wk"], s["wv"], s["pe"] = m.weights(c)
    s["dy"] = [m.normal(n, hq, d) for _ in range(1 if c["layer"] else 2)]
    if c["layer"]:
        s["gate"], s["inv_freq"] = m.uniform(n, hq, 3), _inv_freq(d)
    # The selected-block branch follows a selection that the program holds, as one that recomputes activations does: two
    # correct block scores may break a tie differently, and that must not move the outputs that are compared.
    s["idx"] = m.selection(lens, hkv, c["bs"], c["topk"])
    # The gradient of pe is left out: shifting every compressed key alike leaves a softmax as it is, so what it holds is the
    # summed rounding of the key gradients.
    s["leaves"] = [s[x].requires_grad_(True) for x in ("q", "k", "v", "wk", "wv", "gate") if s.get(x) is not None]
    return s


def _prepare_generate(c, m):
    lens = _lens(c)
    n, b, hq, hkv, d = sum(lens), len(lens), c["hq"], c["hkv"], c["d"]
    rows = lambda r: [m.normal(r, hq, d), m.keys(r, hkv, d), m.normal(r, hkv, d), m.uniform(r, hq, 3)]
    s = dict(c=c, cu=_cu(lens), prompt=rows(n), steps=[rows(b) for _ in range(c["steps"])])
    wk, wv, pe = m.weights(c)
    fn = COMPRESS[c["compress"]]
    cache = NSACache(b, max(lens) + c["steps"] + 64, hkv, d, c["ks"], c["st"], c["window"], DTYPES[c["dtype"]], DEVICE)
    s["args"] = dict(rope=RotaryEmbedding(_inv_freq(d)), cache=cache, compress_weight=(wk, wv), compress_func=(fn, fn), intra_block_pe=pe,
                     kernel_size=c["ks"], kernel_stride=c["st"], block_size=c["bs"], topk=c["topk"], init_blocks=1, local_blocks=2,
                     window_size=c["window"])
    if c["graph"]:
        nsa_infer(s["cu"], 0, *s["prompt"], **s["args"])
        s["graph"] = DecodeGraph(s["cu"], *s["steps"][0], **s["args"])
    return s


def _prepare_decode(c, m):
    lens, b, hq, hkv, d, rows = _lens(c), len(_lens(c)), c["hq"], c["hkv"], c["d"], c["cache"]
    comp = max(1, _windows(rows, c))
    s = dict(c=c, q=m.normal(b, hq, d), seqlens=torch.tensor(lens, dtype=torch.int32, device=DEVICE),
             comp_lens=torch.tensor([_windows(x, c) for x in lens], dtype=torch.int32, device=DEVICE))
    s["k"], s["v"] = m.keys(b * rows, hkv, d).view(b, rows, hkv, d), m.normal(b, rows, hkv, d)
    s["ck"], s["cv"] = m.normal(b, comp, hkv, d), m.normal(b, comp, hkv, d)
    # the last token of each sequence chooses its blocks; held for the reason given in _prepare_train
    nb = (rows + c["bs"] - 1) // c["bs"]
    own = ((s["seqlens"] - 1) // c["bs"])[None, :, None]
    ids = torch.arange(nb, device=DEVICE)[None, None]
    key = torch.rand(hkv, b, nb, generator=m.g, device=DEVICE)
    key = torch.where((ids == 0) | (ids > own - 2), 2.0, key).masked_fill_(ids > own, -1.0)
    score, pick = key.topk(min(c["topk"], nb), dim=-1)
    pick = torch.where(score < 0, nb, pick).sort(-1).values
    s["idx"] = torch.where(pick == nb, -1, pick).to(torch.int32)
    return s


def _prepare_dense(c, m):
    lens = _lens(c)
    n, hq, hkv, d = sum(lens), c["hq"], c["hkv"], c["d"]
    s = dict(c=c, cu=_cu(lens), longest=max(lens), q=m.normal(n, hq, d), k=m.keys(n, hkv, d), v=m.normal(n, hkv, d), dy=m.normal(n, hq, d))
    s["leaves"] = [s[x].requires_grad_(True) for x in ("q", "k", "v")]
    return s


def _prepare_compress(c, m):
    lens = _lens(c)
    w, _, pe = m.weights(c)
    s = dict(c=c, cu=_cu(lens), x=m.keys(sum(lens), c["hkv"], c["d"]), w=w, pe=pe,
             dy=m.normal(sum(_windows(x, c) for x in lens), c["hkv"], c["d"]))
    s["leaves"] = [t.requires_grad_(True) for t in (s["x"], w, pe) if t is not None]
    return s


# ------------------------------------------------------------------------------------------------------------------- runs
def run(state):
    return {"train": _run_train, "generate": _run_generate, "decode": _run_decode, "dense": _run_dense,
            "compress": _run_compress}[state["c"]["kind"]](state)


def _run_train(s):
    c, cu = s["c"], s["cu"]
    ks, st, bs = c["ks"], c["st"], c["bs"]
    fn = COMPRESS[c["compress"]]
    ck, cu_k = fn(s["k"], s["wk"], cu, ks, st, s["pe"])
    cv, _ = fn(s["v"], s["wv"], cu, ks, st, None)
    q, k = s["q"], s["k"]
    if c["layer"]:
        q, ck, k = ops.rope(q, s["inv_freq"], cu), ops.rope(ck, s["inv_freq"], cu_k, 0, st), ops.rope(k, s["inv_freq"], cu)
    o_cmp, idx = ops.compressed_attention(q, ck, cv, ks, st, bs, c["topk"], cu, cu_k, s["max_q"], s["max_k"], None, 1, 2)
    o_sel = ops.topk_sparse_attention(q, k, s["v"], s["idx"], bs, cu)
    if not c["layer"]:
        return (o_cmp, o_sel, idx) + torch.autograd.grad([o_cmp, o_sel], s["leaves"], s["dy"])
    o_win = ops.sliding_window_attention(q, k, s["v"], cu, s["max_q"], c["window"])
    y = ops.gate_combine(s["gate"], o_cmp, o_sel, o_win)
    return (y, idx) + torch.autograd.grad([y], s["leaves"], s["dy"])


def _run_generate(s):
    cu, args = s["cu"], s["args"]
    outs = [nsa_infer(cu, 0, *s["prompt"], **args)]
    for i, rows in enumerate(s["steps"]):
        outs.append(s["graph"](*rows).clone() if "graph" in s else nsa_infer(cu, i + 1, *rows, **args))
    cache = args["cache"]
    return outs, [cache.sparse_kv_cache, cache.compress_kv_cache, cache.before_compress_kv_cache, cache.sliding_kv_cache,
                  cache.sparse_kv_len, cache.compress_kv_len, cache.before_compress_kv_len, cache.sliding_kv_len]


def _run_decode(s):
    c = s["c"]
    o_cmp, idx = ops.compressed_attention_decode(s["q"], s["ck"], s["cv"], s["seqlens"], s["comp_lens"], c["ks"], c["st"], c["bs"], c["topk"],
                                                 max_seqlen=c["cache"])
    o_sel = ops.topk_sparse_attention_decode(s["q"], s["k"], s["v"], s["idx"], c["bs"], s["seqlens"])
    return o_cmp, idx, o_sel, ops.flash_attention_decode(s["q"], s["k"], s["v"], s["seqlens"])


def _run_dense(s):
    o = ops.flash_attention_varlen(s["q"], s["k"], s["v"], s["cu"], s["cu"], s["longest"], s["longest"], causal=s["c"]["causal"])
    return (o,) + torch.autograd.grad([o], s["leaves"], [s["dy"]])


def _run_compress(s):
    c = s["c"]
    y, cu_y = COMPRESS[c["compress"]](s["x"], s["w"], s["cu"], c["ks"], c["st"], s["pe"])
    return (y, cu_y) + torch.autograd.grad([y], s["leaves"], [s["dy"]])


# ------------------------------------------------------------------------------------------------------------------- work
def _pairs(lens, c):
    """Visible (query, key) pairs of the compressed, the selected-block, the window and the causal branch."""
    cmp_, sel, win, dense = 0, 0, 0, 0
    bs, topk, w = c["bs"], c.get("topk", 0), c.get("window", 0)
    for n in lens:
        for t in range(n):
            cmp_ += _windows(t + 1, c)
            blocks = t // bs + 1
            sel += t + 1 if blocks <= topk else (topk - 1) * bs + t % bs + 1
        win += sum(min(t + 1, w + 1) for t in range(min(n, w + 1))) + max(0, n - w - 1) * (w + 1)
        dense += n * (n + 1) // 2 if c.get("causal", True) else n * n
    return cmp_, sel, win, dense


def work(case):
    c, lens = case, _lens(case)
    n, hq, hkv, d = sum(lens), c["hq"], c["hkv"], c["d"]
    m = sum(_windows(x, c) for x in lens)
    q, kv, ckv, gate = 2 * n * hq * d, 2 * n * hkv * d, 2 * m * hkv * d, 2 * n * hq * 3
    linear = c.get("compress") == "linear"
    weights = 2 * hkv * c["ks"] * d * (d if linear else 1) if c.get("compress") in ("linear", "weighted") else 0
    compress_flops = 2 * c["ks"] * d * (d if linear else 1) * m * hkv
    cmp_, sel, win, dense = _pairs(lens, c) if c["kind"] in ("train", "generate", "dense") else (0, 0, 0, 0)
    if c["kind"] == "train":
        flops = 3.5 * 4 * d * hq * (cmp_ + sel + (win if c["layer"] else 0)) + 3 * 2 * compress_flops
        idx = 4 * hkv * n * min(c["topk"], (max(lens) + c["bs"] - 1) // c["bs"])
        # q, k, v, the upstream gradients, the gates and the weights in; the outputs and their gradients out; the ids both ways
        rest = q * (2 + 1 + 1) if c["layer"] else q * (2 + 2 + 2)
        return {"bytes": rest + 4 * kv + 4 * weights + 2 * idx + (2 * gate if c["layer"] else 0), "flops": flops}
    if c["kind"] == "generate":
        flops = 4 * d * hq * (cmp_ + sel + win) + 2 * compress_flops
        # prefill: inputs and output once, the caches filled
        total = 2 * q + 2 * kv + gate + 2 * kv + 2 * ckv + 2 * weights
        for i in range(c["steps"]):
            for x in lens:
                t = x + i + 1
                rows = _windows(t, c) + min(t, c["topk"] * c["bs"]) + min(t, c["window"])
                total += 2 * 2 * rows * hkv * d + 2 * (2 * hq * d + 3 * hq) + 2 * 2 * 2 * hkv * d
                flops += 4 * rows * hq * d
        return {"bytes": total, "flops": flops}
    if c["kind"] == "decode":
        rows = sum(_windows(x, c) + min(x, c["topk"] * c["bs"]) + x for x in lens)
        return {"bytes": 2 * 2 * rows * hkv * d + len(lens) * 2 * 4 * hq * d, "flops": 4 * rows * hq * d}
    if c["kind"] == "dense":
        return {"bytes": 4 * q + 4 * kv, "flops": 3.5 * 4 * d * hq * dense}
    # x in twice over the two directions but for average pooling, whose gradient does not need it; dx out, y out, dy in
    return {"bytes": kv * (2 if c["compress"] == "avg" else 3) + 2 * ckv + 3 * weights, "flops": (3 if linear else 2) * compress_flops}


def tolerance(case):
    """16-bit results of fp32 sums: a few roundings of 2^-9 (bf16) or 2^-12 (fp16) between inputs and outputs.  Selected block
    ids may differ where two scores tie within the rounding of the compressed keys.  In ``generate`` such a tie moves one of
    the blocks that a row attends to, so single elements of that row may be off by as much as the output itself."""
    rel = 1e-2 if case["dtype"] == "bf16" else 2e-3
    if case["kind"] == "generate":
        return {"rel": rel, "max": 0.9}
    if case["kind"] in ("train", "decode"):
        return {"rel": rel, "differ": 5e-3}
    return {"rel": rel}
