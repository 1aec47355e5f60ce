"""nsa_infer with one compression for the keys and another for the values: prefill and decode steps against the oracle, the fused step
against the separate operators, and the weights that a step refuses."""
import math

import pytest
import torch

from oracle import nsa_oracle as O

pytestmark = pytest.mark.gpu
HQ, HKV, D, KS, ST, BS, TOPK, W = 8, 2, 128, 32, 16, 64, 4, 64
FNS = {"linear": O.linear_compress, "weighted": O.weightedpool_compress, "avg": O.avgpool_compress}


class Session:
    """A prefilled cache and what a step takes."""

    def __init__(self, mode_k, mode_v, dtype=torch.bfloat16, lens=(30, 100), max_length=256):
        import native_sparse_attention_triton_b200 as pkg
        from native_sparse_attention_triton_b200 import infer
        from native_sparse_attention_triton_b200.kv_cache import NSACache
        self.infer, self.dtype, self.lens, self.modes = infer, dtype, list(lens), (mode_k, mode_v)
        self.g = torch.Generator().manual_seed(17)
        fns = {"linear": pkg.ops.linear_compress, "weighted": pkg.ops.weightedpool_compress, "avg": pkg.ops.avgpool_compress}
        self.w = [self.weight(m) for m in (mode_k, mode_v)]
        self.pe = self.rnd(HKV, KS, D) * 0.02
        self.inv_freq = 1.0 / (10000.0 ** (torch.arange(0, D, 2, dtype=torch.float32) / D))
        self.cu = torch.tensor([0] + torch.tensor(self.lens).cumsum(0).tolist(), dtype=torch.int32).cuda()
        self.cache = NSACache(len(lens), max_length, HKV, D, KS, ST, W, dtype)
        self.args = dict(rope=infer.RotaryEmbedding(self.inv_freq.cuda()), cache=self.cache,
                         compress_weight=tuple(None if w is None else w.cuda() for w in self.w), compress_func=(fns[mode_k], fns[mode_v]),
                         intra_block_pe=self.pe.cuda(), kernel_size=KS, kernel_stride=ST, block_size=BS, topk=TOPK, init_blocks=1,
                         local_blocks=2, window_size=W)
        n = sum(self.lens)
        self.prompt = [self.rnd(n, HQ, D), self.rnd(n, HKV, D), self.rnd(n, HKV, D), torch.rand(n, HQ, 3, generator=self.g).to(dtype)]
        self.hist = [[t[self.cu[b]:self.cu[b + 1]] for b in range(len(lens))] for t in self.prompt[1:3]]

    def rnd(self, *s):
        return torch.randn(*s, generator=self.g).to(self.dtype)

    def weight(self, mode):
        if mode == "avg":
            return None
        return self.rnd(HKV, KS * D, D) / math.sqrt(KS * D) if mode == "linear" else self.rnd(HKV, KS) / math.sqrt(KS)

    def prefill(self):
        return self.infer.nsa_infer(self.cu, 0, *[t.cuda() for t in self.prompt], **self.args)

    def rows(self):
        b = len(self.lens)
        return [self.rnd(b, HQ, D), self.rnd(b, HKV, D), self.rnd(b, HKV, D), torch.rand(b, HQ, 3, generator=self.g).to(self.dtype)]

    def check(self, out, rows):
        """The step's output for these rows, appended to the histories, against the oracle."""
        f32 = lambda t: None if t is None else t.float()
        for b in range(len(self.lens)):
            for hist, new in zip(self.hist, rows[1:3]):
                hist[b] = torch.cat([hist[b], new[b:b + 1]])
            ref = O.nsa_decode_token(f32(rows[0][b]), f32(self.hist[0][b]), f32(self.hist[1][b]), f32(rows[3][b]), self.inv_freq,
                                     FNS[self.modes[0]], FNS[self.modes[1]], f32(self.w[0]), f32(self.w[1]), f32(self.pe), KS, ST, BS, TOPK,
                                     1, 2, W)
            err = (out[b].float().cpu() - ref).abs() / ref.abs().clamp(min=1.0)
            # the sum of three branches, each within the single-operator tolerance and of 16-bit rotated rows
            assert float(err.max()) <= 4e-2 and float(err.mean()) <= 3e-3, (b, float(err.max()), float(err.mean()))


@pytest.mark.parametrize("mode_k,mode_v", [("weighted", "avg"), ("avg", "weighted"), ("linear", "avg"), ("weighted", "linear")])
def test_generation(mode_k, mode_v):
    import native_sparse_attention_triton_b200 as pkg
    s = Session(mode_k, mode_v)
    s.prefill()
    for step in range(1, 21):
        rows = s.rows()
        s.check(s.infer.nsa_infer(s.cu, step, *[t.cuda() for t in rows], **s.args), rows)
    assert pkg.device_status() == 0


@pytest.mark.parametrize("mode_k,mode_v", [("weighted", "avg"), ("avg", "weighted")])
def test_fused_step_equals_operators(monkeypatch, mode_k, mode_v):
    a, b = Session(mode_k, mode_v), Session(mode_k, mode_v)
    a.prefill(), b.prefill()
    fused = a.infer._fused_decode_step
    taken = []
    monkeypatch.setattr(a.infer, "_fused_decode_step", lambda *x: taken.append(fused(*x)) or taken[-1])
    for step in range(1, 21):
        rows = [t.cuda() for t in a.rows()]
        one = a.infer.nsa_infer(a.cu, step, *rows, **a.args)
        with monkeypatch.context() as m:
            m.setattr(b.infer, "_fused_decode_step", lambda *x: None)
            two = b.infer.nsa_infer(b.cu, step, *rows, **b.args)
        assert taken[-1] is one
        err = (one.float() - two.float()).abs() / two.float().abs().clamp(min=1.0)
        assert float(err.max()) <= 4e-2 and float(err.mean()) <= 4e-3
    for x, y in zip(a.cache._tensors(), b.cache._tensors()):
        assert x.dtype != torch.int32 or torch.equal(x, y)
    # the same fp32 sums, rounded twice: an ulp or two of values around 1
    assert float((a.cache.compress_kv_cache.float() - b.cache.compress_kv_cache.float()).abs().max()) <= 4e-2


@pytest.mark.parametrize("mode_k,mode_v,which", [("weighted", "avg", 0), ("avg", "weighted", 1), ("weighted", "weighted", 1), ("linear", "linear", 1)])
def test_weights_are_checked_on_their_own_side(mode_k, mode_v, which):
    s = Session(mode_k, mode_v)
    s.prefill()
    rows = [t.cuda() for t in s.rows()]
    before = [t.clone() for t in s.cache._tensors()]
    w = s.args["compress_weight"][which]
    for bad, error in ((w.float(), AssertionError), (w.half(), AssertionError), (w[:1], AssertionError), (None, AssertionError), (w.cpu(), RuntimeError)):
        given = list(s.args["compress_weight"])
        given[which] = bad
        with pytest.raises(error):
            s.infer.nsa_infer(s.cu, 1, *rows, **{**s.args, "compress_weight": tuple(given)})
    for x, y in zip(s.cache._tensors(), before):
        assert torch.equal(x, y)


@pytest.mark.parametrize("mode_k,mode_v,which", [("avg", "avg", 0), ("weighted", "avg", 1)])
def test_prefill_refuses_weights_for_average_pooling(mode_k, mode_v, which):
    s = Session(mode_k, mode_v)
    given = list(s.args["compress_weight"])
    given[which] = torch.ones(HKV, KS, dtype=s.dtype, device="cuda")
    with pytest.raises(AssertionError):
        s.infer.nsa_infer(s.cu, 0, *[t.cuda() for t in s.prompt], **{**s.args, "compress_weight": tuple(given)})


@pytest.fixture
def no_host_copies():
    """Every synchronising copy raises."""
    torch.cuda.synchronize()
    yield lambda: torch.cuda.set_sync_debug_mode("error")
    torch.cuda.set_sync_debug_mode("default")


def test_a_step_of_separate_operators_reads_nothing_on_the_host(no_host_copies):
    """A mixture of linear and pooling, in inference mode, where tensors carry no version counter and nothing can be remembered by."""
    with torch.inference_mode():
        s = Session("linear", "avg")
        s.prefill()
        for step in range(1, 4):
            rows = s.rows()
            gpu = [t.cuda() for t in rows]
            no_host_copies()
            out = s.infer.nsa_infer(s.cu, step, *gpu, **s.args)
            torch.cuda.set_sync_debug_mode("default")
            s.check(out, rows)


def test_a_first_step_can_be_captured():
    """No step of this cache has run before the capture, and 80 other cu_seqlens come by before the replays, which cross the end of a
    compression window."""
    import native_sparse_attention_triton_b200 as pkg
    warm = Session("linear", "avg")          # the library's one-time initialisation
    warm.prefill()
    warm.infer.nsa_infer(warm.cu, 1, *[t.cuda() for t in warm.rows()], **warm.args)
    s = Session("linear", "avg")
    s.prefill()
    fixed = [t.cuda() for t in s.rows()]
    state = [t.clone() for t in s.cache._tensors()]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = s.infer.nsa_infer(s.cu, 1, *fixed, **s.args)
    for dst, src in zip(s.cache._tensors(), state):
        dst.copy_(src)
    keep = []
    for n in range(80):
        keep.append(torch.tensor([0, 33 + n], dtype=torch.int32).cuda())
        pkg.ops.avgpool_compress(torch.zeros(33 + n, 1, 64, device="cuda").bfloat16(), None, keep[-1], KS, ST, None)
    junk = [torch.full((3,), 1 << 20, dtype=torch.int32, device="cuda") for _ in range(200)]
    for _ in range(20):
        rows = s.rows()
        for dst, src in zip(fixed, rows):
            dst.copy_(src)
        graph.replay()
        s.check(out, rows)
    assert len(junk) == 200 and pkg.device_status() == 0


def launches(run):
    """Names of the library's launches during run()."""
    import ctypes

    from native_sparse_attention_triton_b200 import _lib
    lib = _lib.lib()
    lib.nsa_profile_enable(1)
    try:
        run()
        buf = ctypes.create_string_buffer(1 << 16)
        assert lib.nsa_profile_collect(buf, len(buf)) >= 0
    finally:
        lib.nsa_profile_enable(0)
    return buf.value.decode()


def test_a_refused_shape_costs_no_launch():
    """A compressed cache whose scores do not fit into a cluster's shared memory: the step takes the operators, and the taps of the
    fused step's linear compression are not launched for nothing."""
    import native_sparse_attention_triton_b200 as pkg
    s = Session("linear", "linear", max_length=70000)
    assert pkg._lib.lib().nsa_decode_step_supported(2, HQ, HKV, D, KS, ST, BS, TOPK, 1, 2, 70000, s.cache.max_comp_length, W, 0) == 0
    big = Session("linear", "linear", lens=(40,), max_length=400000)
    assert pkg._lib.lib().nsa_decode_step_supported(1, HQ, HKV, D, KS, ST, BS, TOPK, 1, 2, 400000, big.cache.max_comp_length, W, 0) == -2
    s.prefill()
    rows = [t.cuda() for t in s.rows()]
    names = launches(lambda: s.infer.nsa_infer(s.cu, 1, *rows, **s.args))
    assert "linear_taps" in names and "decode_step" in names
    big.prefill()
    rows = [t.cuda() for t in big.rows()]
    names = launches(lambda: big.infer._fused_decode_step(big.cache, *rows, big.args["rope"], big.args["compress_weight"],
                                                          big.args["compress_func"], big.args["intra_block_pe"], BS, TOPK, 1, 2))
    assert "linear_taps" not in names and "decode" not in names, names


def test_a_graph_whose_cache_no_longer_fits_says_so():
    s = Session("weighted", "avg")
    s.prefill()
    rows = [t.cuda() for t in s.rows()]
    graph = s.infer.DecodeGraph(s.cu, *rows, **s.args)
    assert graph.graph is None
    graph(*rows)
    s.cache.update_kv = lambda *a, **k: None
    with pytest.raises(RuntimeError):
        graph(*rows)


def test_captured_graphs_replay():
    """A step of separate operators, captured: two graphs alive on two sessions replay over the end of a compression window and give the
    bits of eager steps from the same state; making a graph leaves the state as it was."""
    import native_sparse_attention_triton_b200 as pkg
    pairs, graphs = [(Session("linear", "avg"), Session("linear", "avg")), (Session("weighted", "linear"), Session("weighted", "linear"))], []
    for a, b in pairs:
        assert torch.equal(a.prefill(), b.prefill())
        rows = [t.cuda() for t in a.rows()]
        b.rows()
        before = [t.clone() for t in a.infer.DecodeGraph._state(a.cache)]
        graphs.append(a.infer.DecodeGraph(a.cu, *rows, **a.args))
        assert graphs[-1].graph is not None
        for x, y in zip(a.infer.DecodeGraph._state(a.cache), before):
            assert torch.equal(x, y)
    for step in range(1, 25):
        for (a, b), graph in zip(pairs, graphs):
            rows = a.rows()
            gpu = [t.cuda() for t in rows]
            out = graph(*gpu)
            assert torch.equal(out, b.infer.nsa_infer(b.cu, step, *gpu, **b.args)), step
            a.check(out, rows)
    for a, b in pairs:
        for x, y in zip(a.cache._tensors(), b.cache._tensors()):
            assert torch.equal(x, y)
    assert pkg.device_status() == 0
