"""Scratch of the split-KV decode kernel: captured graphs keep working whatever other calls on their stream do with the buffer that
eager calls share, and the cluster kernels take none."""
import pytest
import torch

from oracle import nsa_oracle as O

pytestmark = pytest.mark.gpu
KS, ST, BS, TOPK = 32, 16, 64, 4


def inputs(B, Hkv, G, d, L, seed):
    g = torch.Generator().manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g).bfloat16().cuda()
    lens = torch.randint(1, L + 1, (B,), generator=g).int()
    Lc = (L - KS) // ST + 1
    clens = torch.clamp((lens - KS) // ST + 1, min=0).int()
    return rnd(B, Hkv * G, d), rnd(B, L, Hkv, d), rnd(B, L, Hkv, d), rnd(B, Lc, Hkv, d), rnd(B, Lc, Hkv, d), lens.cuda(), clens.cuda()


def both(ops, q, k, v, ck, cv, lens, clens):
    o, idx = ops.compressed_attention_decode(q, ck, cv, lens, clens, KS, ST, BS, TOPK, max_seqlen=k.shape[1])
    return o, idx, ops.flash_attention_decode(q, k, v, lens)


def test_replays_after_the_streams_buffer_was_regrown_dirtied_and_given_back():
    import native_sparse_attention_triton_b200 as pkg
    run = lambda x: both(pkg.ops, *x)
    # 450 pairs: compressed attention on the split-KV kernel; 124 pairs of long rows: dense attention too
    cases = [inputs(150, 3, 2, 64, 200, 1), inputs(31, 4, 4, 128, 4200, 2)]
    bigger, smaller = inputs(300, 4, 2, 128, 300, 3), inputs(230, 2, 2, 64, 100, 4)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graphs = []
    with torch.cuda.stream(stream):
        want = [[t.clone() for t in run(x)] for x in cases]
    torch.cuda.synchronize()
    for x in cases:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out = run(x)
        graphs.append((graph, out))
    for again in range(3):
        with torch.cuda.stream(stream):
            run((bigger, smaller, cases[0])[again])
            for i in range(70):                       # every stream's buffer given back
                other = torch.cuda.Stream()
                with torch.cuda.stream(other):
                    run(smaller)
                other.synchronize()
            junk = [torch.full((n,), 3.0, device="cuda") for n in (1 << 12, 1 << 16, 1 << 20, 1 << 22)]
            for (graph, out), w in zip(graphs, want):
                for t in out:
                    t.fill_(1)
                graph.replay()
                for a, b in zip(out, w):
                    assert torch.equal(a, b), again
        torch.cuda.synchronize()
        del junk
    x = cases[0]
    ref = O.flash_attention_decode(x[0].float(), x[1].float(), x[2].float(), x[5])
    assert float((want[0][2].float() - ref).abs().max()) <= 2e-2 * float(ref.abs().max().clamp(min=1.0))
    assert pkg.device_status() == 0


def test_cluster_kernels_take_no_scratch():
    import native_sparse_attention_triton_b200 as pkg
    x = inputs(4, 2, 16, 128, 2000, 5)
    both(pkg.ops, *x)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    with torch.cuda.stream(torch.cuda.Stream()):   # a stream that has no buffer yet
        out = both(pkg.ops, *x)
        torch.cuda.synchronize()
    kept = sum((t.numel() * t.element_size() + 511) // 512 * 512 for t in out)
    assert torch.cuda.memory_allocated() - before <= kept
