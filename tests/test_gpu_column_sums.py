"""Column sums of the output gradient in the backward of compression with a position embedding: a cluster of eight CTAs shares the
rows, so that with fewer than eight rows some have none, and 512 rows are one round of the loads in flight.  Small whole numbers, whose
sums and quotients by the kernel size are exact in fp16."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 6, 7, 8, 9, 63, 65, 511, 512, 513, 1537])
@pytest.mark.parametrize("H,d", [(1, 64), (3, 128)])
def test_position_embedding_gradient_is_the_column_sum(rows, H, d):
    import native_sparse_attention_triton_b200 as pkg
    ks = st = 32
    g = torch.Generator().manual_seed(rows)
    n = rows * st + 5
    x, pe = torch.randn(n, H, d, generator=g).half().cuda(), torch.zeros(H, ks, d).half().cuda().requires_grad_(True)
    dy = torch.randint(-1, 2, (rows, H, d), generator=g).half().cuda()
    y, _ = pkg.ops.avgpool_compress(x, None, torch.tensor([0, n], dtype=torch.int32).cuda(), ks, st, pe)
    for _ in range(3):
        dpe, = torch.autograd.grad(y, pe, dy, retain_graph=True)
        assert torch.equal(dpe.float(), (dy.float().sum(0) / ks)[:, None].expand(H, ks, d))
    assert pkg.device_status() == 0


@pytest.mark.parametrize("mode", ["linear", "weighted", "avg"])
def test_gradient_at_an_odd_offset(mode):
    import native_sparse_attention_triton_b200 as pkg
    H, d, ks, st, n = 2, 128, 32, 16, 500
    g = torch.Generator().manual_seed(1)
    rnd = lambda *s: torch.randn(*s, generator=g).bfloat16().cuda().requires_grad_(True)
    fn = {"linear": pkg.ops.linear_compress, "weighted": pkg.ops.weightedpool_compress, "avg": pkg.ops.avgpool_compress}[mode]
    x, pe = rnd(n, H, d), rnd(H, ks, d)
    w = {"linear": lambda: rnd(H, ks * d, d), "weighted": lambda: rnd(H, ks), "avg": lambda: None}[mode]()
    leaves = [t for t in (x, w, pe) if t is not None]
    y, _ = fn(x, w, torch.tensor([0, n], dtype=torch.int32).cuda(), ks, st, pe)
    flat = torch.randn(y.numel() + 1, generator=g).bfloat16().cuda()
    odd = flat[1:].view_as(y)
    assert odd.data_ptr() % 16 and odd.is_contiguous()
    for a, b in zip(torch.autograd.grad(y, leaves, odd, retain_graph=True), torch.autograd.grad(y, leaves, odd.clone())):
        assert torch.equal(a, b)
