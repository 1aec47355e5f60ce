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


def _pool_pass(lens, mode, g, H=4, d=128, ks=32, st=16):
    import native_sparse_attention_triton_b200 as pkg
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32).cuda()
    x, w = torch.randn(sum(lens), H, d, generator=g).half().cuda(), (torch.rand(H, ks, generator=g) / ks).half().cuda()
    pe = torch.zeros(H, ks, d).half().cuda()
    leaves = [t.requires_grad_(True) for t in ((x, w, pe) if mode == "weighted" else (x, pe))]
    y, cu_y = (pkg.ops.weightedpool_compress if mode == "weighted" else pkg.ops.avgpool_compress)(x, w if mode == "weighted" else None, cu, ks, st, pe)
    return leaves, y, cu, cu_y, torch.randint(-1, 2, y.shape, generator=g).half().cuda()


# 131 072 tokens or more: the streaming pass.  In it the columns are summed beside the rest while there are few CTAs, here up to one for 32
# chunks of 16 tokens (256 sequences of 512 tokens are at that edge), else by a kernel of their own
@pytest.mark.parametrize("lens,apart", [([140000], False), ([512] * 256, False), ([496] * 272, True), ([64] * 2048, True), ([100000] + [61] * 1000, True)])
@pytest.mark.parametrize("mode", ["weighted", "avg"])
def test_column_sums_of_many_sequences(lens, apart, mode):
    import native_sparse_attention_triton_b200 as pkg
    leaves, y, cu, cu_y, dy = _pool_pass(lens, mode, torch.Generator().manual_seed(len(lens)))
    pkg._lib.profile(True)
    try:
        grads = torch.autograd.grad(y, leaves, dy)
        names = set(pkg._lib.profile_collect())
    finally:
        pkg._lib.profile(False)
    assert any(n.startswith("pool_dx") for n in names) and "pool_dw_finish" in names and ("colsum" in names) == apart, names
    weight = leaves[1].detach().double() if mode == "weighted" else torch.full((4, 32), 1 / 32, dtype=torch.float64, device="cuda")
    dpe = weight[:, :, None] * dy.double().sum(0)[:, None]    # whole sums: exact until they are rounded once, to 2^-11
    assert ((grads[-1].double() - dpe).abs() <= 2.0 ** -11 * dpe.abs() + 2.0 ** -25).all()
    if mode == "weighted":   # dw[h, i] = sum over windows of <dy, x row i + pe row i>, and pe is zero
        dw, x = torch.zeros(4, 32, dtype=torch.float64, device="cuda"), leaves[0].detach()
        starts = torch.repeat_interleave((cu[:-1].long() - 16 * cu_y[:-1].long()), (cu_y[1:] - cu_y[:-1]).long()) + 16 * torch.arange(len(y), device="cuda")
        for i in range(32):
            dw[:, i] = (dy.double() * x[starts + i].double()).sum((0, 2))
        assert (grads[1].double() - dw).norm() <= 2 * 2.0 ** -11 * dw.norm()    # fp32 sums, rounded once to fp16
    assert pkg.device_status() == 0


@pytest.mark.parametrize("mode", ["weighted", "avg"])
def test_a_workspace_of_the_column_sums_alone(mode):
    """The C interface takes a workspace without room for partial rows: weighted pooling then runs on the per-thread kernels, average
    pooling still on the streaming pass."""
    import native_sparse_attention_triton_b200 as pkg
    H, d, ks, st = 4, 128, 32, 16
    leaves, y, cu, cu_y, dy = _pool_pass([131072 + 7, 300], mode, torch.Generator().manual_seed(3))
    want = torch.autograd.grad(y, leaves, dy)
    x, pe, w = leaves[0].detach(), leaves[-1].detach(), leaves[1].detach() if mode == "weighted" else None
    got, ws = [torch.empty_like(t) for t in leaves], torch.empty(H * d, device="cuda")
    p = lambda t: None if t is None else t.data_ptr()
    pkg._lib.profile(True)
    try:
        rc = pkg._lib.lib().nsa_pool_compress_bwd(p(x), p(w), p(pe), p(dy), p(cu), p(cu_y), p(got[0]), p(got[1]) if w is not None else None,
                                                  p(got[-1]), p(ws), ws.numel(), x.shape[0], 2, y.shape[0], 131079, H, d, ks, st, H * d, d, 1,
                                                  torch.cuda.current_stream().cuda_stream)
        names = set(pkg._lib.profile_collect())
    finally:
        pkg._lib.profile(False)
    assert rc == 0 and "colsum" in names and ("pool_dw_finish" in names) == (mode == "avg"), names
    # the same sums in another order, rounded once: at most the next fp16 number
    for a, b in zip(got, want):
        assert ((a.float() - b.float()).abs() <= 2.0 ** -10 * b.float().abs() + 2.0 ** -24).all()
    assert pkg.device_status() == 0
