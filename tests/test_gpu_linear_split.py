"""Linear compression whose taps are shared by the CTAs of a cluster: cluster sizes 1 to 8 (by the number of window tiles), windows
that end a tile of 64 or overrun it by one, sequences too short for a window, against the fp32 oracle."""
import pytest
import torch

from oracle import nsa_oracle as O
from tests.helpers import assert_close_16bit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,d,ks,st,lens,dtype", [
    (1, 128, 32, 16, [32], torch.bfloat16),
    (2, 128, 16, 16, [1024, 5, 1040], torch.float16),            # 64 and 65 windows
    (3, 64, 64, 32, [300, 63, 2100], torch.bfloat16),
    (8, 64, 32, 32, [33 * 64] * 9, torch.bfloat16),              # 144 tiles: clusters of four
    (8, 64, 16, 16, [1030] * 20, torch.bfloat16),                # 320: of one
    (4, 128, 32, 16, [500] * 10, torch.bfloat16),                # 40: of four
    (4, 128, 32, 16, [4144], torch.bfloat16),                    # 258 windows, 20 tiles: below the tcgen05 kernel's range
])
@pytest.mark.parametrize("with_pe", [True, False])
def test_linear_compress(H, d, ks, st, lens, dtype, with_pe):
    import native_sparse_attention_triton_b200 as pkg
    g = torch.Generator().manual_seed(H * d + ks)
    x = torch.randn(sum(lens), H, d, generator=g).to(dtype)
    w = (torch.randn(H, ks * d, d, generator=g) * (ks * d) ** -0.5).to(dtype)
    pe = (torch.randn(H, ks, d, generator=g) * 0.1).to(dtype) if with_pe else None
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
    y, ycu = pkg.ops.linear_compress(x.cuda(), w.cuda(), cu.cuda(), ks, st, None if pe is None else pe.cuda())
    ref, rcu = O.linear_compress(x.float(), w.float(), cu, ks, st, None if pe is None else pe.float())
    assert torch.equal(ycu.cpu(), rcu)
    # the window sum, the bias and their sum are each rounded to 16 bits: three errors of at most 2^-9 (bf16) of values of the
    # result's size, half of that on average, so 3 * 2^-10 bounds the mean
    assert_close_16bit(y, ref, "y", 2e-2, 3 * 2.0 ** -10)
    assert pkg.device_status() == 0
