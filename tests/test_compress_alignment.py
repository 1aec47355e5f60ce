"""The compression backward refuses, on the host, a gradient address that its 16-byte reads cannot serve.  The addresses are made up: no
call may get as far as the device."""
import pytest

from native_sparse_attention_triton_b200 import _lib

BASE, INVALID = 1 << 20, -1


@pytest.mark.parametrize("off", [2, 8, 14])
@pytest.mark.parametrize("linear", [True, False])
def test_misaligned_gradient_is_refused(linear, off):
    lib = _lib.lib()
    x, w, pe, dy, cu, ycu, dx, dw, dpe, ws = [BASE * (i + 1) for i in range(10)]
    N, B, Y, H, D, ks, st = 320, 1, 19, 2, 128, 32, 16
    if linear:
        rc = lib.nsa_linear_compress_bwd(x, w, pe, dy + off, cu, ycu, dx, dw, dpe, ws, N, B, Y, N, H, D, ks, st, H * D, D, 0, None)
    else:
        rc = lib.nsa_pool_compress_bwd(x, w, pe, dy + off, cu, ycu, dx, dw, dpe, ws, 1 << 20, N, B, Y, N, H, D, ks, st, H * D, D, 0, None)
    assert rc == INVALID
