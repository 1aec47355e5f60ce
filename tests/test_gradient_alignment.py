"""The backward entry points refuse, on the host, addresses that their 16-byte accesses cannot serve.  The addresses are made up: no
call may get as far as the device."""
import pytest

from native_sparse_attention_triton_b200 import _lib

BASE, INVALID = 1 << 20, -1


@pytest.mark.parametrize("off", [2, 8, 14])
@pytest.mark.parametrize("linear", [True, False])
def test_misaligned_gradient_of_a_compression_is_refused(linear, off):
    lib = _lib.lib()
    x, w, pe, dy, cu, ycu, dx, dw, dpe, ws = [BASE * (i + 1) for i in range(10)]
    N, B, Y, H, D, ks, st = 320, 1, 19, 2, 128, 32, 16
    if linear:
        rc = lib.nsa_linear_compress_bwd(x, w, pe, dy + off, cu, ycu, dx, dw, dpe, ws, N, B, Y, N, H, D, ks, st, H * D, D, 0, None)
    else:
        rc = lib.nsa_pool_compress_bwd(x, w, pe, dy + off, cu, ycu, dx, dw, dpe, ws, 1 << 20, N, B, Y, N, H, D, ks, st, H * D, D, 0, None)
    assert rc == INVALID


@pytest.mark.parametrize("which", range(8))
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("entry", ["varlen", "window", "selected"])
def test_misaligned_rows_of_an_attention_are_refused(entry, d, which):
    lib = _lib.lib()
    q, k, v, o, do, dq, dk, dv = [BASE * (i + 1) + (8 if i == which else 0) for i in range(8)]
    lse, cu, ids, ws, big = BASE << 5, BASE << 6, BASE << 7, BASE << 8, 1 << 40
    N, B, Hq, Hkv = 320, 1, 8, 2
    rows, kv = [Hq * d, d], [Hkv * d, d]
    s = _lib.strides_array(*rows, *kv, *kv, *rows, *rows, *rows, *kv, *kv, N * 4, 4, 1)
    if entry == "varlen":
        rc = lib.nsa_varlen_attn_bwd(q, k, v, o, do, lse, cu, cu, dq, dk, dv, ws, big, N, N, B, N, N, Hq, Hkv, d, 1, 1, 1, s, 0.1, 0, None)
    elif entry == "window":
        rc = lib.nsa_window_attn_bwd(q, k, v, o, do, lse, cu, dq, dk, dv, ws, big, N, B, N, Hq, Hkv, d, 64, s, 0.1, 0, None)
    else:
        rc = lib.nsa_topk_sparse_attn_bwd(q, k, v, o, do, lse, ids, cu, None, dq, dk, dv, ws, big, N, B, Hq, Hkv, d, 4, 64, s, 0.1, 0, None)
    assert rc == INVALID
