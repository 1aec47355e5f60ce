"""The decode entry points refuse, on the host, addresses and strides that their 16-byte copies cannot serve.  The addresses are made
up: no call may get as far as the device (without one a launch would answer with a CUDA error, 1000 and above)."""
import pytest

from native_sparse_attention_triton_b200 import _lib

BASE, INVALID = 1 << 20, -1
B, L, HQ, HKV, D = 2, 256, 8, 2, 128


def call(entry, ptrs, strides, batch=B, cache_len=L):
    lib, s = _lib.lib(), _lib.strides_array(*strides)
    q, k, v, o = ptrs
    ids = BASE + (1 << 30)
    if entry == "dense":
        return lib.nsa_flash_attn_decode(q, k, v, ids, o, None, 0, 1, batch, cache_len, HQ, HKV, D, s, 0.1, 0, None)
    if entry == "selected":
        return lib.nsa_topk_sparse_attn_decode(q, k, v, ids, ids, o, None, 0, 1, batch, cache_len, HQ, HKV, D, 4, 64, s, 0.1, 0, None)
    return lib.nsa_compressed_attn_decode(q, k, v, ids, ids, o, ids, None, 0, 1, batch, cache_len, 4096, HQ, HKV, D, 32, 16, 64, 4, 1, 2, s,
                                          0.1, 0, None)


@pytest.mark.parametrize("entry", ["dense", "selected", "compressed"])
@pytest.mark.parametrize("which", range(4))
@pytest.mark.parametrize("off", [2, 8, 14])
def test_misaligned_base_is_refused(entry, which, off):
    strides = [HQ * D, D] + [L * HKV * D, HKV * D, D] * 2 + [HQ * D, D, 8, 4, 1]
    ptrs = [BASE * (i + 1) for i in range(4)]
    ptrs[which] += off
    assert call(entry, ptrs, strides) == INVALID
    assert call(entry, ptrs, strides, batch=500) == INVALID              # the ranges of the split-KV kernel
    assert call(entry, ptrs, strides, batch=70, cache_len=8192) == INVALID


@pytest.mark.parametrize("entry", ["dense", "selected", "compressed"])
@pytest.mark.parametrize("which", range(10))
def test_odd_strides_are_refused(entry, which):
    strides = [HQ * D, D] + [L * HKV * D, HKV * D, D] * 2 + [HQ * D, D, 8, 4, 1]
    strides[which] += 4
    assert call(entry, [BASE * (i + 1) for i in range(4)], strides) == INVALID
