"""nsa_decode_step_supported answers for a step's sizes without a device, so that a caller knows before its first launch."""
import pytest

from native_sparse_attention_triton_b200 import _lib

GOOD = dict(batch=4, hq=32, hkv=2, d=128, ks=32, st=16, bs=64, topk=8, init=1, local=2, sel=8320, cmp=519, win=512, dtype=0)


@pytest.mark.parametrize("change,rc", [
    ({}, 0), (dict(d=64, dtype=1), 0), (dict(batch=1, hq=16, hkv=1), 0), (dict(topk=64), 0), (dict(topk=100, sel=640), 0),
    (dict(d=96), -2), (dict(hq=34, hkv=2), -2), (dict(bs=48), -2), (dict(topk=65), -2), (dict(bs=128, topk=33), -2),
    # a cluster of eight holds 16 heads x (rows / 8) logits, and every row's and block's score, in 227 KB with its tiles
    (dict(sel=131072, cmp=8191), -2), (dict(batch=100, hkv=4, hq=64, sel=32768, cmp=2047), -2),
    (dict(hq=33), -1), (dict(topk=2), -1), (dict(batch=0), -1), (dict(st=12), -1), (dict(cmp=0), -1), (dict(win=0), -1), (dict(bs=0), -1),
])
def test_sizes(change, rc):
    c = {**GOOD, **change}
    assert _lib.lib().nsa_decode_step_supported(c["batch"], c["hq"], c["hkv"], c["d"], c["ks"], c["st"], c["bs"], c["topk"], c["init"],
                                                c["local"], c["sel"], c["cmp"], c["win"], c["dtype"]) == rc
