"""Which caches the fused prefill and decode step take over the bookkeeping of."""
import types

import torch

from native_sparse_attention_triton_b200 import infer
from native_sparse_attention_triton_b200.kv_cache import NSACache


def cache(cls=NSACache):
    return cls(1, 64, 1, 64, 32, 16, 16, torch.bfloat16, "cpu")


def test_only_caches_with_their_own_bookkeeping_are_plain(monkeypatch):
    assert infer._is_plain(cache())

    class Named(NSACache):
        pass

    class Counting(NSACache):
        def update_kv(self, *args, **kwargs):
            return super().update_kv(*args, **kwargs)

    assert infer._is_plain(cache(Named)) and not infer._is_plain(cache(Counting))
    assert not infer._is_plain(types.SimpleNamespace(prepare_compress=None, update_kv=None, _fill=None))
    for name in ("prepare_compress", "update_kv", "_fill"):
        replaced, bound = cache(), cache()
        setattr(replaced, name, lambda *args, **kwargs: None)
        setattr(bound, name, types.MethodType(lambda self, *args, **kwargs: None, bound))
        assert not infer._is_plain(replaced) and not infer._is_plain(bound)
        with monkeypatch.context() as m:
            m.setattr(NSACache, name, lambda self, *args, **kwargs: None)
            assert not infer._is_plain(cache())
    assert infer._is_plain(cache())
