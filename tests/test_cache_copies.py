"""The native calls' record of a cache's storage holds addresses: it belongs to the cache it was made for."""
import copy
import io
import os
import pickle

import pytest
import torch


from flashquest_b200 import build

pytestmark = pytest.mark.skipif(not os.path.exists(build.BIND), reason="library not built (python -m flashquest_b200.build)")


def _cache(bits, device="cpu"):
    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    from flashquest_b200.cache.persistent_turbo import PersistentTurboKVCache
    return {3: PersistentTurboKVCache, 4: PersistentInt4KVCache, 8: PersistentInt8KVCache}[bits](
        batch_size=1, num_layers=2, num_kv_heads=2, head_dim=64, max_seq_len=64, page_size=16, dtype=torch.float16, device=device)


def _saved(cache):
    f = io.BytesIO()
    torch.save(cache, f)
    f.seek(0)
    return torch.load(f, weights_only=False)


def _addresses(cache):
    return {getattr(cache.desc(), name) for name, kind in cache.desc()._fields_ if getattr(kind, "__name__", "") == "c_void_p"}


@pytest.mark.parametrize("bits", [3, 4, 8])
@pytest.mark.parametrize("how", [copy.deepcopy, _saved, lambda c: pickle.loads(pickle.dumps(c))], ids=["deepcopy", "save", "pickle"])
def test_copies_have_a_record_of_their_own(bits, how):
    cache = _cache(bits)
    cache.desc()                                     # as after the first append
    cache._fq_engines = {"step": object()}
    other = how(cache)
    assert not hasattr(other, "_fq_engines") and hasattr(cache, "_fq_engines")
    assert not (_addresses(cache) & _addresses(other))
    assert other.K_partial.shape == cache.K_partial.shape and other._seen_tokens == cache._seen_tokens


@pytest.mark.parametrize("bits", [3, 4, 8])
def test_record_follows_replaced_storage(bits):
    cache = _cache(bits)
    names = [n for n, t in vars(cache).items() if torch.is_tensor(t)]
    keep = []
    for name in names:                               # one at a time: every address counts
        before = cache.desc()
        keep.append(getattr(cache, name))
        setattr(cache, name, keep[-1].clone())
        assert cache.desc() is not before and getattr(cache, name).data_ptr() in _addresses(cache)
        assert keep[-1].data_ptr() not in _addresses(cache)
        assert cache.desc() is cache.desc()
