"""The caches refuse K and V that a launch would read past, or write past its storage for, before anything is launched."""
import pytest
import torch


@pytest.mark.parametrize("bits", [3, 4, 8])
@pytest.mark.parametrize("page", [8, 16])
@pytest.mark.parametrize("k,v", [((2, 4, 5, 64), (2, 4, 5, 64)), ((3, 3, 5, 64), (3, 3, 5, 64)), ((2, 3, 5, 128), (2, 3, 5, 128)),
                                 ((2, 3, 5, 32), (2, 3, 5, 32)), ((2, 3, 5, 64), (2, 3, 4, 64)), ((2, 3, 5, 64), (1, 3, 5, 64))])
def test_wrong_shapes_are_refused(bits, page, k, v):
    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    from flashquest_b200.cache.persistent_turbo import PersistentTurboKVCache
    cache = {3: PersistentTurboKVCache, 4: PersistentInt4KVCache, 8: PersistentInt8KVCache}[bits](
        batch_size=2, num_layers=1, num_kv_heads=3, head_dim=64, max_seq_len=64, page_size=page, dtype=torch.float16, device="cpu")
    with pytest.raises((ValueError, RuntimeError), match="K_new and V_new must be"):
        cache.update_quantized(torch.zeros(k, dtype=torch.float16), torch.zeros(v, dtype=torch.float16), 0)
    assert cache.get_seq_length() == 0


@pytest.mark.parametrize("shape", [(2, 1, 5, 64), (1, 3, 5, 64)])
def test_int8_takes_no_fewer_heads_or_sequences(shape):
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    cache = PersistentInt8KVCache(batch_size=2, num_layers=1, num_kv_heads=3, head_dim=64, max_seq_len=64, page_size=16, dtype=torch.float16, device="cpu")
    x = torch.zeros(shape, dtype=torch.float16)
    with pytest.raises(RuntimeError, match="K_new and V_new must be"):
        cache.update_quantized(x, x, 0)
