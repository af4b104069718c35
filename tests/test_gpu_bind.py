"""The CPython module over the C ABI (csrc/fq_bind.cpp) as a host program meets it: threads and streams."""
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

B, HQ, HKV, D, PAGE = 1, 4, 2, 64, 16


def _engine(layers=1):
    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.eager.decode_step import QuestDecodeInt4
    cache = PersistentInt4KVCache(batch_size=B, num_layers=layers, num_kv_heads=HKV, head_dim=D, max_seq_len=128, page_size=PAGE, dtype=torch.float16)
    g = torch.Generator(device="cuda").manual_seed(5)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).half()
    for layer in range(layers):
        cache.update_quantized(r(B, HKV, 70, D), r(B, HKV, 70, D), layer)
    return cache, QuestDecodeInt4(cache, num_q_heads=HQ, retention=0.5, num_sinks=1, window_pages=1, q_dtype=torch.float16), r


@pytest.mark.parametrize("call", ["step", "forward", "append"])
def test_other_threads_run_while_the_launch_queue_is_full(call):
    cache, engine, r = _engine()
    k, v, q = r(B, HKV, 1, D), r(B, HKV, 1, D), r(B, HQ, 1, D)
    flat = lambda t: t.view(B, 1, -1)
    cos, sin = r(1, 1, D), r(1, 1, D)
    run = {"step": lambda: engine.step(k, v, q, 0), "append": lambda: cache.update_quantized(k, v, 0),
           "forward": lambda: engine.forward_token(flat(q), flat(k), flat(v), cos, sin, 0)}[call]

    def repeat(n):
        for _ in range(n):
            cache._seen_tokens[0] = 70
            run()
    repeat(3)
    torch.cuda.synchronize()
    stop, gaps = threading.Event(), []

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now
    thread = threading.Thread(target=tick)
    thread.start()
    torch.cuda._sleep(int(0.5 * 1.9e9))                     # about half a second in front of the launches
    began = time.perf_counter()
    repeat(3000 if call == "append" else 800)
    took = time.perf_counter() - began
    stop.set()
    thread.join()
    torch.cuda.synchronize()
    assert took > 0.3, "the launch queue did not fill: nothing was tested"
    assert max(gaps) < 0.1, max(gaps)


def _restride(t, axis, by):
    """The same tensor with another stride on an axis of length 1."""
    assert t.shape[axis] == 1
    strides = list(t.stride())
    strides[axis] += by
    return t.as_strided(t.shape, strides)


@pytest.mark.parametrize("kind,Hq,Hkv", [(4, 4, 2), (3, 4, 2), (8, 4, 2), (3, 1, 1), (4, 1, 1)])
def test_strides_of_axes_of_length_one_do_not_matter(kind, Hq, Hkv):
    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    from flashquest_b200.cache.persistent_turbo import PersistentTurboKVCache
    from flashquest_b200.eager.decode_step import QuestDecodeInt4, QuestDecodeInt8, QuestDecodeTurbo
    cls, eng = {3: (PersistentTurboKVCache, QuestDecodeTurbo), 4: (PersistentInt4KVCache, QuestDecodeInt4), 8: (PersistentInt8KVCache, QuestDecodeInt8)}[kind]
    g = torch.Generator(device="cuda").manual_seed(6)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).half()
    cache = cls(batch_size=1, num_layers=1, num_kv_heads=Hkv, head_dim=64, max_seq_len=128, page_size=16, dtype=torch.float16)
    cache.update_quantized(r(1, Hkv, 70, 64), r(1, Hkv, 70, 64), 0)
    engine = eng(cache, num_q_heads=Hq, retention=0.5, num_sinks=1, window_pages=1, q_dtype=torch.float16)
    k, v, q = r(1, Hkv, 1, 64), r(1, Hkv, 1, 64), r(1, Hq, 1, 64)
    want = [t.clone() for t in engine.step(k, v, q, 0)]
    odd = [_restride(_restride(t, 0, by), 2, by) for t, by in ((k, 8), (v, 24), (q, 40))]
    if Hq == 1:
        odd = [_restride(t, 1, 16) for t in odd]
    cache._seen_tokens[0] = 70
    assert all(torch.equal(a, b) for a, b in zip(want, engine.step(*odd, 0)))


@pytest.mark.parametrize("form", ["dense", "rows"])
@pytest.mark.parametrize("n", [1, 37])
def test_int8_takes_rows_off_a_16_byte_boundary(form, n):
    """As its torch.cat form did: a dense tensor two bytes off, and rows of D + 1 values."""
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    from flashquest_b200.eager.decode_step import QuestDecodeInt8
    g = torch.Generator(device="cuda").manual_seed(9)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).half()

    def off(t):
        if form == "dense":
            out = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape)
        else:
            out = torch.empty(*t.shape[:-1], t.shape[-1] + 1, dtype=t.dtype, device="cuda")[..., :-1]
        return out.copy_(t)
    k0, v0, k, v, q = r(2, 2, 30, 64), r(2, 2, 30, 64), r(2, 2, n, 64), r(2, 2, n, 64), r(2, 4, 1, 64)
    results = []
    for f in (lambda t: t, off):
        cache = PersistentInt8KVCache(batch_size=2, num_layers=1, num_kv_heads=2, head_dim=64, max_seq_len=128, page_size=16, dtype=torch.float16)
        engine = QuestDecodeInt8(cache, num_q_heads=4, retention=0.5, num_sinks=1, window_pages=1, q_dtype=torch.float16)
        cache.update_quantized(f(k0), f(v0), 0)
        out = [t.clone() for t in engine.step(f(k), f(v), q, 0)]
        results.append(out + [t.clone() for t in cache.get_views(0).values() if torch.is_tensor(t)])
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("kind", [3, 4, 8])
def test_layers_of_one_cache_on_two_streams(kind):
    """Every buffer between the launches of a token has a part for each layer."""
    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    from flashquest_b200.cache.persistent_turbo import PersistentTurboKVCache
    from flashquest_b200.eager.decode_step import QuestDecodeInt4, QuestDecodeInt8, QuestDecodeTurbo
    cls, eng = {3: (PersistentTurboKVCache, QuestDecodeTurbo), 4: (PersistentInt4KVCache, QuestDecodeInt4), 8: (PersistentInt8KVCache, QuestDecodeInt8)}[kind]
    L, batch, hq, hkv, d, n = 2, 8, 6, 2, 128, 4099
    g = torch.Generator(device="cuda").manual_seed(12)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    cache = cls(batch_size=batch, num_layers=L, num_kv_heads=hkv, head_dim=d, max_seq_len=4608, page_size=16, dtype=torch.bfloat16)
    for layer in range(L):
        cache.update_quantized(r(batch, hkv, n, d), r(batch, hkv, n, d), layer)
    engine = eng(cache, num_q_heads=hq, retention=0.25, num_sinks=1, window_pages=1)
    for name in ("scores", "compact", "workspace", "scratch"):
        buf = getattr(engine, name, None)
        assert buf is None or (buf.shape[0] == L and buf[0].data_ptr() != buf[1].data_ptr())
    flat = [(r(batch, 1, hq * d), r(batch, 1, hkv * d), r(batch, 1, hkv * d)) for _ in range(L)]
    cos, sin = r(1, 1, d), r(1, 1, d)

    def token(layer):
        cache._seen_tokens[layer] = n
        return engine.forward_token(*flat[layer], cos, sin, layer)
    want = [token(layer).clone() for layer in range(L)]
    rot = engine._rot.clone()                                       # q, k, v of the rotary launch
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(L)]
    for _ in range(20):
        for layer, s in enumerate(streams):
            with torch.cuda.stream(s):
                token(layer)
        torch.cuda.synchronize()
        for layer in range(L):
            assert torch.equal(engine.O[layer].unsqueeze(2), want[layer])
            assert torch.equal(engine._rot[layer], rot[layer])
