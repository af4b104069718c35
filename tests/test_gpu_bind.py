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
